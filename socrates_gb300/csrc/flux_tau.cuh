// flux_tau.cuh -- the mixed-precision column solve in optical-depth form.
//
// A cell (layer of one g-point) enters as three optical depths: absorption
// a, rescaled scattering s and s g' (g' the rescaled asymmetry).  All three
// are linear in the gases, aerosol and cloud condensate, so a band stages
// them once per layer (float4: grey a, s, s g', and the factor of the gas
// term) and a g-point adds k u to the first: no division by the extinction,
// no single-scattering albedo, no renormalised phase function.  With
//
//   S = sum tau  = A (a + s) - C s - B s g'      (two_coeff_basic.F90:99-160)
//   D = diff tau = D0 a
//   x = lambda tau = sqrt(S D),  e = exp(-x),  h = 1 - e^2
//   W = 2 x (1 + e^2) + h (S + D)
//
// the layer of trans_source_coeff.F90:144-200 is
//
//   T = 4 x e / W          R = h (S - D) / W
//   1 - T     = (2 x (1-e)^2 + h (S + D)) / W      (T of thin solar layers from this)
//   1 - T - R = (2 x (1-e)^2 + 2 h D) / W
//
// (gamma = (S - x)/(S + x) multiplied out, x^2 = S D), one division and no
// cancelling difference; the solar source (solar_coefficient_basic.F90:
// 124-219) takes a second one.
//
// P lanes share a column, each with CH layers in registers.  A lane stacks
// its layers from the top into one composite and keeps, per layer, the six
// coefficients that give the flux below and the divergence from the two
// fluxes entering the chunk:
//
//   F_up(top of j) = a_j F_up(bottom of j) + e_j F_dn(chunk top) + g_j
//   div_j          = p_j F_up(bottom of j) + q_j F_dn(chunk top) + v_j
//
// so the chunk is eliminated once (solver_homogen_direct.F90:94-131, from
// the top down).  A prefix scan of the composites and a suffix scan of the
// chunks' affine maps close the column.  The downward fluxes are accumulated
// per g-point at the chunk tops and at the surface only: between, they follow
// once per column from the divergences (TauKernel::finish).
#pragma once

#include <cuda_runtime.h>
#include "socgpu_internal.h"
#include "twostream_math.cuh"

namespace socgpu {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kTauBlock = 4;      // layers of a lane whose McICA cells are evaluated together

// Bounds of a cell's absorption depth: from below the FP64 reference's cap
// on the single-scattering albedo (1 - omega >= 32 epsilon) and a floor that
// keeps S D normal, from above a depth past which a layer is opaque.  NaN
// passes through.
__device__ __forceinline__ float bound_abs(float a, float s) {
  const float lo = fmaf((float)(3.2e1 * kEps64), s, 1.0e-18f);
  float r;
  asm("{\n .reg .f32 t;\n max.NaN.ftz.f32 t, %1, %2;\n min.NaN.ftz.f32 %0, t, 0f58635FA9;\n}" : "=f"(r) : "f"(a), "f"(lo));
  return r;
}

// The scheme's constants (SchemeF) as the cell uses them.
struct SchemeT {
  float A, AC, B, D, hK;     // A, A - C, B, D, K / 2
  __device__ __forceinline__ explicit SchemeT(const FluxParams &p)
      : A(p.scheme_f[0]), AC(p.scheme_f[0] - p.scheme_f[2]), B(p.scheme_f[1]), D(p.scheme_f[3]),
        hK(0.5f * p.scheme_f[4]) {}
};

struct CellT { float T, R, T0, c1, c2, om; };    // om = 1 - T - R

struct LayerT { float e, em1, inv, R, omt, om; };
__device__ __forceinline__ LayerT layer_tau(float S, float D, float x, float &T) {
  LayerT l;
  l.e = exp2f(-kLog2e * x);
  l.em1 = one_minus_exp(x, l.e);
  const float h = fmaf(l.em1, l.e, l.em1), x2 = x + x;
  const float hs = h * (S + D), xm = x2 * l.em1 * l.em1;
  l.inv = 1.0f / fmaf(x2, fmaf(l.e, l.e, 1.0f), hs);
  T = 2.0f * x2 * l.e * l.inv;
  l.R = h * (S - D) * l.inv;
  l.omt = (xm + hs) * l.inv;
  l.om = fmaf(2.0f * h, D, xm) * l.inv;
  return l;
}

// c1 and c2 of the solar source: gam_up and gam_dn over the common factor
// 1 / (x^2 - z^2), z the slant depth; hs = s sec_0 / 2, hx = hs ksi_0.
__device__ __forceinline__ void solar_tau(float S, float D, float x, float z, float hs, float hx, float T0,
                                          float omt0, float R, float omt, float &c1, float &c2) {
  const float r = 1.0f / ((x - z) * (x + z));
  const float gu = r * fmaf(hs, S - z, -hx * (D - z));
  const float opd = fmaf(r, fmaf(hs, S + z, hx * (D + z)), 1.0f);
  c1 = gu * fmaf(T0, omt, omt0) - R * opd;
  c2 = opd * (omt - omt0) - gu * R * T0;
}

// Next to the removable singularity x = z (lambda = sec_0): evaluated at
// (S, D, x) scaled to either side of it and interpolated, as
// solar_c12_singular.  Out of line: few cells take it.
static __device__ __noinline__ float2 solar_tau_singular(float S, float D, float x, float z, float hs, float hx,
                                                         float T0, float omt0) {
  const float ra = z * (1.0f - kSolarSingularTol) / x, rb = z * (1.0f + kSolarSingularTol) / x;
  float T, a1, a2, b1, b2;
  const LayerT la = layer_tau(ra * S, ra * D, ra * x, T);
  solar_tau(ra * S, ra * D, ra * x, z, hs, hx, T0, omt0, la.R, la.omt, a1, a2);
  const LayerT lb = layer_tau(rb * S, rb * D, rb * x, T);
  solar_tau(rb * S, rb * D, rb * x, z, hs, hx, T0, omt0, lb.R, lb.omt, b1, b2);
  const float w = (1.0f - ra) / (rb - ra);
  return make_float2(fmaf(w, b1 - a1, a1), fmaf(w, b2 - a2, a2));
}

// The coefficients of a cell of depths (a, s, s g').
template <int SRC, bool NOSCAT>
__device__ __forceinline__ CellT cell_tau(const SchemeT &sc, int quad, float a, float s, float sg, float sec0) {
  CellT c;
  const float tau = a + s;
  const float sq = (float)kSqEps64;
  if constexpr (NOSCAT) {
    const CoefF f = fast_lw_mix(quad, tau);
    c.T = f.T; c.R = 0.0f; c.T0 = 1.0f; c.c1 = f.c1; c.c2 = f.c2; c.om = f.omtr;
    return c;
  }
  const float S = fmaf(sc.A, a, fmaf(sc.AC, s, -sc.B * sg)), D = sc.D * a;
  const float x = sqrtf(S * D);
  const LayerT l = layer_tau(S, D, x, c.T);
  c.R = l.R; c.om = l.om;
  if constexpr (SRC == SOCGPU_IP_SOLAR) {
    // the transmission of a thin layer from 1 - T: one rounding at 1 in place
    // of four or five, which a column's layers multiply (GA9 short wave,
    // upward flux against 64 bits: 1.1 times the error of the form of
    // trans_source_coeff.F90 without this, 0.75 times with it, for 0.1 to 0.4 %
    // of the time, 3 % at 1000 x 60.  In the infra-red, where the sources
    // dominate, it changes nothing)
    if (l.omt < 0.5f) c.T = 1.0f - l.omt;
    const float z = tau * sec0;
    c.T0 = exp2f(-kLog2e * z);
    const float omt0 = one_minus_exp(z, c.T0);
    const float hs = 0.5f * sec0 * s, hx = sc.hK * sg;
    solar_tau(S, D, x, z, hs, hx, c.T0, omt0, l.R, l.omt, c.c1, c.c2);
    if (fabsf(x - z) < kSolarSingularTol * z) {
      const float2 v = solar_tau_singular(S, D, x, z, hs, hx, c.T0, omt0);
      c.c1 = v.x; c.c2 = v.y;
    }
  } else {
    // infra-red (trans_source_coeff.F90:200-257)
    const float inv_s = 1.0f / (S + sq);
    c.T0 = 1.0f;
    c.c1 = (l.omt + l.R + sq) * inv_s;
    c.c2 = 0.0f;
    if (quad) {
      // D - (1 - T - R) without cancellation (two_coeff_mix), gamma
      // multiplied out: x (S (phi + psi) + x (phi - psi)) / (S (S (1+e) + x (1-e)))
      const float ph = phi_exp(x, l.em1), ps = psi_exp(x, l.e);
      const float q = fmaf(S, 1.0f + l.e, x * l.em1);
      const float dmo = x * fmaf(S, ph + ps, x * (ph - ps)) / (S * q);
      const float num = (tau > (float)kTolQuad64) ? fmaf(2.0f * dmo, 1.0f / (D + sq), -l.om) : dmo;
      c.c2 = -num * inv_s;
    }
  }
  return c;
}

// A stack of layers: reflection for light from above and below, the
// transmission (the same both ways), and the sources leaving it.
struct CompT { float R1, R2, T, Su, Sd; };

__device__ __forceinline__ CompT stack_tau(const CompT &a, const CompT &b) {   // a above b
  const float d = 1.0f / fmaf(-a.R2, b.R1, 1.0f);
  const float ta = d * a.T, tb = d * b.T;
  CompT o;
  o.R1 = fmaf(a.T * b.R1, ta, a.R1);
  o.R2 = fmaf(b.T * a.R2, tb, b.R2);
  o.T = b.T * ta;
  o.Su = fmaf(ta, fmaf(b.R1, a.Sd, b.Su), a.Su);
  o.Sd = fmaf(tb, fmaf(a.R2, b.Su, a.Sd), b.Sd);
  return o;
}

// ---------------------------------------------------------------------------
// The solve of one monochromatic column.  Sm is FluxKernel's view of the
// shared memory; slots as there (lane r's j-th layer in slot j P + r).
template <int P, int CH, bool NOSCAT, bool MCICA, int SRC, class Sm>
struct TauSolve {
  static constexpr int LP = P * CH;
  static constexpr bool kLw = SRC == SOCGPU_IP_INFRA_RED;
  // McICA cells are evaluated in a rolled loop, kBlock layers of the lane at a
  // time, and handed to the unrolled elimination through shared memory (a
  // lane reads back what it wrote): unrolled, the cell with its cloud types
  // is more code than the instruction cache holds (solar, 8000 x 85 in the 8 x
  // 11 tile: 7.1 of 16 stall cycles per instruction were fetches, 1450 us).
  static constexpr int kBlock = MCICA ? kTauBlock : CH;

  // The band's staged optics and, in a cloudy solve, the subcolumn.
  struct Band {
    const float4 *opt;         // [LP] a, s, s g' of the grey constituents; factor of the gas term
    const float4 *copt;        // [n_condensed][LP] a, s, s g', unscaled depth of each condensed component
    const float *cs;           // [LP] the subcolumn's condensate scaling, null in a clear solve
    const float *tkd;          // [LP] unscaled grey depth (i_direct_tau = ip_direct_noscaling), else null
    const float *fm1;          // [LP] adjust_solar_ke - 1 (k_eqv_scl, solar), else null
    const float *dB, *dB2;
    const float *kg;           // [LP] the gas absorption where it is not k0 in every layer, else null
    float k0;
    __device__ __forceinline__ float gas(int s) const { return kg ? kg[s] : k0; }
  };

  // Cloud types present in slot s of a cloudy solve (at most two, bit t).
  __device__ static __forceinline__ unsigned types_of(const Sm &S, float cs, int s) {
    return (cs * S.frac[s] > 0.0f ? 1u : 0u) | (cs * S.frac[LP + s] > 0.0f ? 2u : 0u);
  }
  // Depths of the cell with the components of type t (mcica_sample.F90:472-700).
  __device__ static __forceinline__ void add_type(const FluxParams &p, const Band &b, float cs, int s, int t, float &a,
                                                  float &sc, float &sg, float &un) {
    for (int k = 0; k < p.n_condensed; ++k)
      if (p.comp_type[k] - 1 == t) {
        const float4 c = b.copt[(size_t)k * LP + s];
        a = fmaf(cs, c.x, a); sc = fmaf(cs, c.y, sc); sg = fmaf(cs, c.z, sg); un = fmaf(cs, c.w, un);
      }
  }
  // A second cloud type in the cell: its coefficients, weighted, added to c.
  __device__ static __noinline__ CellT second_type(const FluxParams &p, Band b, float cs, float fc, int s, int t,
                                                   float kg, float sec0, CellT c) {
    const float4 o = b.opt[s];
    float a = fmaf(kg, o.w, o.x), sc = o.y, sg = o.z, un = 0.0f;
    add_type(p, b, cs, s, t, a, sc, sg, un);
    const CellT d = cell_tau<SRC, NOSCAT>(SchemeT(p), p.l_ir_source_quad, bound_abs(a, sc), sc, sg, sec0);
    c.T = fmaf(fc, d.T, c.T); c.R = fmaf(fc, d.R, c.R); c.T0 = fmaf(fc, d.T0, c.T0);
    c.c1 = fmaf(fc, d.c1, c.c1); c.c2 = fmaf(fc, d.c2, c.c2); c.om = fmaf(fc, d.om, c.om);
    return c;
  }

  // The coefficients of slot s: the clear cell, or in a cloudy layer of the
  // subcolumn the sum over its cloud types (mcica_column.F90:336-470).  A
  // lane evaluates one cell whether it is clear or holds one type, so the
  // lanes of a warp do not diverge.
  __device__ static __forceinline__ CellT cell(const FluxParams &p, const Sm &S, const SchemeT &sc, const Band &b,
                                               int s, float sec0) {
    const float4 o = b.opt[s];
    const float kg = b.gas(s);
    float a = fmaf(kg, o.w, o.x), sd = o.y, sg = o.z;
    if (!MCICA || !b.cs)
      return cell_tau<SRC, NOSCAT>(sc, p.l_ir_source_quad, bound_abs(a, sd), sd, sg, sec0);
    const float cs = b.cs[s];
    unsigned types = types_of(S, cs, s);
    float fc = 1.0f, un = 0.0f;
    if (types) {
      const int t = __ffs(types) - 1;
      fc = S.frac[(size_t)t * LP + s];
      add_type(p, b, cs, s, t, a, sd, sg, un);
    }
    CellT c = cell_tau<SRC, NOSCAT>(sc, p.l_ir_source_quad, bound_abs(a, sd), sd, sg, sec0);
    c.T *= fc; c.R *= fc; c.T0 *= fc; c.c1 *= fc; c.c2 *= fc; c.om *= fc;
    types &= types - 1;
    if (types) c = second_type(p, b, cs, S.frac[LP + s], s, 1, kg, sec0, c);
    return c;
  }

  // The direct transmission of slot s (UNSCALED: of the depth before
  // delta-rescaling), times the k_eqv_scl factor.
  template <bool UNSCALED>
  __device__ static __forceinline__ float direct(const FluxParams &p, const Sm &S, const Band &b, int s, float sec0) {
    const float4 o = b.opt[s];
    const float gas = b.gas(s) * o.w, grey = UNSCALED ? b.tkd[s] : o.x + o.y, zk = -kLog2e * sec0;
    float T0;
    unsigned types = 0u;
    float cs = 0.0f;
    if (MCICA && b.cs) { cs = b.cs[s]; types = types_of(S, cs, s); }
    if (!MCICA || !types) {
      T0 = exp2f(zk * (gas + grey));
    } else {
      T0 = 0.0f;
      while (types) {
        const int t = __ffs(types) - 1;
        float a = 0.0f, sd = 0.0f, sg = 0.0f, un = 0.0f;
        add_type(p, b, cs, s, t, a, sd, sg, un);
        T0 = fmaf(S.frac[(size_t)t * LP + s], exp2f(zk * (gas + grey + (UNSCALED ? un : a + sd))), T0);
        types &= types - 1;
      }
    }
    return b.fm1 ? fmaf(T0, b.fm1[s], T0) : T0;
  }
  // The beam at the chunk top and at the surface for f_inc = 1, from the
  // chunk's transmission: an exclusive product scan.
  __device__ static __forceinline__ float beam_scan(float incl, int r, float &bottom) {
#pragma unroll
    for (int d = 1; d < P; d <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, incl, d, P);
      if (r >= d) incl *= y;
    }
    bottom = __shfl_sync(0xffffffffu, incl, P - 1, P);
    const float top = __shfl_up_sync(0xffffffffu, incl, 1, P);
    return r == 0 ? 1.0f : top;
  }
  // The unscaled beam (ip_direct_noscaling, solar_source.F90:157-176): the
  // reported direct flux; returns it at the surface.
  __device__ static __forceinline__ float unscaled_beam(const FluxParams &p, const Sm &S, const Band &b, int r,
                                                        float sec0, float f_inc, float w, float *accd) {
    float t = 1.0f, bottom;
#pragma unroll 1
    for (int j = 0; j < CH; ++j) t *= direct<true>(p, S, b, j * P + r, sec0);
    float f = f_inc * beam_scan(t, r, bottom);
    if (r == 0) accd[LP] += w * f;
#pragma unroll 1
    for (int j = 0; j < CH; ++j) {
      f *= direct<true>(p, S, b, j * P + r, sec0);
      accd[j * P + r] += w * f;
    }
    return f_inc * bottom;
  }

  // acc2: the group's (up, divergence) per slot, slot LP holding the upward
  // flux at the top; accd: its direct flux per slot (solar) or its downward
  // flux (without scattering); anc: the downward flux at the top of each
  // lane's chunk and (entry P) at the surface (with scattering).  w: the weight.
  // buf: the lane's kBlock cells (McICA), 32 lanes apart.
  __device__ static __forceinline__ void solve(const FluxParams &p, const Sm &S, const Band &b, int r, float sec0,
                                               const float *bs, float w, float2 *acc2, float *accd, float *anc,
                                               float4 *buf) {
    const SchemeT sc(p);
    const float f_inc_down = bs[0], alb = bs[2];
    float fd = 0.0f, src = 0.0f;
    // the beam runs relative to the chunk top under McICA (a pass over the
    // cells for the chunk's transmission would evaluate their clouds twice);
    // under clear skies that pass is cheaper than keeping the beam per layer
    constexpr bool kRel = MCICA && !kLw;
    if constexpr (!kLw && !kRel) {
      float t = 1.0f, bottom;
#pragma unroll
      for (int j = 0; j < CH; ++j) t *= direct<false>(p, S, b, j * P + r, sec0);
      fd = bs[1] * beam_scan(t, r, bottom);
      if (b.tkd) bottom = unscaled_beam(p, S, b, r, sec0, bs[1], w, accd);
      else {
        if (r == 0) accd[LP] = fmaf(w, fd, accd[LP]);
        bottom *= bs[1];
      }
      src = (bs[3] - alb) * bottom;
    } else if constexpr (kLw) {
      src = (1.0f - alb) * bs[4];
    } else {
      fd = 1.0f;
    }

    if constexpr (NOSCAT) {
      // solver_no_scat.F90:75-94: a downward and an upward affine scan
      float T[CH], su[CH], sd[CH], om[CH];
      float A = 1.0f, B = 0.0f;              // F_dn(chunk bottom) = A F_dn(chunk top) + B
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int s = j * P + r;
        const CellT c = cell(p, S, sc, b, s, sec0);
        const float u = c.c1 * b.dB[s], q = p.l_ir_source_quad ? c.c2 * b.dB2[s] : 0.0f;
        T[j] = c.T; om[j] = c.om; su[j] = q + u; sd[j] = q - u;
        A = c.T * A; B = fmaf(c.T, B, sd[j]);
      }
#pragma unroll
      for (int d = 1; d < P; d <<= 1) {
        const float yA = __shfl_up_sync(0xffffffffu, A, d, P), yB = __shfl_up_sync(0xffffffffu, B, d, P);
        if (r >= d) { B = fmaf(A, yB, B); A *= yA; }
      }
      const float bottom = fmaf(A, f_inc_down, B);         // inclusive: F_dn below this chunk
      float fdn = __shfl_up_sync(0xffffffffu, bottom, 1, P);
      if (r == 0) fdn = f_inc_down;
      const float f_surf = fmaf(alb, __shfl_sync(0xffffffffu, bottom, P - 1, P), src);
      float C = 1.0f, E = 0.0f;              // F_up(chunk top) = C F_up(chunk bottom) + E
      // the divergence's known part om F_dn(top) - (su + sd) into sd; without
      // scattering the downward flux is known here, and accumulated
      if (r == 0) accd[LP] += w * fdn;
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const float v = fmaf(om[j], fdn, -(su[j] + sd[j]));
        fdn = fmaf(T[j], fdn, sd[j]);
        accd[j * P + r] += w * fdn;
        sd[j] = v;
      }
#pragma unroll
      for (int j = CH - 1; j >= 0; --j) { C *= T[j]; E = fmaf(T[j], E, su[j]); }
#pragma unroll
      for (int d = 1; d < P; d <<= 1) {
        const float yC = __shfl_down_sync(0xffffffffu, C, d, P), yE = __shfl_down_sync(0xffffffffu, E, d, P);
        if (r + d < P) { E = fmaf(C, yE, E); C *= yC; }
      }
      float fu = __shfl_down_sync(0xffffffffu, fmaf(C, f_surf, E), 1, P);
      if (r == P - 1) fu = f_surf;
#pragma unroll
      for (int j = CH - 1; j >= 0; --j) {
        const int s = j * P + r;
        float2 v = acc2[s];
        v.x = fmaf(w, fu, v.x);
        v.y = fmaf(w, fmaf(om[j], fu, sd[j]), v.y);
        acc2[s] = v;
        fu = fmaf(T[j], fu, su[j]);
      }
      if (r == 0) acc2[LP].x += w * fu;
      return;
    }

    // the chunk's layers from the top: the composite c of those above layer
    // j gives the layer's six coefficients, then takes the layer in
    float ca[CH], ce[CH], cg[CH], cp[CH], cq[CH], cv[CH];
    CompT c{0.0f, 0.0f, 1.0f, 0.0f, 0.0f};
    float bt[kRel ? CH : 1];               // the beam below each layer, relative to the chunk top
#pragma unroll
    for (int j0 = 0; j0 < CH; j0 += kBlock) {
    if constexpr (MCICA) {
#pragma unroll 1
      for (int j = j0; j < min(j0 + kBlock, CH); ++j) {
        const CellT x = cell(p, S, sc, b, j * P + r, sec0);
        buf[(j - j0) * 32] = make_float4(x.T, x.R, x.T0, x.c1);
        ((float2 *)(buf + kBlock * 32 - threadIdx.x % 32))[(j - j0) * 32 + threadIdx.x % 32] = make_float2(x.c2, x.om);
      }
    }
#pragma unroll
    for (int j = j0; j < (j0 + kBlock < CH ? j0 + kBlock : CH); ++j) {
      const int s = j * P + r;
      CellT x;
      if constexpr (MCICA) {
        const float4 u = buf[(j - j0) * 32];
        const float2 v = ((const float2 *)(buf + kBlock * 32 - threadIdx.x % 32))[(j - j0) * 32 + threadIdx.x % 32];
        x = CellT{u.x, u.y, u.z, u.w, v.x, v.y};
      } else {
        x = cell(p, S, sc, b, s, sec0);
      }
      float su, sd, ss;
      if constexpr (!kLw) {
        float T0 = x.T0, c2 = x.c2;
        if (b.fm1) {                         // solar_source.F90:115-130 with l_scale_solar
          const float f = b.fm1[s];
          c2 = fmaf(T0, f, c2);
          T0 = fmaf(T0, f, T0);
        }
        su = x.c1 * fd; sd = c2 * fd;        // solar_source.F90:146-155
        ss = su + sd;
        fd *= T0;
        if constexpr (kRel) bt[j] = fd;
        else if (!b.tkd) accd[s] += w * fd;
      } else {                               // ir_source.F90:93-119
        const float u = x.c1 * b.dB[s], q = p.l_ir_source_quad ? x.c2 * b.dB2[s] : 0.0f;
        su = q + u; sd = q - u; ss = q + q;
      }
      const float dd = 1.0f / fmaf(-c.R2, x.R, 1.0f);
      const float a = x.T * dd, dr = dd * x.R;
      const float e = dr * c.T, g = dd * fmaf(x.R, c.Sd, su);
      ca[j] = a; ce[j] = e; cg[j] = g;
      cp[j] = x.om * fmaf(c.R2, a, 1.0f);
      cq[j] = x.om * fmaf(c.R2, e, c.T);
      cv[j] = fmaf(x.om, fmaf(c.R2, g, c.Sd), -ss);
      c.R1 = fmaf(c.T, e, c.R1);
      c.Su = fmaf(c.T, g, c.Su);
      c.Sd = fmaf(a, fmaf(c.R2, su, c.Sd), sd);
      c.R2 = fmaf(x.T * c.R2, a, x.R);
      c.T *= a;
    }
    }
    if constexpr (kRel) {
      // the sources in the beam's own units
      float bottom;
      fd = bs[1] * beam_scan(fd, r, bottom);
      c.Su *= fd; c.Sd *= fd;
      bottom *= bs[1];
      if (b.tkd) {
        bottom = unscaled_beam(p, S, b, r, sec0, bs[1], w, accd);
      } else {
        if (r == 0) accd[LP] = fmaf(w, fd, accd[LP]);
#pragma unroll
        for (int j = 0; j < CH; ++j) accd[j * P + r] += (w * fd) * bt[j];
      }
      src = (bs[3] - alb) * bottom;
    }
    // the stack above this chunk: an inclusive scan, shifted by one lane
    CompT pre = c;
#pragma unroll
    for (int d = 1; d < P; d <<= 1) {
      CompT y;
      y.R1 = __shfl_up_sync(0xffffffffu, pre.R1, d, P);
      y.R2 = __shfl_up_sync(0xffffffffu, pre.R2, d, P);
      y.T = __shfl_up_sync(0xffffffffu, pre.T, d, P);
      y.Su = __shfl_up_sync(0xffffffffu, pre.Su, d, P);
      y.Sd = __shfl_up_sync(0xffffffffu, pre.Sd, d, P);
      if (r >= d) pre = stack_tau(y, pre);
    }
    // F_dn = rho F_up + sig at the chunk top
    float rho = __shfl_up_sync(0xffffffffu, pre.R2, 1, P);
    float sig = __shfl_up_sync(0xffffffffu, fmaf(pre.T, f_inc_down, pre.Sd), 1, P);
    if (r == 0) { rho = 0.0f; sig = f_inc_down; }
    // F_up(chunk top) = A F_up(chunk bottom) + B
    const float q1 = 1.0f / fmaf(-c.R1, rho, 1.0f);
    const float A0 = c.T * q1, B0 = fmaf(c.R1, sig, c.Su) * q1;
    float A = A0, B = B0, f_surf = 0.0f;
    if (r == P - 1) {
      // the surface closes the last chunk: F_up = alb F_dn + src
      const float rb = fmaf(c.T * rho, A0, c.R2), sb = fmaf(c.T, fmaf(rho, B0, sig), c.Sd);
      f_surf = fmaf(alb, sb, src) / fmaf(-alb, rb, 1.0f);
      anc[P] = fmaf(w, fmaf(rb, f_surf, sb), anc[P]);
      B = fmaf(A, f_surf, B); A = 0.0f;
    }
#pragma unroll
    for (int d = 1; d < P; d <<= 1) {
      const float yA = __shfl_down_sync(0xffffffffu, A, d, P), yB = __shfl_down_sync(0xffffffffu, B, d, P);
      if (r + d < P) { B = fmaf(A, yB, B); A *= yA; }
    }
    float fu = __shfl_down_sync(0xffffffffu, B, 1, P);     // F_up at the chunk bottom
    if (r == P - 1) fu = f_surf;
    const float fdt = fmaf(rho, B, sig);                   // B: F_up at this chunk's top
    anc[r] = fmaf(w, fdt, anc[r]);
#pragma unroll
    for (int j = CH - 1; j >= 0; --j) {
      const int s = j * P + r;
      float2 v = acc2[s];
      v.x = fmaf(w, fu, v.x);
      const float vj = kRel ? cv[j] * fd : cv[j], gj = kRel ? cg[j] * fd : cg[j];
      v.y = fmaf(w, fmaf(cp[j], fu, fmaf(cq[j], fdt, vj)), v.y);
      acc2[s] = v;
      fu = fmaf(ca[j], fu, fmaf(ce[j], fdt, gj));
    }
    if (r == 0) acc2[LP].x += w * fu;
  }
};

}  // namespace socgpu
