// flux_tau_kernel.cuh -- the mixed-precision flux kernel: staging, the loop
// over g-points and the outputs of `cols` adjacent columns per CTA, around
// the column solve of flux_tau.cuh.
//
// The profile index runs fastest in memory, so one column's values lie
// n_profile * 8 bytes apart: a CTA that stages a single column moves a
// 32-byte sector per 8-byte value and a cache line per lane.  Four adjacent
// columns use the whole sector.  Each column has its own block of shared
// memory and its own warps; the columns meet only in the staging and the
// output loops, whose threads run over (layer, column) with the column
// fastest.  A thread stages one layer of one column for every band of the
// batch, so the layer's fields, logarithms and gas amounts are read and
// formed once and not once per band.
#pragma once

#include <algorithm>
#include "flux_kernel.cuh"
#include "flux_tau.cuh"

namespace socgpu {

// The layout of `cols` columns of batch p with nbat bands staged at a time
// and n_groups solve groups (of P lanes) per column.
inline TauLayout tau_layout(const FluxParams &p, int LP, int P, int cols, int warps, int nbat, bool mcica) {
  TauLayout l{};
  const bool lw = p.isolir == SOCGPU_IP_INFRA_RED;
  const bool unscaled = !lw && p.i_direct_tau == SOCGPU_IP_DIRECT_NOSCALING;
  const int n_groups = warps * 32 / P;
  l.cols = cols; l.warps = warps; l.nbat = nbat;
  size_t o = 0;
  auto take = [&](size_t words) { size_t r = (o + 15) & ~(size_t)15; o = r + words * 4; return (unsigned)r; };
  const size_t nb = nbat, n = LP;
  l.opt = take(nb * n * 4);
  l.copt = mcica ? take(nb * p.n_condensed * n * 4) : 0;
  l.tkd = unscaled ? take(nb * n) : 0;
  // a single absorber's amount is part of the staged depths
  l.amt = (p.max_abs > 1 || p.term_scr) ? take(nb * p.max_abs * n) : 0;
  l.aux = (p.keqv && !lw) ? take(nb * p.max_abs * n) : 0;
  l.bscal = take(nb * kBandScal);
  l.planck = lw ? take(nb * (n + 1)) : 0;
  l.dB = lw ? take(nb * n) : 0;
  l.dB2 = lw ? take(nb * n) : 0;
  l.pl = lw ? take(n + 1) : 0;
  l.p = p.term_scr ? take(n) : 0;
  l.t = p.term_scr ? take(n) : 0;
  l.mass = take(n);
  l.frac = mcica ? take(2 * n) : 0;
  l.csub = mcica ? take((size_t)p.n_subcol_gen * n) : 0;
  l.lkf = p.lk_on ? take(4 * n) : 0;
  l.lki = p.lk_on ? take(n) : 0;
  l.sbf = p.n_sb > 0 ? take((size_t)p.n_sb * n) : 0;
  l.sbj = p.n_sb > 0 ? take((size_t)p.n_sb * n) : 0;
  // a group's row of gas absorption, where it is not one k for all layers
  l.scr = (p.term_scr || p.max_abs > 1) ? take((size_t)n_groups * n) : 0;
  // a group's accumulators: the groups of a warp start P slots apart modulo
  // the 32 banks
  l.acc_stride = LP + 1;
  while ((2 * l.acc_stride) % 32 != (2 * P) % 32) ++l.acc_stride;
  l.accd_stride = LP + 1;
  while (l.accd_stride % 32 != P % 32) ++l.accd_stride;
  l.acc2 = take((size_t)n_groups * l.acc_stride * 2);
  // the direct flux, or without scattering the downward flux
  const bool third = !lw || p.i_scatter_method != SOCGPU_IP_SCATTER_FULL;
  l.accd = third ? take((size_t)n_groups * l.accd_stride) : 0;
  // the downward flux at the tops of the lanes' chunks and at the surface
  l.anc = p.i_scatter_method == SOCGPU_IP_SCATTER_FULL ? take((size_t)n_groups * (P + 1)) : 0;
  // adjacent columns 32 bytes apart modulo the banks: the lanes of a staging
  // store (two slots of four columns per quarter-warp) meet no conflict
  while (o % 128 != 32) ++o;
  l.stride = (unsigned)o;
  return l;
}

// A CTA's shared memory: the columns' blocks, the band records and under
// McICA each warp's cells (six words for kTauBlock layers of every lane).
inline size_t tau_bytes(const FluxParams &p) {
  const size_t cells = p.mcica ? (size_t)p.tau.cols * p.tau.warps * kTauBlock * 32 * 24 : 0;
  return (size_t)p.tau.stride * p.tau.cols + sizeof(BandLite) * p.tau.nbat + cells;
}

// What the current device grants a kernel: SMs, dynamic shared memory of a CTA,
// shared memory of an SM, and what a resident CTA takes of it besides (the
// device's 1 KB and the kernel's static part).
struct TauChip { int n_sm; size_t cta, sm, besides; };

// The layout of batch p with `cols` columns to a CTA of `warps` warps: the most
// bands at a time, at least `least`, that leave 16 warps resident; one band of
// one column may take all of a CTA's shared memory.
inline bool tau_place(FluxParams &p, int LP, int P, int warps, int cols, int least, bool mcica, const TauChip &chip) {
  const size_t want = std::min(chip.cta, chip.cta * warps / 16);
  for (int nb = p.last_band - p.first_band + 1; nb >= least; --nb) {
    p.tau = tau_layout(p, LP, P, cols, warps / cols, nb, mcica);
    const size_t bytes = tau_bytes(p);
    if (bytes <= want || (nb == 1 && cols == 1 && bytes <= chip.cta)) return true;
  }
  return false;
}

// The columns per CTA, and the bands staged at a time, of a CTA of `warps`
// warps.  Few columns are spread over the SMs, one or two to a CTA while the
// chip holds them all at a time (16 warps to an SM); past that,
// four adjacent columns if all their bands fit the share of shared memory
// that leaves 16 warps resident, else two with at least half the bands; else
// one.  Measured on GB300 (us, mixed, 8 warps): solar 10000 x 100 454 with
// four columns, 475 with two, 715 with one; long wave 1000 x 60 39, 52, 78;
// scattering long wave 3001 x 137 377 (bands in batches), 364, 393; solar
// McICA 8000 x 85 1400 (in batches), 1252, 1445.
// The rule looks at the columns of the caller's call: a few columns in wide
// arrays are spread like any other few (27 x 137 solar in arrays of 2500
// columns: 57.5 us by the leading extent, 22.6 by the columns), and the windows that a
// host call is cut into sum in the order of the whole call.
// False: one band of one column does not fit.
inline bool tau_fit(FluxParams &p, int LP, int P, int warps, bool mcica, const TauChip &chip) {
  const int resident = 16 * chip.n_sm / warps, nb = p.last_band - p.first_band + 1;
  const int most = warps % 4 != 0 || p.width <= resident ? 1 : p.width <= 2 * resident ? 2 : 4;
  for (int cols = most; cols >= 1; cols /= 2)
    if (tau_place(p, LP, P, warps, cols, cols == 4 ? nb : cols == 2 ? (nb + 1) / 2 : 1, mcica, chip)) return true;
  return false;
}

// Equivalent extinction, whose minor absorbers' solves leave most of a CTA
// waiting: the time of one wave of CTAs grows little with the columns on an
// SM, and with the columns a warp takes one after another.  The shape with the
// least (waves x time of a wave) is taken, each at the residence that its
// registers and shared memory allow.  The relative times are those of the GA9
// short-wave and long-wave files over 38 to 137 layers and 300 to 4000 columns
// on GB300, which agree to a fifth (us of a full wave, short wave at 38 / 70 /
// 137 layers: one column on 8 warps 50 / 60 / 71, at three CTAs to an SM 54 / 67,
// one on 4 warps 71 / 87 / 144, two 111 / 157 / 240, four 193 / 283 / 350; under
// McICA one on 4 warps takes 1.4 to 2.3 times one on 8, more with more layers
// to a lane).  A line between 8 and 4 warps at 304 columns, with never more than
// 16 resident warps, was slower than this by up to a third (38 x 400 69 us, now
// 54; long wave 38 x 700 173, now 121).
// mb: resident CTAs of 8 warps in registers; the relative times on tiles built
// for three or more of them (short chunks) and on the others.
struct TauShape { int warps, cols, mb; double time, time_long; };
constexpr TauShape kKeqvShapes[] = {{8, 1, 2, 1.0, 1.0}, {8, 1, 3, 1.1, 0.0}, {8, 1, 4, 1.35, 0.0}, {4, 1, 2, 1.5, 1.9},
                                    {4, 1, 3, 1.6, 0.0}, {4, 2, 2, 2.6, 3.1}, {4, 4, 2, 4.65, 5.0}};
// The shape of n items that run together (of `given` warps unless that is 0) on
// a tile built for up to `dense` resident CTAs, and the items' layouts; warps
// 0: none fits, or an item is not of equivalent extinction.
inline TauShape tau_choose(FluxParams *items, int n, int LP, int P, int given, bool mcica, int dense, const TauChip &chip) {
  TauShape best{};
  double least = 0.0;
  for (int i = 0; i < n; ++i)
    if (!items[i].keqv) return best;
  for (const TauShape &s : kKeqvShapes) {
    if (s.mb > std::max(dense, 2) || (given && s.warps != given)) continue;
    size_t bytes = 0;
    long long ctas = 0;
    bool fits = true;
    for (int i = 0; i < n && fits; ++i) {
      const int nb = items[i].last_band - items[i].first_band + 1;
      fits = tau_place(items[i], LP, P, s.warps, s.cols, s.cols == 2 ? (nb + 1) / 2 : 1, mcica, chip);
      bytes = std::max(bytes, tau_bytes(items[i]));
      ctas += (items[i].width + s.cols - 1) / s.cols;
    }
    if (!fits) continue;
    const long long on_sm = std::max<long long>(1, std::min<long long>(std::min(s.mb, dense) * 8 / s.warps, chip.sm / (bytes + chip.besides)));
    double wave = dense > 2 ? s.time : s.time_long;
    if (mcica && s.warps == 4 && s.cols == 1) wave = LP / P <= 3 ? 1.49 : LP / P == 4 ? 1.6 : 2.1;
    const double t = wave * (double)((ctas + on_sm * chip.n_sm - 1) / (on_sm * chip.n_sm));
    if (best.warps == 0 || t < least) { best = s; least = t; }
  }
  for (int i = 0; i < n && best.warps; ++i) {
    const int nb = items[i].last_band - items[i].first_band + 1;
    tau_place(items[i], LP, P, best.warps, best.cols, best.cols == 2 ? (nb + 1) / 2 : 1, mcica, chip);
  }
  return best;
}

// Whether a class of ctas CTAs, most of them with one column on 8 warps, runs
// with three of them resident on an SM in place of two: fewer waves, each a
// tenth longer.  Graphs of 38-layer solar columns on GB300 (us): 32 items of
// 16 columns 33 with two resident, 35 with three; 32 of 64 105 and 86; 16 of
// 200 160 and 133; long wave without scattering 41 and 43, 131 and 105, 201
// and 162.
inline bool tau_narrow(long long ctas, const TauChip &chip) {
  const auto waves = [&](long long n) { return (double)((ctas + n * chip.n_sm - 1) / (n * chip.n_sm)); };
  return 1.1 * waves(3) < waves(2);
}

// A value of the caller's column arrays.  The staging reads each once, so it
// does not take a line of the L1 cache, which holds the band tables.
__device__ __forceinline__ double ld_col(const double *a) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(a));
  return v;
}
__device__ __forceinline__ float in_col(const double *a) { return narrow(ld_col(a)); }

template <int P, int CH, bool NOSCAT, bool MCICA, int SRC>
struct TauKernel {
  using FK = FluxKernel<float, true, P, CH, NOSCAT, MCICA, SRC>;
  using Sm = typename FK::Smem;
  using Solve = TauSolve<P, CH, NOSCAT, MCICA, SRC, Sm>;
  static constexpr int LP = P * CH;
  static constexpr bool kLw = SRC == SOCGPU_IP_INFRA_RED;
  static constexpr bool kThird = !kLw || NOSCAT;    // accd in use

  // Column c's arrays; group gi of the column.
  __device__ static __forceinline__ Sm bind(unsigned char *base, const TauLayout &l, int c, int gi) {
    Sm s{};
    unsigned char *b = base + (size_t)c * l.stride;
    s.opt = (float4 *)(b + l.opt); s.copt = (float4 *)(b + l.copt); s.tkd = (float *)(b + l.tkd);
    s.amt = (float *)(b + l.amt); s.aux = (float *)(b + l.aux); s.bscal = (float *)(b + l.bscal);
    s.planck = (float *)(b + l.planck); s.dB = (float *)(b + l.dB); s.dB2 = (float *)(b + l.dB2);
    s.pl = (float *)(b + l.pl);
    s.p = (float *)(b + l.p); s.t = (float *)(b + l.t); s.mass = (float *)(b + l.mass);
    s.frac = (float *)(b + l.frac); s.csub = (float *)(b + l.csub);
    s.lkf = (float *)(b + l.lkf); s.lki = (int *)(b + l.lki); s.sbf = (float *)(b + l.sbf); s.sbj = (int *)(b + l.sbj);
    s.scr = (float *)(b + l.scr) + (size_t)gi * LP;
    s.acc2 = (float2 *)(b + l.acc2); s.accd = (float *)(b + l.accd); s.anc = (float *)(b + l.anc);
    return s;
  }

  // A band whose solved gas absorption is one absorber's k times an amount,
  // the same k in every layer.
  __device__ static __forceinline__ bool single_gas(const FluxParams &p, const BandInfo &bd) {
    return p.l_gas && (bd.n_abs == 1 || (p.keqv && bd.n_abs > 1)) && bd.gas[0].i_scale_k != SOCGPU_IP_SCALE_TERM;
  }

  // Bands bstart .. bstart + nb - 1 of nc columns from col0: the depths of
  // the grey constituents and gas amounts (radiance_calc.F90:883-1600 band
  // loop), the clouds' and the Planck terms.  `first`: the band-independent
  // fields too.
  __device__ static void stage(const FluxParams &p, unsigned char *base, const BandLite *lite, int col0, int nc,
                               int bstart, int nb, bool first) {
    const TauLayout &l = p.tau;
    const int L = p.n_layer, C = l.cols;
    const size_t ndp = p.nd_profile, ndl = p.nd_layer;
    const bool unscaled = !kLw && p.i_direct_tau == SOCGPU_IP_DIRECT_NOSCALING;
    for (int q = threadIdx.x; q < C * LP; q += blockDim.x) {
      const int c = q & (C - 1), i = q / C, s = FK::slot(i), col = col0 + c;
      if (c >= nc) continue;
      const Sm S = bind(base, l, c, 0);
      if (i >= L) {
        // padding slots are transparent
        for (int bi = 0; bi < nb; ++bi) {
          S.opt[bi * LP + s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (unscaled) S.tkd[bi * LP + s] = 0.0f;
          if (kLw) { S.dB[bi * LP + s] = 0.0f; S.dB2[bi * LP + s] = 0.0f; }
        }
        if (MCICA) S.frac[s] = S.frac[LP + s] = 0.0f;
        continue;
      }
      const size_t at = (size_t)col + ndp * i;
      const float pv = in_col(p.p + at), tv = in_col(p.t + at), m = in_col(p.mass + at);
      if (first) {
        S.mass[s] = m;
        if (p.term_scr) { S.p[s] = pv; S.t[s] = tv; }
        if (p.lk_on) FK::lookup_slot(p, S.lkf, S.lki, S.sbf, S.sbj, pv, tv, col, s, i);
      }
      stage_grey(p, S, lite, col, i, s, bstart, nb, pv, tv, m, unscaled);
      if (kLw) stage_planck(p, S, lite, col, i, s, nb, tv);
      if (MCICA) stage_cloud(p, S, col, i, s, bstart, nb, m, first);
    }
  }

  __device__ static __forceinline__ void stage_grey(const FluxParams &p, const Sm &S, const BandLite *lite, int col,
                                                    int i, int s, int bstart, int nb, float pv, float tv, float m,
                                                    bool unscaled) {
    const size_t ndp = p.nd_profile, ndl = p.nd_layer, at = (size_t)col + ndp * i, plane = ndp * ndl;
    const bool aero = p.l_aerosol_mode && p.n_mode > 0;
    const size_t bstep = plane * p.nd_mode;
    const float mmr0 = aero ? in_col(p.mode_mix_ratio + at) : 0.0f;
    float water = 0.0f, rho = 0.0f, scale = 1.0f;
    if (p.l_continuum) {
      water = in_col(p.gas_mix_ratio + at + plane * p.i_water);
      rho = in_col(p.density + at);
    }
    // the first absorber's mixing ratio and the first mode's optics are read
    // one band ahead
    double gm = 0.0, na = 0.0, ns = 0.0, ng = 0.0;
    auto ahead = [&](int bi) {
      if (p.l_gas && lite[bi].n_abs > 0) gm = ld_col(p.gas_mix_ratio + at + plane * lite[bi].species);
      if (aero) {
        const size_t ao = at + bstep * (bstart + bi);
        na = ld_col(p.mode_absorption + ao); ns = ld_col(p.mode_scattering + ao); ng = ld_col(p.mode_asymmetry + ao);
      }
    };
    ahead(0);
#pragma unroll 1
    for (int bi = 0; bi < nb; ++bi) {
      const int b = bstart + bi, q = bi * LP + s;
      const BandLite &bd = lite[bi];
      const double gm_ = gm, na_ = na, ns_ = ns, ng_ = ng;
      if (bi + 1 < nb) ahead(bi + 1);
      // grey optics: grey_opt_prop.F90:470-790 (Rayleigh, aerosols, continua)
      float kes = p.l_rayleigh ? bd.rayleigh : 0.0f, kabs = 0.0f, phf = 0.0f, fwd = 0.0f;
      if (p.l_aerosol) FK::classic_aerosol(p, col, i, b, kabs, kes, phf, fwd);
      if (p.l_aer_prsc) {
        // prescribed species: the sums of the prescribed-property kernel
        const int nb_all = p.last_band - p.first_band + 1;
        const size_t pp = (size_t)nb_all * p.n_layer;
        const size_t q0 = ((size_t)col * 4 * nb_all + (b - (p.first_band - 1))) * p.n_layer + i;
        kabs += in_col(p.aer_prsc + q0);
        kes += in_col(p.aer_prsc + pp + q0);
        phf += in_col(p.aer_prsc + 2 * pp + q0);
        if (p.l_rescale) fwd += in_col(p.aer_prsc + 3 * pp + q0);
      }
      if (aero) {
        add_mode(p, mmr0, narrow(na_), narrow(ns_), narrow(ng_), kabs, kes, phf, fwd);
        for (int j = 1; j < p.n_mode; ++j) {
          const size_t a4 = at + plane * ((size_t)j + (size_t)p.nd_mode * b);
          add_mode(p, in_col(p.mode_mix_ratio + at + plane * j), in_col(p.mode_absorption + a4),
                   in_col(p.mode_scattering + a4), in_col(p.mode_asymmetry + a4), kabs, kes, phf, fwd);
        }
      }
      if (p.l_continuum)
        for (int j = 0; j < bd.n_cont; ++j) {
          const BandCont &c = p.bands[b].cont[j];
          kabs += c.k_f * continuum(p, c, pv, tv, rho, water);
        }
      // the depths (flux_tau.cuh): absorption, scattering with the forward
      // peak taken out, times the asymmetry left
      float a = kabs * m, sd = 0.0f, sg = 0.0f, u = m;
      if (p.i_scatter_method == SOCGPU_IP_SCATTER_FULL) {
        sd = (kes - fwd) * m;
        sg = (phf - fwd) * m;
      } else if (p.i_scatter_method != SOCGPU_IP_NO_SCATTER_ABS) {
        a = (kabs + kes) * m;
      }
      if (unscaled) S.tkd[q] = (kabs + kes) * m;
      // gas amounts (radiance_calc.F90:1330-1470): scaled in pressure and
      // temperature under ip_scale_band, else the mixing ratio
      const int n_abs = p.l_gas ? min(bd.n_abs, p.max_abs) : 0;
      if (n_abs > 0) {
        float v = narrow(gm_);
        const bool single = (n_abs == 1 || p.keqv) && bd.i_scale_k != SOCGPU_IP_SCALE_TERM;
        if (bd.i_scale_k == SOCGPU_IP_SCALE_BAND) {
          // consecutive bands that scale alike share the factor
          if (bi == 0 || !bd.same)
            scale = scale_factor_mix(bd.i_scale_fnc, pv, tv, bd.p_ref, bd.t_ref, bd.scale, bd.l_doppler, bd.doppler_cor);
          v *= scale;
          v = v > 0.0f ? v : 0.0f;
        }
        if (single) u = v * m;
        if (p.max_abs > 1 || p.term_scr) {
          S.amt[(size_t)bi * p.max_abs * LP + s] = v;
          for (int j = 1; j < n_abs; ++j) {
            const BandGas &gs = p.bands[b].gas[j];
            v = in_col(p.gas_mix_ratio + at + plane * gs.species);
            if (gs.i_scale_k == SOCGPU_IP_SCALE_BAND) {
              v *= scale_factor_mix(gs.i_scale_fnc, pv, tv, gs.p_ref_f, gs.t_ref_f, gs.scale_f, gs.l_doppler,
                                    gs.doppler_cor_f);
              v = v > 0.0f ? v : 0.0f;
            }
            S.amt[((size_t)bi * p.max_abs + j) * LP + s] = v;
          }
        }
      }
      S.opt[q] = make_float4(a, sd, sg, u);
    }
  }

  __device__ static __forceinline__ void add_mode(const FluxParams &p, float mmr, float ka, float ksc, float g,
                                                  float &kabs, float &kes, float &phf, float &fwd) {
    kabs = fmaf(mmr, ka, kabs);
    const float ks = mmr * ksc, kg = ks * g;
    kes += ks;
    phf += kg;
    if (p.l_rescale) {
      if (p.n_order_forward == 1) fwd += kg;
      else if (p.n_order_forward == 2) fwd = fmaf(kg, g, fwd);
      else {
        float gp = 1.0f;
        for (int o = 0; o < p.n_order_forward; ++o) gp *= g;
        fwd = fmaf(ks, gp, fwd);
      }
    }
  }

  // The amount of a continuum (rescale_continuum.F90): self, the molar
  // density of water times water; foreign, the air's times water.
  __device__ static __forceinline__ float continuum(const FluxParams &p, const BandCont &c, float pv, float tv,
                                                    float rho, float water) {
    float a = __powf(pv / c.p_ref_f, c.scale_f[0]);
    if (c.fnc == SOCGPU_IP_SCALE_POWER_LAW) {
      a = a * __powf(tv / c.t_ref_f, c.scale_f[1]);
    } else if (c.fnc == SOCGPU_IP_SCALE_POWER_QUAD) {
      const float x = tv / c.t_ref_f - 1.0f;
      a = a * (1.0f + c.scale_f[1] * x + c.scale_f[2] * (x * x));
    }
    if (c.type == SOCGPU_IP_SELF_CONTINUUM) {
      a = a * (rho * water * (1.0f / 0.0180153f)) * water;
    } else if (c.type == SOCGPU_IP_FRN_CONTINUUM) {
      a = p.l_mixing_ratio ? a * rho * water * (1.0f / 0.028966f) : a * rho * water * (1.0f - water) * (1.0f / 0.028966f);
    }
    return a;
  }

  // The argument of the band records' Planck polynomials, T / T_ref - 1: with
  // the reference's T / T_ref the terms cancel in the seventh
  // digit of FP32 (the records' coefficients are expanded about T_ref in
  // FP64).
  __device__ static __forceinline__ float planck_arg(const FluxParams &p, float t) {
    return (t - p.t_ref_planck_f) / p.t_ref_planck_f;
  }
  // diff_planck_source (diff_planck_source_mod.F90:102-136)
  __device__ static __forceinline__ void stage_planck(const FluxParams &p, const Sm &S, const BandLite *lite, int col,
                                                      int i, int s, int nb, float tv) {
    const size_t ndp = p.nd_profile;
    const float x0 = planck_arg(p, in_col(p.t_level + col + ndp * i));
    const float x1 = planck_arg(p, in_col(p.t_level + col + ndp * (i + 1)));
    const float xl = planck_arg(p, tv);
    for (int bi = 0; bi < nb; ++bi) {
      const float *c = lite[bi].planck;
      S.planck[bi * (LP + 1) + s] = planck_mix(c, p.n_deg_fit, x1);
      if (i == 0) S.planck[bi * (LP + 1) + LP] = planck_mix(c, p.n_deg_fit, x0);
      S.dB[bi * LP + s] = planck_diff_mix(c, p.n_deg_fit, x1, x0);
      if (p.l_ir_source_quad)
        S.dB2[bi * LP + s] = 2.0f * (planck_diff_mix(c, p.n_deg_fit, x1, xl) + planck_diff_mix(c, p.n_deg_fit, x0, xl));
    }
  }

  // The layer's cloud fractions, subcolumn scalings and the depths of its
  // condensed components per unit scaling.
  __device__ static __forceinline__ void stage_cloud(const FluxParams &p, const Sm &S, int col, int i, int s, int bstart,
                                                     int nb, float m, bool first) {
    const int ict = p.id_ct, nc = p.n_condensed;
    const bool in = i >= ict;
    const size_t ndp = p.nd_profile, ndc = p.nd_layer - ict, qc = (size_t)col + ndp * (size_t)(in ? i - ict : 0);
    const float w = in ? in_col(p.w_cloud + qc) : 0.0f;
    if (first) {
      // a clear layer is known by its fractions
      for (int t = 0; t < 2; ++t)
        S.frac[t * LP + s] = (w > 0.0f && t < p.n_cloud_type) ? in_col(p.frac_cloud + qc + ndp * ndc * t) : 0.0f;
      for (int k = 0; k < p.n_subcol_gen; ++k)
        S.csub[k * LP + s] = in ? in_col(p.c_sub + qc + ndp * ndc * k) : 0.0f;
    }
    for (int k = 0; k < nc; ++k) {
      float re = 0.0f, qm = 0.0f;
      if (w > 0.0f) {
        re = in_col(p.condensed_dim_char + qc + ndp * ndc * k);
        qm = in_col(p.condensed_mix_ratio + qc + ndp * ndc * k);
      }
      const bool water = p.comp_phase[k] == SOCGPU_IP_PHASE_WATER;
      const float *tab = (water ? p.drop_parm_f : p.ice_parm_f) + (size_t)p.comp_parm_index[k] * p.n_band * kCloudParm;
      for (int bi = 0; bi < nb; ++bi) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (re > 0.0f) {
          float kext, coalb, g;
          FK::cloud_optics(p.comp_scheme[k], !water, tab + (size_t)(bstart + bi) * kCloudParm, re, qm, kext, coalb, g);
          const float ks = kext * (1.0f - coalb), ph = ks * g, fw = p.l_rescale ? ph * g : 0.0f;
          v = make_float4(kext * coalb * m, (ks - fw) * m, (ph - fw) * m, kext * m);
        }
        S.copt[((size_t)bi * nc + k) * LP + s] = v;
      }
    }
  }

  // Per-band boundary values (solve_band_random_overlap.F90:565-600,
  // column_solver.F90), by the last threads of the CTA, which have the least
  // to stage.
  __device__ static void stage_boundary(const FluxParams &p, unsigned char *base, const BandLite *lite, int col0, int nc,
                                        int bstart, int nb) {
    const int C = p.tau.cols, L = p.n_layer;
    const size_t ndp = p.nd_profile;
    for (int q = blockDim.x - 1 - threadIdx.x; q < C * nb; q += blockDim.x) {
      const int c = q & (C - 1), bi = q / C, b = bstart + bi, col = col0 + c;
      if (c >= nc) continue;
      float *v = bind(base, p.tau, c, 0).bscal + bi * kBandScal;
      v[2] = in_col(p.rho_alb + col + ndp * (0 + 2 * (size_t)b));
      v[3] = in_col(p.rho_alb + col + ndp * (1 + 2 * (size_t)b));
      v[5] = p.weight_band ? load_in<float>(p.weight_band + b) : 1.0f;
      if (kLw) {
        const float *k = lite[bi].planck;
        const float xs = planck_arg(p, in_col(p.t_level + col + ndp * L));
        v[0] = -planck_mix(k, p.n_deg_fit, planck_arg(p, in_col(p.t_level + col)));
        v[1] = 0.0f;
        // the surface's Planck flux given per band (l_flux_ground, tiles), or
        // that of its temperature, less that of the lowest level
        v[4] = p.flux_ground ? in_col(p.flux_ground + col + ndp * b) - planck_mix(k, p.n_deg_fit, xs)
                             : planck_diff_mix(k, p.n_deg_fit, planck_arg(p, in_col(p.t_ground + col)), xs);
      } else {
        v[0] = in_col(p.solar_irrad + col) * lite[bi].solar / in_col(p.zen_0 + col);
        v[1] = v[0];
        v[4] = 0.0f;
      }
    }
  }

  // k_eqv of every slot into the grey absorption, and the solar direct-beam
  // factor less one (solve_band_k_eqv_scl.F90:975-1040), by the column's own
  // threads (t of nt).
  __device__ static void fold_keqv(const FluxParams &p, const Sm &S, int bstart, int nb, float sec0, int t, int nt) {
    const int L = p.n_layer, max_abs = p.max_abs;
    const bool unscaled = !kLw && p.i_direct_tau == SOCGPU_IP_DIRECT_NOSCALING;
    for (int q = t; q < nb * LP; q += nt) {
      const int bi = q / LP, s = q - bi * LP;
      if (FK::layer_of_slot(s) >= L) {
        if (!kLw) S.aux[(size_t)bi * max_abs * LP + s] = 0.0f;
        continue;
      }
      const int na = p.l_gas ? min(p.bands[bstart + bi].n_abs, max_abs) : 0;
      float keq = 0.0f, adj = 0.0f;
      for (int j = 1; j < na; ++j) {
        keq += S.amt[((size_t)bi * max_abs + j) * LP + s];
        if (!kLw) adj += S.aux[((size_t)bi * max_abs + j) * LP + s];
      }
      const float d = keq * S.mass[s];
      S.opt[q].x += d;
      if (unscaled) S.tkd[q] += d;
      if (!kLw) S.aux[(size_t)bi * max_abs * LP + s] = expm1f(adj + fminf(d * sec0, 36.04365338911715f));
    }
  }

  // One g-point: the clear solve and, under McICA, the solves of its
  // subcolumns with their blending weights (mcica_sample.F90:453-925).
  __device__ static __forceinline__ void gpoint(const FluxParams &p, const Sm &S, int col, int g, int bstart, float sec0,
                                                int r, float2 *acc2, float *accd, float *anc, float4 *buf,
                                                bool active) {
    const GPoint &gp = p.gpoints[g];
    const int b = gp.band, bi = b - bstart;
    const BandInfo &bd = p.bands[b];
    const float *bs = S.bscal + bi * kBandScal;
    // a group without a g-point solves one with no weight
    const float w_g = active ? bs[5] * gp.weight_f : 0.0f;
    const size_t row = (size_t)bi * LP;
    typename Solve::Band bnd;
    bnd.opt = S.opt + row;
    bnd.copt = MCICA ? S.copt + row * p.n_condensed : nullptr;
    bnd.cs = nullptr;
    bnd.tkd = (!kLw && p.i_direct_tau == SOCGPU_IP_DIRECT_NOSCALING) ? S.tkd + row : nullptr;
    bnd.fm1 = (!kLw && p.keqv) ? S.aux + row * p.max_abs : nullptr;
    bnd.dB = S.dB + row;
    bnd.dB2 = S.dB2 + row;
    if (single_gas(p, bd)) {
      bnd.kg = nullptr;
      bnd.k0 = gp.kf[0];
    } else if (!p.l_gas || gp.n_abs == 0) {
      bnd.kg = nullptr;
      bnd.k0 = 0.0f;
    } else {
      // into the group's row (the lane's own slots)
      float kg[CH];
      FK::gas_k_lane(p, S, FK::load_gas(gp, bd, p.max_abs), gp, bd, S.amt + row * p.max_abs, r, p.n_layer, kg);
#pragma unroll
      for (int j = 0; j < CH; ++j) S.scr[j * P + r] = kg[j];
      bnd.kg = S.scr;
      bnd.k0 = 0.0f;
    }
    if constexpr (!MCICA) {
      Solve::solve(p, S, bnd, r, sec0, bs, w_g, acc2, accd, anc, nullptr);
    } else {
      const int iex = gp.iex_major;
      const int first = __ldg(p.first_subcol_k + b + (size_t)p.nd_band_sp * iex);
      const int last = __ldg(p.first_subcol_k + b + (size_t)p.nd_band_sp * (iex + 1)) - 1;
      const int nsub = __ldg(p.subcol_k + b + (size_t)p.nd_band_sp * iex);
      const float fcl = load_in<float>(p.frac_cloudy + col);
      const int ncld = p.n_subcol_cld ? __ldg(p.n_subcol_cld + col) : 0;
      const int nfill = min(p.n_subcol_req, p.n_subcol_gen);
      const float w_sub = w_g * fcl / (float)(nsub > 0 ? nsub : 1), w_clr = w_g * (1.0f - fcl);
      // one loop over the clear solve (it = 0) and the subcolumns, so that
      // the solve's code appears once; every group of the warp takes part in
      // each round.  A clear or an overcast column skips the solves that
      // carry no weight (the fraction is the column's, so the whole warp does).
      const int n_iter = last - first + 2;
      const int n_iter_warp = __reduce_max_sync(0xffffffffu, n_iter);
      for (int it = fcl == 1.0f ? 1 : 0; it < (fcl == 0.0f ? 1 : n_iter_warp); ++it) {
        float w = it == 0 ? w_clr : w_sub;
        bnd.cs = nullptr;
        if (it > 0) {
          int idx = (it < n_iter ? first + it - 1 : first) % p.n_subcol_req;
          if (idx == 0) idx = p.n_subcol_req;
          int j = __ldg(p.subcol_reorder + (idx - 1));
          if (p.n_subcol_cld && ncld > 0 && j > ncld && j <= nfill) j = (j - 1) % ncld + 1;
          if (it >= n_iter) w = 0.0f;
          if (j < 1 || j > p.n_subcol_gen) {   // out-of-range table entry: report, no weight
            if (p.error_flag) atomicOr(p.error_flag, 1);
            j = 1;
            w = 0.0f;
          }
          bnd.cs = S.csub + (size_t)(j - 1) * LP;
        }
        Solve::solve(p, S, bnd, r, sec0, bs, w, acc2, accd, anc, buf);
      }
    }
  }

  // The columns' outputs from the groups' accumulators: sums in group order,
  // the downward flux at every level, and the stores, adjacent columns together.
  //
  // The downward flux is known at the tops of the lanes' chunks and at the
  // surface.  Between, its step from one of these is that of the upward flux
  // plus the divergences between, from the anchor above or the one below,
  // whichever leaves the smaller rounding: under thick cloud the flux below it
  // is a small rest of the one above, and a sum from the column's top was off
  // by more than all of it (overcast, 137 layers, 1.8e-5 W/m2 at the surface:
  // -3.6e-3).
  __device__ static void finish(const FluxParams &p, unsigned char *base, int col0, int nc) {
    const TauLayout &l = p.tau;
    const int L = p.n_layer, C = l.cols, n_groups = l.warps * 32 / P;
    const size_t ndp = p.nd_profile;
    // the staged depths are consumed: their space holds the column's sums, up
    // [0, L], down [0, L] (without scattering), divergence [0, L), anchors [0, P]
    auto up_of = [&](int c) { return (float *)(base + (size_t)c * l.stride + l.opt); };
    const int n1 = L + 1;
    for (int q = threadIdx.x; q < C * n1; q += blockDim.x) {
      const int c = q & (C - 1), lev = q / C;
      if (c >= nc) continue;
      unsigned char *b = base + (size_t)c * l.stride;
      float2 *acc2 = (float2 *)(b + l.acc2);
      const float *accd = (const float *)(b + l.accd);
      const int s = FK::level_slot(lev);
      // the rounding of the upward sum is kept: the downward flux is formed
      // from it, and may be far smaller
      float u = 0.0f, u_lo = 0.0f, d = 0.0f, dir = 0.0f;
      for (int k = 0; k < n_groups; ++k) {
        const float2 v = acc2[k * l.acc_stride + s];
        const float t = __fadd_rn(u, v.x), z = __fadd_rn(t, -u);
        u_lo += __fadd_rn(__fadd_rn(u, -__fadd_rn(t, -z)), __fadd_rn(v.x, -z));
        u = t;
        d += v.y;
        if (kThird) dir += accd[k * l.accd_stride + s];
      }
      if (!NOSCAT) acc2[s].x = u_lo;
      float *up = up_of(c);
      up[lev] = u;
      if (lev > 0) up[2 * n1 + lev - 1] = d;      // a layer's divergence is at its bottom level
      if (NOSCAT) up[n1 + lev] = dir;             // the downward flux
      if (p.flux_direct) p.flux_direct[(size_t)(col0 + c) + ndp * lev] = kLw ? 0.0 : widen(dir);
    }
    // the anchors, by the last threads: compensated but for the top's, which
    // is the direct flux's sum bit for bit (the diffuse flux is zero there)
    for (int q = blockDim.x - 1 - threadIdx.x; !NOSCAT && q < C * (P + 1); q += blockDim.x) {
      const int c = q & (C - 1), a = q / C;
      if (c >= nc) continue;
      const float *anc = (const float *)(base + (size_t)c * l.stride + l.anc);
      float d = 0.0f, lo = 0.0f;
      for (int k = 0; k < n_groups; ++k) {
        const float v = anc[k * (P + 1) + a], t = __fadd_rn(d, v), z = __fadd_rn(t, -d);
        lo += __fadd_rn(__fadd_rn(d, -__fadd_rn(t, -z)), __fadd_rn(v, -z));
        d = t;
      }
      up_of(c)[2 * n1 + L + a] = a == 0 ? d : d + lo;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < C * n1; q += blockDim.x) {
      const int c = q & (C - 1), lev = q / C;
      if (c >= nc) continue;
      const unsigned char *b = base + (size_t)c * l.stride;
      const float *up = up_of(c), *div = up + 2 * n1;
      const size_t o = (size_t)(col0 + c) + ndp * lev;
      const float pl = kLw ? ((const float *)(b + l.pl))[FK::level_slot(lev)] : 0.0f, u = up[lev];
      float u_lo = 0.0f, down;
      if constexpr (NOSCAT) {
        down = up[n1 + lev];
      } else {
        const float2 *acc2 = (const float2 *)(b + l.acc2);
        const float *anc = div + L;
        auto lo_of = [&](int i) { return acc2[FK::level_slot(i)].x; };
        u_lo = lo_of(lev);
        const int r = lev / CH, i0 = r * CH, i1 = min(i0 + CH, L);
        if (lev == L) {
          down = anc[P];
        } else {
          const float d0 = anc[r], d1 = anc[i1 == L ? P : r + 1];
          float s0 = 0.0f, a0 = fabsf(d0), s1 = 0.0f, a1 = fabsf(d1);
          for (int i = i0; i < lev; ++i) { s0 += div[i]; a0 += fabsf(div[i]); }
          for (int i = lev; i < i1; ++i) { s1 += div[i]; a1 += fabsf(div[i]); }
          down = (lev == i0 || !(a1 < a0)) ? d0 + ((u - up[i0]) + ((u_lo - lo_of(i0)) - s0))
                                           : d1 + ((u - up[i1]) + ((u_lo - lo_of(i1)) + s1));
        }
      }
      p.flux_up[o] = widen(u + (pl + u_lo));
      p.flux_down[o] = widen(down + pl);
      if (lev < L) {
        const float d = div[lev];
        if (p.flux_div) p.flux_div[o] = widen(d);
        // heating rate (l_run_cdf.F90:1340-1380)
        if (p.heating_rate)
          p.heating_rate[o] = widen(8.64e4f * d / (((const float *)(b + l.mass))[FK::slot(lev)] * 1.005e3f));
      }
    }
  }

  // Columns unit * cols .. of batch p.
  __device__ static void run(const FluxParams &p, int unit) {
    extern __shared__ __align__(128) unsigned char smem[];
    const TauLayout &l = p.tau;
    const int C = l.cols, col0 = unit * C, nc = min(C, p.n_profile - col0);
    const int nb_all = p.last_band - p.first_band + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane % P;
    // the column of this warp and its place among the column's groups
    const int c = warp & (C - 1), wi = warp / C, gw = 32 / P, gi = wi * gw + lane / P, n_groups = l.warps * gw;
    const Sm S = bind(smem, l, c, gi);
    const int col = col0 + min(c, nc - 1);
    const float sec0 = (!kLw && p.zen_0) ? in_col(p.zen_0 + col) : 1.0f;
    BandLite *lite = (BandLite *)(smem + (size_t)C * l.stride);
    // the warp's cells (McICA), this lane's
    float4 *buf = (float4 *)(lite + l.nbat) + warp * (Solve::kBlock * 48) + lane;
    float2 *acc2 = S.acc2 + (size_t)gi * l.acc_stride;
    float *accd = S.accd + (size_t)gi * l.accd_stride, *anc = S.anc + (size_t)gi * (P + 1);
    if (!NOSCAT)
      for (int q = wi * 32 + lane; q < n_groups * (P + 1); q += l.warps * 32) S.anc[q] = 0.0f;
    for (int q = wi * 32 + lane; q < n_groups * l.acc_stride; q += l.warps * 32) S.acc2[q] = make_float2(0.0f, 0.0f);
    if (kThird)
      for (int q = wi * 32 + lane; q < n_groups * l.accd_stride; q += l.warps * 32) S.accd[q] = 0.0f;
    if (kLw)
      for (int q = wi * 32 + lane; q <= LP; q += l.warps * 32) S.pl[q] = 0.0f;

    for (int bb = 0; bb < nb_all; bb += l.nbat) {
      const int nb = min(l.nbat, nb_all - bb), bstart = p.first_band - 1 + bb;
      for (int q = threadIdx.x; q < nb * (int)(sizeof(BandLite) / 4); q += blockDim.x)
        ((int *)lite)[q] = __ldg((const int *)(p.lite + bstart) + q);
      __syncthreads();
      stage(p, smem, lite, col0, nc, bstart, nb, bb == 0);
      stage_boundary(p, smem, lite, col0, nc, bstart, nb);
      __syncthreads();
      if (p.keqv) {
        if (c < nc) {
          const unsigned gm = (P == 32) ? 0xffffffffu : (((1u << P) - 1u) << (lane & ~(P - 1)));
          int item = 0;
          for (int bi = 0; bi < nb; ++bi) {
            const int na = p.l_gas ? min(p.bands[bstart + bi].n_abs, p.max_abs) : 0;
            for (int j = 1; j < na; ++j, ++item)
              if (item % n_groups == gi) FK::minor_gas(p, S, bi, bstart + bi, j, sec0, r, gm);
          }
        }
        __syncthreads();
        if (c < nc) fold_keqv(p, S, bstart, nb, sec0, wi * 32 + lane, l.warps * 32);
        __syncthreads();
      }
      const int g_lo = p.bands[bstart].g_first;
      const int g_hi = p.bands[bstart + nb - 1].g_first + p.bands[bstart + nb - 1].g_count;
      if (c < nc) {
        // every group of the warp runs each of its rounds, so that the
        // full-warp shuffles see all lanes
        for (int g0 = g_lo + wi * gw; g0 < g_hi; g0 += n_groups) {
          const int g = g0 + lane / P;
          gpoint(p, S, col, g < g_hi ? g : g_lo, bstart, sec0, r, acc2, accd, anc, buf, g < g_hi);
        }
        if (kLw) {
          // the band Planck fluxes of adjust_ir_radiance.F90:75-95
          for (int s = wi * 32 + lane; s <= LP; s += l.warps * 32) {
            const int lev = (s == LP) ? 0 : FK::layer_of_slot(s) + 1;
            if (lev > p.n_layer) continue;
            float add = S.pl[s];
            for (int bi = 0; bi < nb; ++bi) add = fmaf(S.planck[bi * (LP + 1) + s], S.bscal[bi * kBandScal + 5], add);
            S.pl[s] = add;
          }
        }
      }
      __syncthreads();
    }
    finish(p, smem, col0, nc);
  }
};

// Resident CTAs of 8 warps asked of the register allocator: 16 warps per SM (128
// registers) for chunks up to 13 layers, 8 above.  More for the short chunks
// did not pay under McICA: at 24 and 32 resident warps (80 and 64 registers)
// solar McICA 8000 x 85 takes 1399 and 1373 us instead of 1253.
constexpr int tau_min_ctas(int ch) { return ch <= 13 ? 2 : 1; }
// The most that a shape is built for beside that, for columns that have a CTA
// to themselves (tau_choose, tau_narrow): the built-in tiles with short
// chunks, whose few layers leave most of a CTA waiting.  With four and five
// layers on 32 lanes it did not pay (GA9 short wave 100 x 304 62 us at two CTAs,
// 64 at three; 137 x 608 143 and 150).
constexpr int tau_dense_ctas(int P, int ch, bool mcica) {
  if (mcica) return tau_min_ctas(ch);
  return P == 16 && ch == 3 ? 4 : (P == 16 && ch == 4) || (P == 32 && ch == 3) || (P == 8 && ch == 5) ? 3 : tau_min_ctas(ch);
}

template <int P, int CH, bool NOSCAT, bool MCICA, int SRC, int MB>
__global__ void __launch_bounds__(256, MB) tau_kernel(const __grid_constant__ FluxParams p) {
  TauKernel<P, CH, NOSCAT, MCICA, SRC>::run(p, blockIdx.x);
}

// Persistent form over many batches (flux_kernel_batched): the work indices
// count groups of tau.cols columns.
template <int P, int CH, bool NOSCAT, bool MCICA, int SRC, int MB>
__global__ void __launch_bounds__(256, MB)
tau_kernel_batched(const FluxParams *__restrict__ items, const long long *__restrict__ col_start, int n_items,
                   long long total) {
  __shared__ __align__(16) FluxParams sp;
  __shared__ int s_item;
  int cur = -1;
  for (long long w = blockIdx.x; w < total; w += gridDim.x) {
    if (threadIdx.x == 0) {
      int lo = 0, hi = n_items - 1;   // last batch whose first index is <= w
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (col_start[mid] <= w) lo = mid; else hi = mid - 1;
      }
      s_item = lo;
    }
    __syncthreads();
    const int it = s_item;
    if (it != cur) {
      const int *src = reinterpret_cast<const int *>(items + it);
      int *dst = reinterpret_cast<int *>(&sp);
      for (int q = threadIdx.x; q < (int)(sizeof(FluxParams) / 4); q += blockDim.x) dst[q] = src[q];
      cur = it;
    }
    __syncthreads();
    TauKernel<P, CH, NOSCAT, MCICA, SRC>::run(sp, (int)(w - col_start[it]));
    __syncthreads();
  }
}

}  // namespace socgpu
