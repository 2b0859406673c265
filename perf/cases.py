"""Work that users of socgpu have it do, for timing and for comparing outputs.

Every case goes through a public entry point: socgpu_radiance_calc_device (DeviceCase.run) on arrays that
stay on the GPU, socgpu_radiance_calc (radiance_calc) on host arrays, a graph of many requests (Batch.run), or
socgpu_cloud_gen_device.  The kinds:

  sw           solar, PIFM80 with delta-rescaling, Rayleigh and modal aerosol, 48 g-points: what a model calls for
               a segment of sunlit columns, and the workload of bench.py
  lw           infra-red without scattering, 81 g-points: the plain long-wave call
  lw_scat      infra-red with scattering by aerosol, 81 g-points: the defaults of `runes` for the long wave
  sw_mcica, lw_mcica   all-sky columns with 16 McICA subcolumns and single sampling: the usual way to treat clouds
  sw_region    a clear and a cloudy region with maximum overlap (Hogan's solver): the other cloud scheme
  sw_ga9       the operational GA9 short-wave file: lookup tables, equivalent extinction, continuum
  host_sw      the call a Fortran model makes, on pageable host arrays, in FP64
  batch        many uneven requests of all kinds and layer counts, as a server's wave or a replayed graph
  cloud_gen    the McICA subcolumn generator, Philox, exponential-random overlap

Sizes run from a physics segment of a few columns (latency) to a whole domain on one GPU, and layer counts over those
of operational models (38 to 137).
"""
from __future__ import annotations

import ctypes as C
import math
from dataclasses import replace
from pathlib import Path

import numpy as np
import torch

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase
from socrates_gb300.spectrum import Spectrum

GA9 = Path(__file__).resolve().parent.parent / "tests" / "golden" / "runes_ga9.npz"
N_SUBCOL = 16
FIELDS = ("flux_up", "flux_down", "flux_direct", "flux_div", "heating_rate")
LAYERS = (38, 60, 85, 137)
REQUEST_KINDS = ("lw", "sw", "lw_mcica", "sw_mcica")
# the most columns drawn for each kind, so that no drawn case costs more than the largest listed one
MOST = {"sw": 10000, "lw": 20000, "lw_scat": 6000, "sw_mcica": 8000, "lw_mcica": 6000, "sw_region": 2048, "sw_ga9": 4000,
        "host_sw": 2000, "batch": 96, "cloud_gen": 16384}


def listed():
    return [
        # a physics segment of a few sunlit columns: launches and latency count
        dict(name="sw_segment_27x38", kind="sw", n=27, layers=38, precision="mixed"),
        # a rank's clear-sky long wave
        dict(name="lw_1000x60", kind="lw", n=1000, layers=60, precision="mixed"),
        # the headline workload: sunlit columns of a domain
        dict(name="sw_10000x100", kind="sw", n=10000, layers=100, precision="mixed"),
        # long wave with scattering at the layer count of a global forecast model, an odd number of columns
        dict(name="lw_scat_3001x137", kind="lw_scat", n=3001, layers=137, precision="mixed"),
        # the FP64 path, for models that want the reference's digits
        dict(name="sw_fp64_1500x85", kind="sw", n=1500, layers=85, precision="fp64"),
        # all-sky columns, both sources
        dict(name="sw_mcica_8000x85", kind="sw_mcica", n=8000, layers=85, precision="mixed"),
        dict(name="lw_mcica_6000x85", kind="lw_mcica", n=6000, layers=85, precision="mixed"),
        # two cloud regions
        dict(name="sw_region_1025x70", kind="sw_region", n=1025, layers=70, precision="mixed"),
        # the operational short-wave file
        dict(name="sw_ga9_2000x70", kind="sw_ga9", n=2000, layers=70, precision="mixed"),
        # the whole call of a Fortran model on its own arrays
        dict(name="host_sw_500x60", kind="host_sw", n=500, layers=60, precision="fp64"),
        # a wave of uneven requests
        dict(name="batch_64", kind="batch", n=64, layers=0, precision="mixed"),
        # subcolumns for a domain
        dict(name="cloud_gen_8192x85", kind="cloud_gen", n=8192, layers=85, precision="fp64"),
    ]


def draw(rng):
    kind = rng.choice(tuple(MOST))
    lo = 16 if kind == "batch" else 1
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(MOST[kind])))))
    layers = 0 if kind == "batch" else rng.choice(LAYERS + (33, 47, 70, 71, 100, 101))
    precision = "fp64" if kind in ("host_sw", "cloud_gen") else "mixed"
    if kind in ("sw", "lw", "sw_mcica", "lw_mcica") and rng.random() < 0.25:
        precision = "fp64"
        n = max(1, n // 8)
    return dict(kind=kind, n=n, layers=layers, precision=precision)


# ---------------------------------------------------------------------------
# what a program has in hand: the spectral file (read once), the atmosphere, and for all-sky columns their subcolumns
_spectra: dict = {}


def spectrum(kind) -> Spectrum:
    key = "ga9" if kind == "sw_ga9" else kind[:2] if kind[:2] in ("sw", "lw") else "sw"
    key += "_cld" if kind.endswith(("mcica", "region")) else ""
    if key not in _spectra:
        _spectra[key] = (Spectrum.load_npz(GA9, prefix="sw_") if key == "ga9" else
                         synth.sw_spectrum(2, 8, clouds=key.endswith("_cld")) if key.startswith("sw") else
                         synth.lw_spectrum(1, 9, clouds=key.endswith("_cld")))
    return _spectra[key]


def columns(kind, n, layers, seed):
    """(spectrum, column, mcica) of n columns."""
    sp = spectrum(kind)
    if kind == "sw_ga9":
        return sp, synth.operational_case(sp, n, layers, seed=seed, solar=True), None
    col = synth.atmosphere(n, layers, sp.type_absorb, seed)
    if kind.startswith("lw"):
        synth.add_lw_surface(col, sp.n_band)
    else:
        synth.add_sw_surface(col, sp.n_band, seed)
    if kind in ("sw", "lw_scat", "host_sw"):
        synth.add_aerosol(col, sp, seed)
    mc = None
    if kind.endswith(("mcica", "region")):
        synth.add_clouds(col, seed, N_SUBCOL)
    if kind.endswith("mcica"):
        c_sub, n_cld = R.cloud_gen(col, N_SUBCOL, abi.IP_EXPONENTIAL_RAND, abi.RNG_PHILOX)
        isolir = abi.IP_SOLAR if kind.startswith("sw") else abi.IP_INFRA_RED
        mc = R.set_cld_mcica(sp, col, isolir, abi.IP_MCICA_SINGLE_SAMPLING, c_sub=c_sub, n_subcol_cld=n_cld)
    return sp, col, mc


def control(kind, precision) -> R.Control:
    kw = dict(precision=abi.PRECISION_FP64 if precision == "fp64" else abi.PRECISION_MIXED)
    if kind == "lw":
        return R.lw_noscat_control(**kw)
    if kind == "lw_scat":
        return R.lw_control(l_aerosol_mode=True, **kw)
    if kind == "lw_mcica":
        return R.lw_control(i_cloud=abi.IP_CLOUD_MCICA, **kw)
    if kind == "sw_mcica":
        return R.sw_control(i_cloud=abi.IP_CLOUD_MCICA, **kw)
    if kind == "sw_region":
        return R.sw_control(i_cloud=abi.IP_CLOUD_MIX_MAX, i_solver=abi.IP_SOLVER_MIX_DIRECT_HOGAN, **kw)
    if kind == "sw_ga9":
        return R.sw_control(l_continuum=True, i_gas_overlap=abi.IP_OVERLAP_K_EQV_SCL, **kw)
    return R.sw_control(l_aerosol_mode=True, **kw)


class Calls:
    """Problems on the GPU whose outputs lie one after another in one buffer, field by field."""

    def __init__(self, problems):
        self.cases = [self.device_case(*p) for p in problems]
        self.mixed = problems[0][0].precision == abi.PRECISION_MIXED
        sizes = {f: sum(self.size(c, f) for c in self.cases) for f in FIELDS}
        self.fields = [f for f in FIELDS if sizes[f]]
        self.sizes = [sizes[f] for f in self.fields]
        self.out = torch.zeros(sum(self.sizes), dtype=torch.float64, device="cuda")
        at = 0
        for f in self.fields:
            for c in self.cases:
                if self.size(c, f):
                    setattr(c.radout, f, C.cast(C.c_void_p(self.out.data_ptr() + 8 * at), C.POINTER(C.c_double)))
                at += self.size(c, f)

    @staticmethod
    def device_case(ctl, sp, col, mc):
        if ctl.i_cloud != abi.IP_CLOUD_MIX_MAX:
            return DeviceCase(ctl, sp, col, mc)
        # cloud regions take the cloud fields without subcolumns
        no_subcol = R.McicaState(1, 1, None, None, None, None, None, None)
        return DeviceCase(ctl, sp, col, no_subcol)

    @staticmethod
    def size(c, f):
        if f == "flux_direct" and c.control.isolir != abi.IP_SOLAR:
            return 0
        return c.n * (c.L if f in ("flux_div", "heating_rate") else c.L + 1)

    def outputs(self):
        # a model that asks for mixed precision keeps its fluxes in 32 bits, which is what they were computed in
        v = self.out.float() if self.mixed else self.out
        return dict(zip(self.fields, v.split(self.sizes)))


def requests(n):
    """(kind, layers, columns) of n requests: log-normal widths, median 256."""
    rng = np.random.default_rng(4)
    width = np.clip(np.rint(rng.lognormal(np.log(256.0), 1.0, n)), 1, 2048).astype(int)
    return [(REQUEST_KINDS[k], LAYERS[j], int(w))
            for k, j, w in zip(rng.integers(0, 4, n), rng.integers(0, 4, n), width)]


def problems(case, seed):
    if case["kind"] == "batch":
        return [(control(k, case["precision"]), *columns(k, w, j, seed + 7919 * i))
                for i, (k, j, w) in enumerate(requests(case["n"]))]
    return [(control(case["kind"], case["precision"]), *columns(case["kind"], case["n"], case["layers"], seed))]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host_sw":
        ctl, sp, col, _ = problems(case, seed)[0]
        R.register_spectrum(sp)
        return dict(kind=kind, args=(ctl, sp, col))
    if kind == "cloud_gen":
        n, L = case["n"], case["layers"]
        col = synth.atmosphere(n, L, np.array([1, 2, 3], np.int32), seed)
        synth.add_clouds(col, seed, N_SUBCOL)

        def dev(a, dtype=np.float64):
            return torch.from_numpy(np.asarray(a, dtype=dtype).ravel(order="F").copy()).cuda()
        cd = col.cld
        t = [dev(cd["rand_seed"], np.int32), dev(cd["dp_corr_cloud"]), dev(cd["dp_corr_cond"]), dev(np.zeros((n, L))),
             dev(cd["w_cloud"]), dev(np.zeros((n, L))), dev(np.zeros((n, L))), dev(col.p), dev(np.zeros((2, 2)))]
        n_cld = torch.zeros(n, dtype=torch.int32, device="cuda")
        c_sub = torch.zeros(n * L * N_SUBCOL, dtype=torch.float64, device="cuda")
        args = ([L, 1, L, n, 1, n, N_SUBCOL, 2, 2, 0, abi.IP_EXPONENTIAL_RAND] + [x.data_ptr() for x in t]
                + [n_cld.data_ptr(), c_sub.data_ptr(), abi.RNG_PHILOX])
        return dict(kind=kind, lib=R.load_library(), args=args, keep=t, out=dict(n_subcol_cld=n_cld, c_sub=c_sub))
    calls = Calls(problems(case, seed))
    return dict(kind=kind, calls=calls, batch=Batch(calls.cases) if kind == "batch" else None)


def run(state):
    kind = state["kind"]
    if kind == "host_sw":
        return R.radiance_calc(*state["args"])
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "cloud_gen":
        msg = C.create_string_buffer(512)
        st = state["lib"].socgpu_cloud_gen_device(*state["args"], C.c_void_p(stream), msg, 512)
        if st != abi.I_NORMAL:
            raise R.RadianceError(st, msg.value.decode())
        return state["out"]
    calls = state["calls"]
    if state["batch"] is not None:
        state["batch"].run(stream)
    else:
        calls.cases[0].run(stream)
    return calls.outputs()


# FP32 or FP64 operations of one (column, layer, g-point), each exponential, root and division counted once
CELL_FLOPS = {"sw": 80, "lw": 30, "lw_scat": 80, "sw_mcica": 170, "lw_mcica": 170, "sw_region": 250, "sw_ga9": 130}


def work(case):
    """Inputs read once, outputs written once (FP64 arrays), and the arithmetic of every cell."""
    def one(kind, n, L):
        if kind == "cloud_gen":
            return {"bytes": n * L * (8.0 * 4 + 8.0 * N_SUBCOL), "flops": 10.0 * n * L * N_SUBCOL}
        kind = "sw" if kind == "host_sw" else kind
        sp = spectrum(kind)
        nb, solar = sp.n_band, kind.startswith("sw")
        g = 41 if kind == "sw_ga9" else 48 if solar else 81
        per = 3 + (1 if kind == "sw_ga9" else 0) + len(sp.type_absorb)       # p, T, mass, density, gases
        per += (1 + 3 * nb) if kind in ("sw", "lw_scat") else 0              # modal aerosol
        per += 7 if kind.endswith(("mcica", "region")) else 0                # cloud fields
        per += N_SUBCOL if kind.endswith("mcica") else 0
        per += 0 if solar else 1                                             # level temperatures
        out = 5 if solar else 4
        return {"bytes": 8.0 * n * (L * (per + out) + 2 * nb + 4), "flops": float(CELL_FLOPS[kind]) * n * L * g}
    if case["kind"] != "batch":
        return one(case["kind"], case["n"], case["layers"])
    every = [one(k, w, j) for k, j, w in requests(case["n"])]
    return {k: sum(w[k] for w in every) for k in ("bytes", "flops")}


# ---------------------------------------------------------------------------
# The same fluxes in 64 bits by plain torch, vectorised over columns and k-terms and serial over layers: tensors are
# (n, L, K) with K the k-terms of a band (k_eqv_scl and random overlap of one absorber both give one term a g-point).
EPS = 2.220446049250313e-16
SQ_EPS = math.sqrt(EPS)


def exact(case, seed):
    if case["kind"] == "cloud_gen":
        return None                       # masks drawn from integers: compared as they are
    got = [exact_one(k, *p) for k, p in zip([case["kind"]] if case["kind"] != "batch" else
                                            [q[0] for q in requests(case["n"])], problems(case, seed))]
    if case["kind"] == "host_sw":
        return {f: v.cpu().numpy() for f, v in got[0].items()}
    return {f: torch.cat([g[f].T.reshape(-1) for g in got if f in g]) for f in FIELDS if any(f in g for g in got)}


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu", torch.float64)


def two_stream(solar, g, om, tau, sec0):
    """Transmission, reflection, direct transmission and the two source coefficients of each cell (PIFM80 in the
    solar, Elsasser in the infra-red)."""
    if solar:
        total, diff = 2.0 - 1.5 * om * g - 0.5 * om, 2.0 * (1.0 - om)
    else:
        total, diff = 1.66 - 1.5 * om * g, 1.66 * (1.0 - om)
    lam = torch.sqrt(total * diff)
    if solar:
        near = (lam - sec0).abs() < 32 * EPS
        up = torch.where(near, torch.full_like(lam, 1.0 + 32 * EPS), torch.ones_like(lam))
        total, diff, lam = total * up, diff * up, lam * up
        ksi = 1.5 * g / sec0
        factor = 0.5 * om * sec0 / ((lam - sec0) * (lam + sec0))
        g_up = factor * (total - sec0 - ksi * (diff - sec0))
        g_dn = factor * (total + sec0 + ksi * (diff + sec0))
    e = torch.exp(-lam * tau)
    gamma = (total - lam) / (total + lam)
    inv = 1.0 / (1.0 - e * e * gamma * gamma)
    T, Rf = e * (1.0 - gamma * gamma) * inv, gamma * (1.0 - e * e) * inv
    if solar:
        T0 = torch.exp(-tau * sec0)
        return T, Rf, T0, (g_up - Rf * (1.0 + g_dn)) - g_up * T * T0, T0 * (1.0 + g_dn - g_up * Rf) - (1.0 + g_dn) * T
    c1 = (1.0 - T + Rf + SQ_EPS) / (SQ_EPS + tau * total)
    s2 = torch.where(tau > math.sqrt(SQ_EPS), -2.0 * (1.0 - T - Rf + SQ_EPS) / (diff * tau + SQ_EPS), -2.0 + diff * tau)
    return T, Rf, torch.ones_like(T), c1, -(1.0 + Rf + T + s2) / (total * tau + SQ_EPS)


def cell(solar, kgt, kes, kgas, asym, fwd, mass, sec0):
    k = kgt + kgas
    om = torch.clamp(kes / (k + 2.2e-308), max=1.0 - 32 * EPS)
    tau = k * mass * (1.0 - om * fwd)
    om = om * (1.0 - fwd) / (1.0 - om * fwd)
    return two_stream(solar, asym, om, tau, sec0)


def power_quad(sc, p, t, p_ref, t_ref):
    x = t / t_ref - 1.0
    return (p / p_ref) ** sc[0] * (1.0 + x * sc[1] + sc[2] * x * x)


def lookup_factors(sp, p, t):
    """Bilinear weights and indices of every cell in the (ln p, T) grid of the lookup tables."""
    lp, tt = _dev(sp.p_lookup), _dev(sp.t_lookup)                   # (n_pre), (n_tmp, n_pre)

    def shrink(lo, hi):
        return lo + torch.clamp(lo.abs() * EPS, min=EPS), hi - torch.clamp(hi.abs() * EPS, min=EPS)
    lo, hi = shrink(lp[0], lp[-1])
    x = torch.log(p).clamp(lo, hi)
    jp = torch.clamp(torch.searchsorted(lp, x.contiguous(), right=True) - 1, 0, len(lp) - 2)
    fp = (x - lp[jp]) / (lp[jp + 1] - lp[jp])

    def in_t(j):
        grid = tt.T[j]                                              # (n, L, n_tmp)
        y = torch.minimum(torch.maximum(t, grid[..., 0] * (1.0 + EPS)), grid[..., -1] * (1.0 - EPS))
        i = torch.clamp((grid <= y[..., None]).sum(-1) - 1, 0, grid.shape[-1] - 2)
        a, b = grid.gather(-1, i[..., None])[..., 0], grid.gather(-1, i[..., None] + 1)[..., 0]
        return i, (y - a) / (b - a)
    (jt, ft), (jtt, ftt) = in_t(jp), in_t(jp + 1)
    return [((1 - fp) * (1 - ft), jt, jp), (fp * (1 - ftt), jtt, jp + 1), ((1 - fp) * ft, jt + 1, jp),
            (fp * ftt, jtt + 1, jp + 1)]


def terms(sp, b, s, p, t, q, factors):
    """k times the mixing ratio q of every k-term of species s (0-based) in band b: (n, L, K)."""
    nk, fnc = int(sp.i_band_k[b, s]), int(sp.i_scale_fnc[b, s])
    pr, tr = float(sp.p_ref[s, b]), float(sp.t_ref[s, b])
    out = []
    for k in range(nk):
        sc, kv = sp.scale[:, k, b, s], float(sp.k[k, b, s])
        if fnc == 1:                                                # power law
            out.append(kv * ((p / pr) ** sc[0] * (t / tr) ** sc[1] * q).clamp(min=0.0))
        elif fnc == 2:                                              # power law in p, quadratic in T
            out.append(kv * (power_quad(sc, p, t, pr, tr) * q).clamp(min=0.0))
        elif fnc == 9:                                              # lookup table in ln p and T
            tab = _dev(sp.k_lookup[:, :, k, s, b])
            out.append(sum(f * tab[i, j] for f, i, j in factors).clamp(min=0.0) * q)
        else:
            raise ValueError("no 64-bit form of scaling function %d" % fnc)
    return torch.stack(out, -1)


def pade(c, re, qm):
    kext = qm * (c[0] + re * (c[1] + re * c[2])) / (1.0 + re * (c[3] + re * (c[4] + re * c[5])))
    co = (c[6] + re * (c[7] + re * c[8])) / (1.0 + re * (c[9] + re * c[10]))
    g = (c[11] + re * (c[12] + re * c[13])) / (1.0 + re * (c[14] + re * c[15]))
    ks = kext * (1.0 - co)
    return kext, ks, ks * g, ks * g * g


def planck(c, x):
    f = torch.zeros_like(x)
    for a in c[::-1]:
        f = f * x + float(a)
    return f


def adding(T, Rf, su, sd, inc, ground, alb):
    """The adding equations, bottom up then top down: fluxes up and down (n, L + 1, K)."""
    L = T.shape[1]
    a, s, rows = alb.expand_as(ground), ground, [None] * L
    for i in range(L - 1, -1, -1):
        beta = 1.0 / (1.0 - a * Rf[:, i])
        h = s + a * sd[:, i]
        rows[i] = (beta, a * T[:, i], h)
        a, s = Rf[:, i] + beta * rows[i][1] * T[:, i], su[:, i] + beta * T[:, i] * h
    up, dn = [a * inc + s], [inc.expand_as(s)]
    for i in range(L):
        beta, gam, h = rows[i]
        up.append(beta * (h + gam * dn[i]))
        dn.append(sd[:, i] + T[:, i] * dn[i] + Rf[:, i] * up[i + 1])
    return torch.stack(up, 1), torch.stack(dn, 1)


def no_scatter(T, su, sd, inc, d_surf, alb):
    L = T.shape[1]
    dn = [inc.expand_as(T[:, 0])]
    for i in range(L):
        dn.append(sd[:, i] + T[:, i] * dn[i])
    up = [None] * L + [(1.0 - alb) * d_surf + alb * dn[L]]
    for i in range(L - 1, -1, -1):
        up[i] = su[:, i] + T[:, i] * up[i + 1]
    return torch.stack(up, 1), torch.stack(dn, 1)


def beam(T0, inc):
    fd = [inc.expand_as(T0[:, 0])]
    for i in range(T0.shape[1]):
        fd.append(fd[i] * T0[:, i])
    return torch.stack(fd, 1)


def overlap(w):
    """Maximum overlap of a clear and a cloudy region: v[i][j][k], the share of upper region k over lower region j at
    interface i, and u[i][j][k], the share of lower region k under upper region j."""
    n, L = w.shape
    one, zero, tol = torch.ones(n, 1, dtype=w.dtype, device=w.device), torch.zeros(n, 1, dtype=w.dtype, device=w.device), 100 * EPS
    above, v, u = (one, zero), [], []
    for i in range(L + 1):
        below = (1.0 - w[:, i:i + 1], w[:, i:i + 1]) if i < L else (one, zero)
        o = [[torch.minimum(above[k], below[k]) if k == j else zero for j in range(2)] for k in range(2)]
        rest = 1.0 - o[0][0] - o[1][1]
        ru, rl = [above[k] - o[k][k] for k in range(2)], [below[k] - o[k][k] for k in range(2)]
        for k in range(2):
            for j in range(2):
                o[k][j] = torch.where(rest > tol, o[k][j] + ru[k] * rl[j] / rest.clamp(min=tol), o[k][j])
        eye = lambda j, k: one if j == k else zero  # noqa: E731
        v.append([[torch.where(above[k] > tol, o[k][j] / above[k].clamp(min=tol), eye(j, k)) for k in range(2)] for j in range(2)])
        u.append([[torch.where(below[k] > tol, o[j][k] / below[k].clamp(min=tol), eye(j, k)) for k in range(2)] for j in range(2)])
        above = below if i < L else above
    return v, u


def two_regions(clear, cloud, v, u, inc, alb, alb_dir):
    """Hogan's solver for a clear and a cloudy region under the solar source: up, down, direct (n, L + 1, K)."""
    (T, Rf, T0, c1, c2), (Tc, Rc, T0c, c1c, c2c) = clear, cloud
    L = T.shape[1]
    bf, bc = inc.expand_as(T[:, 0]), torch.zeros_like(T[:, 0])
    direct, src = [bf], []
    for i in range(L):
        tc, tf = v[i][1][1] * bc + v[i][1][0] * bf, v[i][0][0] * bf + v[i][0][1] * bc
        src.append((c1[:, i] * tf, c2[:, i] * tf, c1c[:, i] * tc, c2c[:, i] * tc))
        bf, bc = tf * T0[:, i], tc * T0c[:, i]
        direct.append(bf + bc)
    a1 = a2 = alb.expand_as(bf)
    g1, g2 = (alb_dir - alb) * bf, (alb_dir - alb) * bc
    rows = [None] * L
    for i in range(L - 1, -1, -1):
        su, sd, suc, sdc = src[i]
        t1, t2 = a1 * v[i + 1][0][0] + a2 * v[i + 1][1][0], a1 * v[i + 1][0][1] + a2 * v[i + 1][1][1]
        b1, h1 = 1.0 / (1.0 - t1 * Rf[:, i]), g1 + t1 * sd
        b2, h2 = 1.0 / (1.0 - t2 * Rc[:, i]), g2 + t2 * sdc
        rows[i] = (b1, t1 * T[:, i], h1, b2, t2 * Tc[:, i], h2)
        l1, l2 = su + h1 * T[:, i] * b1, suc + h2 * Tc[:, i] * b2
        a1, a2 = Rf[:, i] + t1 * T[:, i] ** 2 * b1, Rc[:, i] + t2 * Tc[:, i] ** 2 * b2
        g1, g2 = u[i][0][0] * l1 + u[i][0][1] * l2, u[i][1][0] * l1 + u[i][1][1] * l2
    up, dn = [g1 + inc * (v[0][0][0] * a1 + v[0][1][0] * a2)], [inc.expand_as(bf)]
    d1, d2 = inc.expand_as(bf), torch.zeros_like(bf)
    for i in range(L):
        d1, d2 = v[i][0][0] * d1 + v[i][0][1] * d2, v[i][1][0] * d1 + v[i][1][1] * d2
        b1, gm1, h1, b2, gm2, h2 = rows[i]
        f1, f2 = (gm1 * d1 + h1) * b1, (gm2 * d2 + h2) * b2
        _, sd, _, sdc = src[i]
        d1, d2 = T[:, i] * d1 + Rf[:, i] * f1 + sd, Tc[:, i] * d2 + Rc[:, i] * f2 + sdc
        up.append(f1 + f2)
        dn.append(d1 + d2)
    return torch.stack(up, 1), torch.stack(dn, 1), torch.stack(direct, 1)


def exact_one(kind, ctl, sp, col, mc):
    """The outputs of one problem, columns in slices that fit the memory comfortably."""
    step = max(1, 40_000_000 // (col.n_layer * 17))
    parts = [exact_slice(kind, ctl, sp, col, mc, slice(a, min(a + step, col.n_profile)))
             for a in range(0, col.n_profile, step)]
    return {f: torch.cat([p[f] for p in parts]) for f in parts[0]}


def exact_slice(kind, ctl, sp, col, mc, sl):
    solar, noscat = kind[:2] != "lw", kind == "lw"
    p, t, mass, gas = (_dev(a[sl]) for a in (col.p, col.t, col.mass, col.gas_mix_ratio))
    n, L = p.shape
    m3 = mass[..., None]
    sec0 = _dev(col.zen_0[sl])[:, None, None] if solar else 1.0
    factors = lookup_factors(sp, p, t) if kind == "sw_ga9" else None
    up, dn, direct = (torch.zeros(n, L + 1, dtype=p.dtype, device=p.device) for _ in range(3))
    div = torch.zeros_like(p)
    cd = col.cld
    if cd:
        wc, frac = _dev(cd["w_cloud"][sl]), _dev(cd["frac_cloud"][sl])
        cmr, cdim = _dev(cd["condensed_mix_ratio"][sl]), _dev(cd["condensed_dim_char"][sl])
        v, u = overlap(wc) if kind == "sw_region" else (None, None)
    for b in range(sp.n_band):
        alb, alb_dir = _dev(col.rho_alb[sl, 0, b])[:, None], _dev(col.rho_alb[sl, 1, b])[:, None]
        # grey optics
        kes = torch.full_like(p, float(sp.rayleigh_coeff[b])) if ctl.l_rayleigh else torch.zeros_like(p)
        kab, phf, fwd = torch.zeros_like(p), torch.zeros_like(p), torch.zeros_like(p)
        if ctl.l_aerosol_mode:
            q = _dev(col.aer["mode_mix_ratio"][sl, :, 0])
            ka, ks, g = (_dev(col.aer["mode_" + f][sl, :, 0, b]) for f in ("absorption", "scattering", "asymmetry"))
            kab, kes, phf, fwd = kab + q * ka, kes + q * ks, q * ks * g, q * ks * g * g
        if ctl.l_continuum:
            rho, water = _dev(col.density[sl]), gas[..., int(sp.index_water) - 1]
            for j in range(int(sp.n_band_continuum[b])):
                sc, kc = sp.scale_cont[:, b, j], int(sp.index_continuum[b, j])
                pr, tr = float(sp.p_ref_cont[j, b]), float(sp.t_ref_cont[j, b])
                a = ((p / pr) ** sc[0] * (t / tr) ** sc[1]) if int(sp.i_scale_fnc_cont[b, j]) == 1 else power_quad(sc, p, t, pr, tr)
                a = a * rho * water * (water / 18.0153e-03 if kc == 1 else (1.0 - water) / 28.966e-03)
                kab = kab + float(sp.k_cont[b, j]) * a
        # gases: the major absorber's terms, and the minor ones' equivalent extinction
        spec = [int(sp.index_absorb[j, b]) - 1 for j in range(int(sp.n_band_absorb[b]))]
        kgas = terms(sp, b, spec[0], p, t, gas[..., spec[0]], factors)
        weight = _dev(sp.w[:kgas.shape[-1], b, spec[0]])
        adj = None
        if ctl.i_gas_overlap == abi.IP_OVERLAP_K_EQV_SCL:
            adj, k_eqv = torch.ones_like(p), torch.zeros_like(p)
            for s in spec[1:]:
                kk = terms(sp, b, s, p, t, gas[..., s], factors)
                f = torch.cumprod(torch.exp(-kk * m3 * sec0), 1) * _dev(sp.w[:kk.shape[-1], b, s])
                surf, f = f[:, -1:], f.sum(-1)
                k_eqv = k_eqv + torch.where(surf.sum(-1) > 0, (kk * surf).sum(-1) / surf.sum(-1).clamp(min=1e-300), kk.amin(-1))
                prev = torch.cat([torch.ones_like(f[:, :1]), f[:, :-1]], 1)
                adj = adj * torch.where(prev > 0, f / prev.clamp(min=1e-300), torch.ones_like(f))
            adj = (adj * torch.exp((k_eqv * mass * sec0[:, 0]).clamp(max=math.log(1.0 / EPS))))[..., None]
            kab = kab + k_eqv
        kgt = kab + kes
        safe = kes.clamp(min=1e-300)
        f_n, a_n = torch.where(kes > 0, fwd / safe, fwd), torch.where(kes > 0, phf / safe, phf)
        a_n = (a_n - f_n) / (1.0 - f_n)
        # boundary values and the Planck source
        if solar:
            inc = (_dev(col.solar_irrad[sl])[:, None] * float(sp.solar_flux_band[b])) / sec0[:, 0]
        else:
            c, tr = sp.thermal_coeff[:, b], float(sp.t_ref_planck)
            B = planck(c, _dev(col.t_level[sl]) / tr)
            dB, dB2 = (B[:, 1:] - B[:, :-1])[..., None], (2.0 * (B[:, 1:] + B[:, :-1] - 2.0 * planck(c, t / tr)))[..., None]
            inc = -B[:, :1]
            d_surf = (planck(c, _dev(col.t_ground[sl]) / tr) - B[:, -1])[:, None]

        def solve(T, Rf, T0, c1, c2):
            if solar:
                if adj is not None:
                    c2, T0 = c2 - T0 + T0 * adj, T0 * adj
                fd = beam(T0, inc)
                su, sd, ground = c1 * fd[:, :-1], c2 * fd[:, :-1], (alb_dir - alb) * fd[:, -1]
                return (*adding(T, Rf, su, sd, inc, ground, alb), fd)
            su, sd = c1 * dB + c2 * dB2, -c1 * dB + c2 * dB2
            if noscat:
                return (*no_scatter(T, su, sd, inc, d_surf, alb), None)
            return (*adding(T, Rf, su, sd, inc, ((1.0 - alb) * d_surf).expand_as(T[:, 0]), alb), None)

        def grey(x):
            return x[..., None]
        if noscat:
            tau = kgas * m3 + grey(kab) * m3
            T = torch.exp(-1.66 * tau)
            c1 = (1.0 - T + SQ_EPS) / (1.66 * tau + SQ_EPS)
            c2 = -torch.where(tau > math.sqrt(SQ_EPS), 1.0 + T - 2.0 * c1, T - 1.0 + 1.66 * tau) / (1.66 * tau + SQ_EPS)
            clear = (T, None, None, c1, c2)
        else:
            clear = cell(solar, grey(kgt), grey(kes), kgas, grey(a_n), grey(f_n), m3, sec0)
        if not cd:
            fu, fd, fdir = solve(*clear)
        else:
            comp = []
            for k, parm in enumerate((sp.drop_parm_list, sp.ice_parm_list)):
                ok = (wc > 0) & (cdim[..., k] > 0)
                comp.append([torch.where(ok, x, torch.zeros_like(x)) for x in pade(parm[:, b, 0], cdim[..., k], cmr[..., k])])

            def cloudy(scale):
                """The types' coefficients weighted by their fractions, each type one component."""
                tot = None
                for k in range(2):
                    ke, ks, ph, fw = ((grey(x) if scale.dim() == 3 else x) * scale for x in comp[k])
                    lift = grey if scale.dim() == 3 else (lambda x: x)
                    ke, ks, ph, fw = ke + lift(kgt), ks + lift(kes), ph + lift(phf), fw + lift(fwd)
                    if scale.dim() == 2:
                        ke, ks, ph, fw = (grey(x) for x in (ke, ks, ph, fw))
                    ok = ks.clamp(min=1e-300)
                    f_c = fw / ok
                    got = cell(solar, ke, ks, kgas, (ph / ok - f_c) / (1.0 - f_c), f_c, m3, sec0)
                    fc = grey(frac[..., k])
                    use = ((scale if scale.dim() == 3 else grey(scale)) * fc > 0) & (grey(wc) > 0)
                    got = [torch.where(use, fc * x, torch.zeros_like(x)) for x in got]
                    tot = got if tot is None else [x + y for x, y in zip(tot, got)]
                return tot
            if kind == "sw_region":
                fu, fd, fdir = two_regions(clear, cloudy(torch.ones_like(p)), v, u, inc, alb, alb_dir)
            else:
                # single sampling: term k takes one subcolumn, those past n_subcol_cld repeating the cloudy ones
                first = mc.first_subcol_k[b, :kgas.shape[-1]]
                order = torch.tensor([int(mc.subcol_reorder[(int(m) - 1) % mc.n_subcol_req]) for m in first], device=p.device)
                n_cld = torch.from_numpy(np.ascontiguousarray(mc.n_subcol_cld[sl])).to(p.device).long()[:, None]
                j = order[None].expand(n, -1)
                fill = (n_cld > 0) & (j > n_cld) & (j <= min(mc.n_subcol_req, mc.n_subcol_gen))
                j = torch.where(fill, (j - 1) % n_cld.clamp(min=1) + 1, j) - 1
                scale = _dev(mc.c_sub[sl]).gather(2, j[:, None, :].expand(n, L, -1))
                wet = ((scale * frac[..., :1] > 0) | (scale * frac[..., 1:2] > 0)) & (grey(wc) > 0)
                mix = [torch.where(wet, x, y) for x, y in zip(cloudy(scale), clear)]
                part = _dev(mc.frac_cloudy[sl])[:, None, None]
                a, c = solve(*mix), solve(*clear)
                fu, fd = (part * x + (1.0 - part) * y for x, y in zip(a[:2], c[:2]))
                fdir = part * a[2] + (1.0 - part) * c[2] if solar else None
        net = fd - fu
        up, dn, div = up + fu @ weight, dn + fd @ weight, div + (net[:, :-1] - net[:, 1:]) @ weight
        if solar:
            direct = direct + fdir @ weight
        else:
            up, dn = up + B, dn + B
    out = dict(flux_up=up, flux_down=dn, flux_div=div, heating_rate=8.64e4 * div / (mass * 1.005e3))
    if solar:
        out["flux_direct"] = direct
    return out
