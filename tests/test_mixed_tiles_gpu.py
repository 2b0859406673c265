"""The mixed kernels at the edges of their tiles and column groups, against
the FP64 oracle: layer counts at and one past every built tile, column counts
about the width from which four columns share a CTA and with one to three
columns in the last group, band ranges, the options that change what is
staged, and a column of NaN beside finite ones.

Tolerance: every layer's step of the solve rounds to FP32, so the fluxes may
differ by a few units in the last place per layer, 4 L 2^-24 of the largest
flux (0.01 W/m2 of 1360 W/m2 over 33 layers, 0.05 over 145); heating rates
stay within the 0.05 K/day of the other mixed tests."""
from dataclasses import replace

import numpy as np
import pytest

import oracle as O
from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase

pytestmark = pytest.mark.gpu


def _case(kind, n, L, seed):
    sp = (synth.sw_spectrum if kind.startswith("sw") else synth.lw_spectrum)(seed, 5, clouds=kind.endswith("mcica"))
    col = synth.atmosphere(n, L, sp.type_absorb, seed)
    if kind.startswith("sw"):
        synth.add_sw_surface(col, sp.n_band, seed)
    else:
        synth.add_lw_surface(col, sp.n_band)
    mc = None
    if kind.endswith("mcica"):
        synth.add_clouds(col, seed, 8)
        isolir = abi.IP_SOLAR if kind.startswith("sw") else abi.IP_INFRA_RED
        mc = R.set_cld_mcica(sp, col, isolir, abi.IP_MCICA_FULL_SAMPLING, rng=abi.RNG_PHILOX)
    elif kind != "lw":
        synth.add_aerosol(col, sp, seed)
    ctl = {"sw": R.sw_control(l_aerosol_mode=True), "lw": R.lw_noscat_control(),
           "lw_scat": R.lw_control(l_aerosol_mode=True), "sw_mcica": R.sw_control(i_cloud=abi.IP_CLOUD_MCICA),
           "lw_mcica": R.lw_control(i_cloud=abi.IP_CLOUD_MCICA)}[kind]
    return ctl, sp, col, mc


def _check(ctl, sp, col, mc, tag):
    gpu = R.radiance_calc(replace(ctl, precision=abi.PRECISION_MIXED), sp, col, mc)
    ref = O.radiance_calc(ctl, sp, col, mc, threads=8)
    top = max(np.abs(ref[k]).max() for k in ("flux_up", "flux_down"))
    for k in ("flux_up", "flux_down", "flux_direct"):
        if k in ref:
            err = np.abs(gpu[k] - ref[k]).max()
            assert err <= 4 * col.n_layer * 2.0 ** -24 * top, (tag, k, err)
    assert np.abs(gpu["heating_rate"] - ref["heating_rate"]).max() <= 0.05, tag
    return gpu


@pytest.mark.parametrize("kind", ["sw", "lw", "lw_scat", "sw_mcica", "lw_mcica"])
@pytest.mark.parametrize("L", [1, 2, 33, 40, 41, 64, 65, 72, 73, 88, 89, 96, 97, 104, 105, 144, 145])
def test_layer_counts_at_tile_edges(gpu_lib, kind, L):
    _check(*_case(kind, 5, L, 11), (kind, L))


@pytest.mark.parametrize("kind", ["sw", "lw", "lw_mcica"])
@pytest.mark.parametrize("n", [1, 3, 511, 512, 513, 514, 515])
def test_column_counts(gpu_lib, kind, n):
    _check(*_case(kind, n, 38, 12), (kind, n))


@pytest.mark.parametrize("lanes,chunk", [(8, 5), (8, 13), (16, 3), (16, 9), (32, 3), (32, 16)])
@pytest.mark.parametrize("warps", [1, 4, 8])
def test_tiles_and_warps(gpu_lib, lanes, chunk, warps):
    """Every lane count with one, four and eight warps per CTA (one and four
    columns), on a layer count that leaves padding in each tile."""
    for mode, kind in ((0, "lw"), (1, "sw"), (2, "sw_mcica")):
        assert gpu_lib.socgpu_tune_set(abi.PRECISION_MIXED, mode, 37, lanes, chunk, warps) == 0
        try:
            _check(*_case(kind, 514, 37, 13), (lanes, chunk, warps, kind))
        finally:
            gpu_lib.socgpu_tune_set(abi.PRECISION_MIXED, mode, 37, 0, 0, 0)


@pytest.mark.parametrize("kind", ["sw", "sw_mcica"])
@pytest.mark.parametrize("opt", [dict(i_direct_tau=abi.IP_DIRECT_NOSCALING), dict(l_rescale=False),
                                 dict(first_band=2, last_band=4), dict(i_2stream=abi.IP_EDDINGTON),
                                 dict(l_gas=False), dict(l_rayleigh=False, l_gas=False, l_aerosol_mode=False)])
def test_options(gpu_lib, kind, opt):
    ctl, sp, col, mc = _case(kind, 513, 47, 14)
    _check(replace(ctl, **opt), sp, col, mc, (kind, opt))


def test_nan_stays_in_its_column(gpu_lib):
    """Columns that share a CTA do not mix: a NaN mass spoils its own column
    and leaves the others as they were, bit for bit."""
    for kind in ("sw", "lw", "sw_mcica"):
        ctl, sp, col, mc = _case(kind, 514, 38, 15)
        ctl = replace(ctl, precision=abi.PRECISION_MIXED)
        a = R.radiance_calc(ctl, sp, col, mc)
        col.mass = col.mass.copy(order="F")
        col.mass[6, 20] = np.nan
        b = R.radiance_calc(ctl, sp, col, mc)
        keep = np.arange(514) != 6
        for k in a:
            np.testing.assert_array_equal(a[k][keep], b[k][keep])
        assert np.isnan(b["flux_up"][6]).all() and np.isnan(b["heating_rate"][6, 20])


def test_batch_of_wide_and_narrow_items(gpu_lib):
    """One class of a replayed graph holds items of one and of four columns
    per CTA; each equals its own call."""
    cases = [DeviceCase(*(lambda c, s, k, m: (replace(c, precision=abi.PRECISION_MIXED), s, k, m))(*_case(kind, n, 60, 16)))
             for kind in ("lw", "sw", "sw_mcica") for n in (3, 513, 600)]
    alone = []
    for c in cases:
        c.run()
        alone.append({k: c.tensors["out_" + k].clone() for k in ("flux_up", "flux_down", "heating_rate")})
        for t in c.tensors:
            if t.startswith("out_"):
                c.tensors[t].zero_()
    Batch(cases).run()
    for c, a in zip(cases, alone):
        for k, v in a.items():
            np.testing.assert_array_equal(c.tensors["out_" + k].cpu().numpy(), v.cpu().numpy())
