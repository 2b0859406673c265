"""Rounding of the mixed kernels against the FP64 kernels, at the level that
their one-column predecessors had: the bounds are those kernels' errors on the
same columns (measured before this file was first run), not a multiple of the
present ones."""
from dataclasses import replace
from pathlib import Path

import numpy as np
import pytest

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.spectrum import Spectrum

pytestmark = pytest.mark.gpu
GA9 = Path(__file__).resolve().parent / "golden" / "runes_ga9.npz"


@pytest.mark.parametrize("L,bound", [(38, 9.68e-7), (70, 1.75e-6), (137, 3.08e-6)])
def test_upward_flux_of_clear_columns(gpu_lib, L, bound):
    """Relative root-mean-square error of the upward flux of 64 GA9 short-wave
    columns: the transmissions of the layers multiply, and so do their roundings."""
    sp = Spectrum.load_npz(GA9, prefix="sw_")
    col = synth.operational_case(sp, 64, L, seed=1, solar=True)
    ctl = R.sw_control(l_continuum=True, i_gas_overlap=abi.IP_OVERLAP_K_EQV_SCL)
    ref = R.radiance_calc(ctl, sp, col)["flux_up"]
    got = R.radiance_calc(replace(ctl, precision=abi.PRECISION_MIXED), sp, col)["flux_up"]
    err = np.sqrt(((got - ref) ** 2).mean() / (ref ** 2).mean())
    assert err <= bound, err


@pytest.mark.parametrize("solar", [True, False])
@pytest.mark.parametrize("L", [40, 70, 105, 137])
@pytest.mark.parametrize("mmr,bound", [(1e-4, 2e-5), (1e-3, 2e-5), (1e-2, 1e-4)])
def test_downward_flux_under_thick_cloud(gpu_lib, solar, L, mmr, bound):
    """Overcast columns, solar fluxes at the surface down to 2e-5 W/m2: the
    downward flux keeps its relative accuracy at every level (the predecessors'
    errors were up to 1.6e-5 for the two thinner clouds and 8.3e-5 for the
    thickest), and it is never negative.  The infra-red's, of the order of the
    emission everywhere, within 4 L 2^-24 of the largest (the bound of the tile
    tests)."""
    sp = synth.sw_spectrum(2, 8, clouds=True) if solar else synth.lw_spectrum(1, 9, clouds=True)
    col = synth.atmosphere(64, L, sp.type_absorb, 5)
    if solar:
        synth.add_sw_surface(col, sp.n_band, 5)
    else:
        synth.add_lw_surface(col, sp.n_band)
    synth.add_clouds(col, 5, 16)
    deep, cd = col.p > 4e4, col.cld
    f = np.asfortranarray
    cd["w_cloud"] = f(np.where(deep, 1.0, 0.0))
    for key, value in (("frac_cloud", 1.0), ("condensed_mix_ratio", mmr)):
        a = np.zeros_like(cd[key])
        a[..., 0] = np.where(deep, value, 0.0)
        cd[key] = f(a)
    a = np.array(cd["condensed_dim_char"])
    a[..., 0] = np.where(deep, 1e-5, a[..., 0])
    cd["condensed_dim_char"] = f(a)
    isolir = abi.IP_SOLAR if solar else abi.IP_INFRA_RED
    mc = R.set_cld_mcica(sp, col, isolir, abi.IP_MCICA_SINGLE_SAMPLING, rng=abi.RNG_PHILOX)
    ctl = (R.sw_control if solar else R.lw_control)(i_cloud=abi.IP_CLOUD_MCICA)
    ref = R.radiance_calc(ctl, sp, col, mc)["flux_down"]
    got = R.radiance_calc(replace(ctl, precision=abi.PRECISION_MIXED), sp, col, mc)["flux_down"]
    if solar:
        assert (np.abs(got - ref) <= bound * ref).all(), (np.abs(got - ref) / ref).max()
        assert got.min() >= 0.0
    else:
        assert np.abs(got - ref).max() <= 4 * L * 2.0 ** -24 * ref.max()


@pytest.mark.parametrize("L,down,direct", [(38, 1.24e-7, 1.87e-7), (70, 1.68e-7, 2.77e-7), (137, 2.78e-7, 4.49e-7)])
def test_sums_over_g_points_of_cloud_regions(gpu_lib, L, down, direct):
    """Relative root-mean-square errors of 64 two-region solar columns: the
    regions are solved in FP64, so what the sums over the g-points round shows."""
    sp = synth.sw_spectrum(2, 8, clouds=True)
    col = synth.atmosphere(64, L, sp.type_absorb, 1)
    synth.add_sw_surface(col, sp.n_band, 1)
    synth.add_clouds(col, 1, 16)
    ctl = R.sw_control(i_cloud=abi.IP_CLOUD_MIX_MAX, i_solver=abi.IP_SOLVER_MIX_DIRECT_HOGAN)
    ref = R.radiance_calc(ctl, sp, col)
    got = R.radiance_calc(replace(ctl, precision=abi.PRECISION_MIXED), sp, col)
    for k, bound in (("flux_down", down), ("flux_direct", direct)):
        err = np.sqrt(((got[k] - ref[k]) ** 2).mean() / (ref[k] ** 2).mean())
        assert err <= bound, (k, err)
