"""Cloud regions with a thread per g-point: more columns than resident CTAs
(each CTA strides over several), more g-points than solve at a time (the
infra-red's 81 against 64), a single layer, and the replayed graph, whose rows
belong to the batch.  FP64 against the oracle within 1e-10 of the largest flux
(the bound of the other region tests), mixed fluxes within 0.1 W/m2; a column's
values do not depend on the columns beside it."""
from dataclasses import replace

import numpy as np
import pytest

import oracle as O
from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase

pytestmark = pytest.mark.gpu


def _case(solar, n, L, seed, solver=abi.IP_SOLVER_MIX_DIRECT_HOGAN, scheme=abi.IP_CLOUD_MIX_MAX):
    sp = synth.sw_spectrum(seed, 8, clouds=True) if solar else synth.lw_spectrum(seed, 9, clouds=True)
    col = synth.atmosphere(n, L, sp.type_absorb, seed)
    if solar:
        synth.add_sw_surface(col, sp.n_band, seed)
    else:
        synth.add_lw_surface(col, sp.n_band)
    synth.add_clouds(col, seed, 4, p_top=0.0)
    mk = R.sw_control if solar else R.lw_control
    return mk(i_cloud=scheme, i_solver=solver), sp, col


@pytest.mark.parametrize("solar", [True, False])
@pytest.mark.parametrize("n,L", [(3, 1), (5, 2), (40, 33), (7, 137)])
@pytest.mark.parametrize("solver", [abi.IP_SOLVER_MIX_DIRECT, abi.IP_SOLVER_MIX_DIRECT_HOGAN])
def test_against_oracle(gpu_lib, solar, n, L, solver):
    ctl, sp, col = _case(solar, n, L, 31, solver)
    ref = O.radiance_calc(ctl, sp, col, threads=8)
    top = max(np.abs(ref[k]).max() for k in ("flux_up", "flux_down"))
    g = R.radiance_calc(ctl, sp, col)
    m = R.radiance_calc(replace(ctl, precision=abi.PRECISION_MIXED), sp, col)
    for k in ("flux_up", "flux_down", "flux_direct"):
        if k in ref:
            assert np.abs(g[k] - ref[k]).max() <= 1e-10 * top, k
            assert np.abs(m[k] - ref[k]).max() <= 0.1, k


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_more_columns_than_ctas(gpu_lib, precision):
    for solar in (True, False):
        ctl, sp, col = _case(solar, 700, 20, 32)
        ctl = replace(ctl, precision=precision)
        whole = R.radiance_calc(ctl, sp, col)
        part = R.radiance_calc(ctl, sp, synth.window(col, 640, 60))
        for k in part:
            np.testing.assert_array_equal(whole[k][640:], part[k])


def test_batch_rows(gpu_lib):
    """Regions, McICA-free, of both sources and precisions in one graph,
    replayed twice, equal their own calls."""
    cases = []
    for solar in (True, False):
        for prec in (abi.PRECISION_FP64, abi.PRECISION_MIXED):
            for n, L in ((30, 20), (5, 60)):
                ctl, sp, col = _case(solar, n, L, 33)
                none = R.McicaState(1, 1, None, None, None, None, None, None)
                cases.append(DeviceCase(replace(ctl, precision=prec), sp, col, none))
    alone = []
    for c in cases:
        c.run()
        alone.append(c.output("flux_up").copy())
    b = Batch(cases)
    for _ in range(2):
        for c in cases:
            c.tensors["out_flux_up"].zero_()
        b.run()
        for c, a in zip(cases, alone):
            np.testing.assert_array_equal(c.output("flux_up"), a)
