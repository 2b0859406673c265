"""Graphs of many narrow items of up to 40 layers, whose kernel is the one with
three resident CTAs, beside a graph small enough for the other: each item has
its own call's fluxes.  The two kernels run the same arithmetic but are
compiled for different register counts, so FP32 contractions may differ: 1e-5
of the largest flux (the bound of the other multi-batch tests)."""
import numpy as np
import pytest

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase

pytestmark = pytest.mark.gpu


def _case(kind, n, L, seed):
    solar = kind == "sw"
    sp = synth.sw_spectrum(91, 8) if solar else synth.lw_spectrum(91, 9)
    col = synth.atmosphere(n, L, sp.type_absorb, seed)
    if solar:
        synth.add_sw_surface(col, sp.n_band, seed)
    else:
        synth.add_lw_surface(col, sp.n_band)
    kw = dict(precision=abi.PRECISION_MIXED)
    ctl = R.sw_control(**kw) if solar else R.lw_noscat_control(**kw) if kind == "lw" else R.lw_control(**kw)
    return DeviceCase(ctl, sp, col)


@pytest.mark.parametrize("kind", ["sw", "lw", "lw_scat"])
@pytest.mark.parametrize("widths", [(1, 7), tuple([3, 61, 17, 304] * 6), (305, 90, 200, 300, 280)])
def test_items_equal_their_own_calls(gpu_lib, kind, widths):
    cases = [_case(kind, n, (33, 38, 40, 2)[i % 4], 92 + i) for i, n in enumerate(widths)]
    own = []
    for c in cases:
        c.run()
        own.append({k: c.output(k).copy() for k in ("flux_up", "flux_down")})
        for k in ("flux_up", "flux_down"):
            c.tensors["out_" + k].zero_()
    b = Batch(cases)
    assert b.info()["kernel_classes"] == 1
    b.run()
    for i, (c, w) in enumerate(zip(cases, own)):
        for k, v in w.items():
            err = np.abs(c.output(k) - v).max() / np.abs(v).max()
            assert err <= 1e-5, (i, k, err)
    b.close()
