"""Equivalent extinction in mixed precision on every CTA shape that the
launcher chooses between: column counts at and one past the waves of each,
layer counts of each tile, both sources, alone and in a replayed graph.

The columns are eight, repeated: the eight's fluxes against the FP64 kernels
within 0.1 W/m2 (the bound of the GA9 parity tests), and every repetition
equal to the first bit for bit (a column's values do not depend on
its place in the CTA).  In the graph the shape follows from all items
together, so the sums' order may differ from an item's own call: 0.1 W/m2."""
from dataclasses import replace
from pathlib import Path

import numpy as np
import pytest

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase
from socrates_gb300.spectrum import Spectrum

pytestmark = pytest.mark.gpu
GA9 = Path(__file__).resolve().parent / "golden" / "runes_ga9.npz"
KEYS = ("flux_up", "flux_down", "heating_rate")


def _problem(solar, L):
    sp = Spectrum.load_npz(GA9, prefix="sw_" if solar else "lw_")
    col = synth.operational_case(sp, 8, L, seed=81, solar=solar)
    kw = dict(l_continuum=True, i_gas_overlap=abi.IP_OVERLAP_K_EQV_SCL)
    return (R.sw_control(**kw) if solar else R.lw_control(l_ir_source_quad=True, **kw)), sp, col


def _repeat(col, n):
    import copy
    c = copy.copy(col)
    c.n_profile = n
    for name, v in vars(col).items():
        if isinstance(v, np.ndarray) and v.ndim >= 1 and v.shape[0] == 8 and name not in ("type_absorb",):
            setattr(c, name, np.asfortranarray(v[np.arange(n) % 8]))
    return c


def _check(got, ref, n, tag):
    for k in KEYS:
        a = got.output(k)
        err = np.abs(a[:8] - ref[k][:min(n, 8)]).max()
        assert k == "heating_rate" or err <= 0.1, (tag, k, err)
        np.testing.assert_array_equal(a, a[np.arange(n) % 8], err_msg=str((tag, k)))


@pytest.mark.parametrize("solar", [True, False])
@pytest.mark.parametrize("L", [33, 48, 49, 64, 65, 96, 97, 137])
def test_column_counts(gpu_lib, solar, L):
    ctl, sp, col = _problem(solar, L)
    ref = R.radiance_calc(replace(ctl, precision=abi.PRECISION_FP64), sp, col)
    for n in (1, 304, 305, 457, 608, 609, 913, 1217, 2433):
        dc = DeviceCase(replace(ctl, precision=abi.PRECISION_MIXED), sp, _repeat(col, n))
        dc.run()
        _check(dc, ref, n, (solar, L, n))


@pytest.mark.parametrize("solar", [True, False])
@pytest.mark.parametrize("counts", [(3, 200, 8), (700, 1, 1300)])
def test_graph(gpu_lib, solar, counts):
    cases, refs = [], []
    for L in (38, 60, 70):
        ctl, sp, col = _problem(solar, L)
        ref = R.radiance_calc(replace(ctl, precision=abi.PRECISION_FP64), sp, col)
        for n in counts:
            cases.append(DeviceCase(replace(ctl, precision=abi.PRECISION_MIXED), sp, _repeat(col, n)))
            refs.append((ref, n, L))
    b = Batch(cases)
    b.run()
    for dc, (ref, n, L) in zip(cases, refs):
        _check(dc, ref, n, (solar, L, n))
    b.close()
