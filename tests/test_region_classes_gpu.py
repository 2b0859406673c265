"""Cloud-region items of one kernel class whose scratch rows differ in size:
layer counts of one tile, band ranges, two and three regions, with fewer and
with more columns than resident CTAs.  Each item of a replayed graph and of a
server wave has the results of its own call.

Tolerance: the kernels run the same arithmetic but are compiled in different
contexts, so FP32 contractions may differ: 1e-5 of the largest flux in mixed
precision, 1e-12 in FP64 (the bounds of the other multi-batch tests)."""
from dataclasses import replace

import numpy as np
import pytest

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase
from socrates_gb300.server import Server

pytestmark = pytest.mark.gpu

KEYS = ("flux_up", "flux_down", "flux_direct")
TRIPLE = dict(i_cloud=abi.IP_CLOUD_TRIPLE, i_solver=abi.IP_SOLVER_TRIPLE_HOGAN,
              i_cloud_representation=abi.IP_CLOUD_CONV_STRAT)


def _items(solar, precision, narrow):
    sp = synth.sw_spectrum(41, 8, clouds=True) if solar else synth.lw_spectrum(41, 9, clouds=True)
    mk = R.sw_control if solar else R.lw_control
    base = mk(i_cloud=abi.IP_CLOUD_MIX_MAX, i_solver=abi.IP_SOLVER_MIX_DIRECT_HOGAN, precision=precision)
    out = []
    for i, (n, L, kw) in enumerate([(40, 70, {}), (40, 66, {}), (40, 70, TRIPLE), (40, 69, dict(first_band=2, last_band=3)),
                                    (1, 65, {})]):
        n = n if narrow or n == 1 else 8 * n
        col = synth.atmosphere(n, L, sp.type_absorb, 51 + i)
        if solar:
            synth.add_sw_surface(col, sp.n_band, 51 + i)
        else:
            synth.add_lw_surface(col, sp.n_band)
        synth.add_clouds(col, 51 + i, 4, p_top=0.0)
        out.append((replace(base, **kw), sp, col))
    return out


def _close(got, want, precision, tag):
    tol = 1e-12 if precision == abi.PRECISION_FP64 else 1e-5
    for k in KEYS:
        if k in want:
            err = np.abs(got[k] - want[k]).max() / np.abs(want[k]).max()
            assert err <= tol, (tag, k, err)


@pytest.mark.parametrize("solar", [True, False])
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
@pytest.mark.parametrize("narrow", [True, False])
def test_graph(gpu_lib, solar, precision, narrow):
    none = R.McicaState(1, 1, None, None, None, None, None, None)
    items = _items(solar, precision, narrow)
    cases = [DeviceCase(*it, none) for it in items]
    b = Batch(cases)
    assert b.info()["kernel_classes"] == 1
    want = [R.radiance_calc(*it) for it in items]
    for _ in range(3):
        for c in cases:
            c.tensors["out_flux_up"].zero_()
        b.run()
        for i, (c, w) in enumerate(zip(cases, want)):
            _close({k: c.output(k) for k in w if k in KEYS}, w, precision, i)
    b.close()


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_server(gpu_lib, precision):
    items = [it for solar in (True, False) for it in _items(solar, precision, True)]
    want = [R.radiance_calc(*it) for it in items]
    marshals = [R.Marshal(*it) for it in items]
    srv = Server(device_bytes=256 << 20, streams=2, max_wave_requests=16)
    tickets = [srv.submit(m, it[1]) for m, it in zip(marshals, items)]
    for t in tickets:
        srv.wait(t, 60.0)
    srv.close()
    for i, (m, w) in enumerate(zip(marshals, want)):
        _close(m.result(), w, precision, i)
