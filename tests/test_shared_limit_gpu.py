"""A kernel's shared-memory limit serves every launch of it: classes of one
graph or server wave that run the same kernel with different sizes, and host
threads that call with columns of different widths and layer counts.  Results
equal each item's own call (1e-12 relative in FP64, 0.1 W/m2 mixed, the bounds
of the other batch and server tests)."""
import ctypes as C
import threading
from pathlib import Path

import numpy as np
import pytest

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase
from socrates_gb300.server import Server
from socrates_gb300.spectrum import Spectrum

pytestmark = pytest.mark.gpu
GA9 = Path(__file__).resolve().parent / "golden" / "runes_ga9.npz"
NO_SUBCOL = R.McicaState(1, 1, None, None, None, None, None, None)


def _all_sky(n, L, region, precision, seed, solar=True):
    """Columns of the default cloud spectra, as McICA or as two regions."""
    sp = synth.sw_spectrum(2, 8, clouds=True) if solar else synth.lw_spectrum(1, 9, clouds=True)
    col = synth.atmosphere(n, L, sp.type_absorb, seed)
    if solar:
        synth.add_sw_surface(col, sp.n_band, seed)
    else:
        synth.add_lw_surface(col, sp.n_band)
    synth.add_clouds(col, seed, 16)
    mk = R.sw_control if solar else R.lw_control
    if region:
        return mk(i_cloud=abi.IP_CLOUD_MIX_MAX, i_solver=abi.IP_SOLVER_MIX_DIRECT_HOGAN, precision=precision), sp, col, NO_SUBCOL
    isolir = abi.IP_SOLAR if solar else abi.IP_INFRA_RED
    mc = R.set_cld_mcica(sp, col, isolir, abi.IP_MCICA_SINGLE_SAMPLING, rng=abi.RNG_PHILOX)
    return mk(i_cloud=abi.IP_CLOUD_MCICA, precision=precision), sp, col, mc


def _ga9(n, L, seed, sp):
    col = synth.operational_case(sp, n, L, seed=seed, solar=True)
    return R.sw_control(l_continuum=True, i_gas_overlap=abi.IP_OVERLAP_K_EQV_SCL, precision=abi.PRECISION_MIXED), sp, col, None


def _mixes():
    yield "fp64 mcica and regions", [_all_sky(5, 85, region, abi.PRECISION_FP64, 61, solar)
                                     for solar in (True, False) for region in (False, True)]
    sp = Spectrum.load_npz(GA9, prefix="sw_")
    yield "wide and narrow ga9", [_ga9(n, 60, 62, sp) for n in (1000, 200)]


def _close(got, want, precision, tag):
    for k in ("flux_up", "flux_down", "flux_direct"):
        if k in want and k in got:
            err = np.abs(got[k] - want[k]).max()
            assert err <= (1e-12 * np.abs(want[k]).max() if precision == abi.PRECISION_FP64 else 0.1), (tag, k, err)


def _call(it):
    return R.radiance_calc(it[0], it[1], it[2], None if it[3] is NO_SUBCOL else it[3])


@pytest.mark.parametrize("i", [0, 1])
def test_graph(gpu_lib, i):
    tag, items = list(_mixes())[i]
    cases = [DeviceCase(*it) for it in items]
    b = Batch(cases)
    b.run()
    for c, it in zip(cases, items):
        _close({k: c.output(k) for k in ("flux_up", "flux_down")}, _call(it), it[0].precision, tag)
    b.close()


@pytest.mark.parametrize("i", [0, 1])
def test_server_wave(gpu_lib, i):
    tag, items = list(_mixes())[i]
    marshals = [R.Marshal(it[0], it[1], it[2], None if it[3] is NO_SUBCOL else it[3]) for it in items]
    srv = Server(device_bytes=512 << 20, streams=1, max_wave_requests=16)
    # several rounds, so that a wave holds both kinds whatever the first one took
    for _ in range(4):
        tickets = [srv.submit(m, it[1]) for m, it in zip(marshals, items)]
        for t in tickets:
            srv.wait(t, 60.0)
    srv.close()
    for m, it in zip(marshals, items):
        _close(m.result(), _call(it), it[0].precision, tag)


def _generator(L, n=64):
    """A call of the subcolumn generator on device arrays, and its masks."""
    import torch
    col = synth.atmosphere(n, L, np.array([1, 2, 3], np.int32), 64)
    synth.add_clouds(col, 64, 16)

    def dev(a, dtype=np.float64):
        return torch.from_numpy(np.asarray(a, dtype=dtype).ravel(order="F").copy()).cuda()
    cd, zero = col.cld, np.zeros((n, L))
    t = [dev(cd["rand_seed"], np.int32), dev(cd["dp_corr_cloud"]), dev(cd["dp_corr_cond"]), dev(zero), dev(cd["w_cloud"]),
         dev(zero), dev(zero), dev(col.p), dev(np.zeros((2, 2)))]
    n_cld, c_sub = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(n * L * 16, dtype=torch.float64, device="cuda")
    args = ([L, 1, L, n, 1, n, 16, 2, 2, 0, abi.IP_EXPONENTIAL_RAND] + [x.data_ptr() for x in t]
            + [n_cld.data_ptr(), c_sub.data_ptr(), abi.RNG_PHILOX])

    def call(stream, keep=t):
        msg = C.create_string_buffer(512)
        st = R.load_library().socgpu_cloud_gen_device(*args, C.c_void_p(stream), msg, 512)
        if st != abi.I_NORMAL:
            raise R.RadianceError(st, msg.value.decode())
    return call, c_sub


def test_threads_of_different_widths(gpu_lib):
    """Host threads on one spectrum, on streams of their own: the launches'
    sizes differ with the width and the layer count, and the generator's with
    the layer count."""
    import torch
    cases = []
    for n, L in ((1, 100), (2, 98), (400, 97), (700, 98)):
        sp, col = synth.config2(n, L, seed=63)
        cases.append(DeviceCase(R.sw_control(l_aerosol_mode=True, precision=abi.PRECISION_MIXED), sp, col))
    calls = [c.run for c in cases]
    outs = [c.tensors["out_flux_up"] for c in cases]
    for L in (10, 40, 120, 137):
        call, c_sub = _generator(L)
        calls.append(call)
        outs.append(c_sub)
    for call in calls:
        call(0)
    torch.cuda.synchronize()
    want = [o.cpu().numpy().copy() for o in outs]
    errors = []

    def repeat(call):
        s = torch.cuda.Stream()
        try:
            for _ in range(2000):
                call(s.cuda_stream)
        except Exception as e:          # reported by the main thread
            errors.append(repr(e))
        s.synchronize()

    threads = [threading.Thread(target=repeat, args=(call,)) for call in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
    for o, w in zip(outs, want):
        np.testing.assert_array_equal(o.cpu().numpy(), w)
