"""The columns that share a CTA of the mixed kernels follow from the columns of
the call, not from the extent of its arrays: a call of a few columns in wide
arrays runs as the same columns in arrays of their own do, bit for bit."""
import numpy as np
import pytest

from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R
from socrates_gb300.device import DeviceCase

pytestmark = pytest.mark.gpu
WIDE = 2500


def _columns(kind, L):
    solar = kind.startswith("sw")
    sp = synth.sw_spectrum(71, 8, clouds=True) if solar else synth.lw_spectrum(71, 9, clouds=True)
    col = synth.atmosphere(WIDE, L, sp.type_absorb, 71)
    if solar:
        synth.add_sw_surface(col, sp.n_band, 71)
    else:
        synth.add_lw_surface(col, sp.n_band)
    kw = dict(precision=abi.PRECISION_MIXED)
    if kind == "lw":
        return R.lw_noscat_control(**kw), sp, col
    return (R.sw_control if solar else R.lw_control)(**kw), sp, col


@pytest.mark.parametrize("kind", ["sw", "lw", "lw_scat"])
@pytest.mark.parametrize("n,L", [(1, 38), (27, 70), (305, 38), (609, 38)])
def test_few_columns_of_wide_arrays(gpu_lib, kind, n, L):
    ctl, sp, col = _columns(kind, L)
    wide = DeviceCase(ctl, sp, col)
    wide.atm.n_profile = n
    wide.run()
    own = DeviceCase(ctl, sp, synth.window(col, 0, n))
    own.run()
    for k in ("flux_up", "flux_down", "heating_rate"):
        np.testing.assert_array_equal(wide.output(k)[:n], own.output(k), err_msg=k)
        assert not wide.output(k)[n:].any()          # the columns past the call are not written
