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
