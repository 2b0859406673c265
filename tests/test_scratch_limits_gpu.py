"""Calls at the limit of shared memory that FP64 batches take: operational
short-wave columns with 64 McICA subcolumns and the unscaled direct beam, whose
one band does not fit beside eight warps' accumulators.  The batch runs them
with fewer warps, and gives the values of the single call (1e-12 of the largest
flux, the bound of the other FP64 batch tests)."""
import numpy as np
import pytest

import cld7460 as K
from socrates_gb300 import abi
from socrates_gb300 import radiance as R
from socrates_gb300.batch import Batch
from socrates_gb300.device import DeviceCase
from test_cloud_region_gpu import _clouded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [130, 144])
def test_batch_with_many_subcolumns(gpu_lib, L):
    sp = K.spectra()["ga9sw"]
    col = _clouded(sp, 6, L, 95, True, abi.IP_CLOUD_ICE_WATER)
    f = np.asfortranarray
    col.cld.update(rand_seed=np.arange(1, 7, dtype=np.int32), dp_corr_cloud=f(np.full((6, L), 1e4)),
                   dp_corr_cond=f(np.full((6, L), 1e4)), n_subcol_gen=64)
    mc = R.set_cld_mcica(sp, col, abi.IP_SOLAR, abi.IP_MCICA_SINGLE_SAMPLING, rng=abi.RNG_PHILOX)
    ctl = R.sw_control(i_cloud=abi.IP_CLOUD_MCICA, l_continuum=True, i_gas_overlap=abi.IP_OVERLAP_K_EQV_SCL,
                       i_direct_tau=abi.IP_DIRECT_NOSCALING)
    case = DeviceCase(ctl, sp, col, mc)
    case.run()
    want = {k: case.output(k).copy() for k in ("flux_up", "flux_down", "flux_direct")}
    for k in want:
        case.tensors["out_" + k].zero_()
    b = Batch([case])
    b.run()
    for k, v in want.items():
        assert np.abs(case.output(k) - v).max() <= 1e-12 * np.abs(v).max(), k
    b.close()
