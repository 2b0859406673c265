"""The subcolumn generator spread over subcolumns (Philox, random and
exponential-random overlap) bit for bit against the oracle: column counts
around a warp, subcolumn counts around the CTA's warps, layer counts around a
mask word, cloud tops below the first layer, clear and overcast columns, and
fractions at and below epsilon, which correlate a column's first cloudy layer
with the subcolumn before."""
import numpy as np
import pytest

import oracle as O
from socrates_gb300 import abi, synth
from socrates_gb300 import radiance as R

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _same(col, n_subcol, overlap, id_cloud_top=1):
    g, gn = R.cloud_gen(col, n_subcol, overlap, abi.RNG_PHILOX, id_cloud_top=id_cloud_top)
    o, on = R.cloud_gen(col, n_subcol, overlap, abi.RNG_PHILOX, id_cloud_top=id_cloud_top, impl=O.cloud_gen_impl)
    np.testing.assert_array_equal(gn, on)
    np.testing.assert_array_equal(g, o)
    return gn


@pytest.mark.parametrize("overlap", [abi.IP_RAND, abi.IP_EXPONENTIAL_RAND])
@pytest.mark.parametrize("n,L,n_subcol", [(1, 1, 1), (31, 32, 16), (32, 33, 17), (33, 64, 3), (70, 65, 40), (40, 137, 16),
                                          (5, 200, 2)])
def test_masks_bit_exact(gpu_lib, overlap, n, L, n_subcol):
    col = synth.atmosphere(n, L, np.array([1, 2, 3], np.int32), 21)
    synth.add_clouds(col, 21, n_subcol, cloud_prob=0.6, p_top=0.0)
    _same(col, n_subcol, overlap)
    if L > 8:
        _same(col, n_subcol, overlap, id_cloud_top=7)


@pytest.mark.parametrize("overlap", [abi.IP_RAND, abi.IP_EXPONENTIAL_RAND, abi.IP_EXPONENTIAL, abi.IP_MAX_RAND])
def test_edge_fractions(gpu_lib, overlap):
    col = synth.atmosphere(64, 40, np.array([1, 2, 3], np.int32), 22)
    synth.add_clouds(col, 22, 16, cloud_prob=0.5, p_top=0.0)
    w = col.cld["w_cloud"]
    w[0] = 0.0                                   # clear
    w[1] = 1.0                                   # overcast
    w[2] = EPS                                   # cloud by the >= test of the lowest layer only
    w[3] = EPS / 2                               # below epsilon everywhere
    # a trace above the first cloudy layer: the layer is correlated with it
    w[4:40, :10] = 0.0
    w[4:40, 9] = EPS / 4
    w[4:40, 10] = 0.7
    w[:, :8] = 0.0
    w[63, 8] = 0.5                               # puts the trace inside the batch's range
    _same(col, 16, overlap)
    col.cld["dp_corr_cloud"][5:20] = 0.0         # no decorrelation scale
    _same(col, 16, overlap)


def test_all_clear(gpu_lib):
    col = synth.atmosphere(40, 20, np.array([1, 2, 3], np.int32), 23)
    synth.add_clouds(col, 23, 16)
    col.cld["w_cloud"][:] = 0.0
    assert _same(col, 16, abi.IP_EXPONENTIAL_RAND).max() == 0
