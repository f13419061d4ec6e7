"""GPU tests of FP32C hydro calls whose lists a block marks because the call has
few items (up to one of 32 targets per SM, lists of more than 256 entries): the
same bits as a warp per list gives in a call of many items, at the edges of both.

Tolerance: none (rows in the same order).  What a warp gives is compared with the
oracle in test_gpu_rows.py.
"""
import numpy as np
import pytest

from research_codes_gb300 import abi, functors
from test_gpu_rows import ETA, _hydro_cloud

pytestmark = pytest.mark.gpu


def _dispatch(epi, epj):
    n_i = [len(a) for a in epi]
    out = [np.zeros(n, abi.Hydro) for n in n_i]
    with functors.Context(precision="fp32c", eta=ETA) as ctx:
        functors.DispatchKernel_HydroForce(ctx, 0, len(epi), epi, n_i, epj, [len(b) for b in epj])
        functors.RetrieveKernel_HydroForce(ctx, 0, len(epi), n_i, out)
    return out


# walks of one target beside it: 150 items (with up to two of its own the last call by blocks), 400 (by warps)
@pytest.mark.parametrize("n_i", [1, 5, 9, 17, 32, 40])
@pytest.mark.parametrize("n_j,neighbours", [(255, 40.0), (256, 40.0), (257, 40.0), (321, 50.0), (1000, 50.0), (1536, 60.0)])
def test_blocks_give_the_bits_of_warps(n_i, n_j, neighbours):
    epi, epj = _hydro_cloud(n_i, n_j, 3 * n_i + n_j, neighbours)
    small = epi[:1], epj[:60]
    got = [_dispatch([epi] + [small[0]] * k, [epj] + [small[1]] * k)[0] for k in (0, 150, 400)]
    for f in abi.Hydro.names:
        assert np.array_equal(got[0][f], got[2][f]) and np.array_equal(got[1][f], got[2][f]), f
