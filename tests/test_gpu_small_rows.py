"""GPU tests of the FP64 row sums with a warp per particle (small calls) and with
eight lanes per particle, at the edges of both: rows of 1 to 128 entries around
each lane's share (32), the last call of a warp per particle and the first
beyond it (8 per SM: 1216 on 152 SMs), against the oracle.

Tolerance: FP64 1e-11, as in test_gpu_functors.py.
"""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as orc
from research_codes_gb300 import abi, functors
from test_gpu_edge_values import ETA, _ball, _density, _density_inputs, _hydro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_i", [1, 3, 4, 1215, 1216, 1217])
@pytest.mark.parametrize("n_j,neighbours", [(1, 1), (31, 31), (33, 33), (64, 64), (97, 97), (128, 128), (1300, 40)])
def test_rows_of_every_length(n_i, n_j, neighbours):
    n_i = min(n_i, n_j)
    epi, epj, near = _ball(n_i, n_j, 67 * n_i + n_j, neighbours=neighbours)
    out, ref = _hydro("fp64", epi, epj), orc.hydro(epi, epj)
    for f in ("acch", "accg", "udot", "vsmx", "diffu"):
        assert rel_err(out[f], ref[f], 1e-3).max() < 1e-11, f
    di, dj = _density_inputs(epi, epj)
    first = orc.density(di, dj, eta=ETA, ksr_max=0.0)["ksr"]
    di["ksr"] = np.where(np.isfinite(first), first, 1.0)   # settled: rows stay valid
    out, ref = _density("fp64", di, dj), orc.density(di, dj, eta=ETA, ksr_max=0.0)
    for f in ("dens", "ksr", "grdh", "divv", "rotv"):
        assert rel_err(out[f], ref[f], 1e-2).max() < 1e-11, f
    assert np.array_equal(out["np"], ref["np"]) and np.array_equal(out["itr"], ref["itr"])


def test_a_row_does_not_depend_on_the_size_of_the_call():
    """The same targets in calls of a warp and of eight lanes per particle: sums
    in another order (1e-13)."""
    epi, epj, near = _ball(1300, 1300, 3)
    di, dj = _density_inputs(epi, epj)
    many = _density("fp64", di, dj), _hydro("fp64", epi, epj)
    few = _density("fp64", di[:700], dj), _hydro("fp64", epi[:700], epj)
    for a, b in zip(many, few):
        for f in a.dtype.names:
            x, y = a[f][:700].astype(float), b[f].astype(float)
            assert np.allclose(x, y, rtol=1e-13, atol=1e-13 * np.abs(x).max()), f
