"""GPU tests of FP64 density dispatches whose particles have no usable row:
around the number from which a warp takes each of them (152 on 152 SMs), more
entries within reach than a warp keeps (512), lists that stay with a block
beside them (more than twelve times the queue, or 16384 entries), first guesses
of h that every pass outgrows, and sources that add nothing; FP64 hydro sums of
particles without rows; against the oracle.

Tolerances: FP64 1e-11, as in test_gpu_functors.py; Omega, div v and |rot v| as
sums, to 1e-11 of the sum of their terms' magnitudes (see test_gpu_rowless.py).
"""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as orc
from research_codes_gb300 import abi, functors
from test_gpu_edge_values import _ball, _hydro
from test_gpu_rowless import _batch, _magnitudes

pytestmark = pytest.mark.gpu


def _check(epi, epj, eta, add_nothing=None):
    n_i = [len(a) for a in epi]
    lists = epj if add_nothing is None else [np.concatenate([b[:len(b) // 2], add_nothing, b[len(b) // 2:]]) for b in epj]
    out = [np.zeros(n, abi.Density) for n in n_i]
    with functors.Context(precision="fp64", eta=eta) as ctx:
        for _ in range(2):   # the second on used buffers and counters
            functors.DispatchKernel_Dens(ctx, 0, len(epi), epi, n_i, lists, [len(b) for b in lists])
            functors.RetrieveKernel_Dens(ctx, 0, len(epi), n_i, out)
    got = np.concatenate(out)
    refs = [orc.density(a, b, eta=eta, ksr_max=0.0) for a, b in zip(epi, epj)]
    ref = np.concatenate(refs)
    mag = np.concatenate([_magnitudes(a, b, r) for a, b, r in zip(epi, epj, refs) if len(a)])
    for f in ("dens", "ksr"):
        assert rel_err(got[f], ref[f], 1e-3).max() < 1e-11, f
    assert (np.abs(1.0 / got["grdh"] - 1.0 / ref["grdh"]) < 1e-11 * (1.0 + mag[:, 0])).all()
    for f, m in (("divv", mag[:, 1]), ("rotv", mag[:, 2])):
        assert (np.abs(got[f] / got["grdh"] - ref[f] / ref["grdh"]) < 1e-11 * m).all(), f
    assert np.array_equal(got["np"], ref["np"]) and np.array_equal(got["itr"], ref["itr"])


@pytest.mark.parametrize("spoil", [151, 152, 153, 800])
def test_around_the_least_number_for_warps(spoil):
    _check(*_batch([200] * 4, 300, 1.18, 0.5, 7, spoil), 1.18)


# 3.0: the first pass reaches most of the ball, more than a warp keeps
@pytest.mark.parametrize("eta,guess", [(1.6, 1.0), (1.18, 0.5), (1.18, 1.6), (1.6, 1.6), (1.18, 3.0)])
@pytest.mark.parametrize("sizes,n_j", [([700], 700), ([1, 31, 33, 0, 64, 600], 1700), ([20] * 35, 127)])
def test_first_guesses(sizes, n_j, eta, guess):
    _check(*_batch(sizes, n_j, eta, guess, 9), eta)


@pytest.mark.parametrize("n_long", [16384, 16385, 20000])
def test_long_lists_beside_the_others(n_long):
    epi, epj = _batch([200] * 4, 300, 1.18, 0.5, 11)
    a, b = _batch([3], n_long, 1.6, 1.2, 13)
    _check(epi[:2] + a + epi[2:], epj[:2] + b + epj[2:], 1.18)


@pytest.mark.parametrize("n_long", [2400, 2401])
def test_long_lists_by_the_length_of_the_queue(n_long):
    """200 without a row: a warp takes lists of up to 2400 entries."""
    epi, epj = _batch([160], 300, 1.18, 0.5, 17)
    a, b = _batch([40], n_long, 1.18, 0.5, 19)
    _check(epi + a, epj + b, 1.18)


@pytest.mark.parametrize("field,value", [("mass", np.inf), ("mass", np.nan), ("pos", np.nan), ("all", 1e39), ("all", 1e200),
                                         ("all", np.inf)])
@pytest.mark.parametrize("guess", [0.5, 1.6])
def test_sources_that_add_nothing(field, value, guess):
    """Beyond every support (in y and z where x is NaN), or infinitely far."""
    bad = np.zeros(5, abi.DensityEPJ)
    bad["id"] = 10 ** 6 + np.arange(5)
    bad["mass"] = value if field == "mass" else 1.0
    bad["pos"] = [30.0, 60.0, 80.0]
    if field == "pos":
        bad["pos"][:, 0] = value
    if field == "all":
        bad["pos"][:, 1] = value
    epi, epj = _batch([350] * 2, 500, 1.18, guess, 15)
    _check(epi, epj, 1.18, bad)


@pytest.mark.parametrize("n_i", [1, 40, 700])
@pytest.mark.parametrize("n_j,neighbours", [(700, 200), (700, 700), (4000, 300), (4000, 3000)])
def test_hydro_sums_of_particles_without_rows(n_i, n_j, neighbours):
    """A few to all entries of a round of a block (1024) within reach."""
    epi, epj, near = _ball(n_i, n_j, 17 * n_i + n_j, neighbours=neighbours)
    out, ref = _hydro("fp64", epi, epj), orc.hydro(epi, epj)
    for f in ("acch", "accg", "udot", "vsmx", "diffu"):
        assert rel_err(out[f], ref[f], 1e-3).max() < 1e-11, f
