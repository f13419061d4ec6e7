"""GPU tests of the neighbour-row kernels (csrc/rows.cuh, csrc/density_rows.cuh)
at the sizes where they can go wrong, against the oracle: rows of 0 to more
than ROW_CAP entries, list lengths around a streaming step (64 entries) and
around the length that a whole block marks (4096), group sizes that
leave several lanes per particle, first guesses of h that leave the row
radius, and coordinates whose squares leave the FP32 range (FP64 mode).

Tolerances as in test_gpu_functors.py (same quantities, same reasons): FP64
1e-11, FP32C 1e-5 (1e-4 on div v and |rot v|), floors 1e-3 (1e-2).
"""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as orc
from research_codes_gb300 import abi, functors

pytestmark = pytest.mark.gpu

ETA = 1.18


def _cloud(n_i, n_j, seed, guess=1.0, neighbours=50.0, scale=1.0):
    """n_i targets among n_j sources of a uniform ball; h for `neighbours`
    sources at the true density times `guess`."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n_j, 3))
    x *= (rng.uniform(size=n_j) ** (1.0 / 3.0) / np.linalg.norm(x, axis=1))[:, None]
    x = (x + 30.0) * scale
    v = rng.normal(size=(n_j, 3))
    m = rng.uniform(0.5, 1.5, n_j) * scale ** 3 / n_j
    h = scale * (neighbours / n_j) ** (1.0 / 3.0)
    near = np.argsort(((x - x[0]) ** 2).sum(1), kind="stable")[:n_i]
    epi = np.zeros(n_i, abi.DensityEPI)
    epj = np.zeros(n_j, abi.DensityEPJ)
    epj["id"], epj["mass"], epj["pos"], epj["vel"] = np.arange(n_j), m, x, v
    for k in ("id", "mass", "pos", "vel"):
        epi[k] = epj[k][near]
    epi["ksr"] = h * guess * rng.uniform(0.97, 1.03, n_i)
    epi["rs"] = 1.1 * epi["ksr"]
    return epi, epj


def _check(prec, epi, epj):
    out = np.zeros(len(epi), abi.Density)
    with functors.Context(precision=prec, eta=ETA) as ctx:
        functors.calcDensity(ctx)(epi, len(epi), epj, len(epj), out)
    ref = orc.density(epi, epj, eta=ETA, ksr_max=0.0)
    tol, dtol = (1e-11, 1e-11) if prec == "fp64" else (1e-5, 1e-4)
    for f in ("dens", "ksr", "grdh"):
        assert rel_err(out[f], ref[f], 1e-3).max() < tol, f
    for f in ("divv", "rotv"):
        assert rel_err(out[f], ref[f], 1e-2).max() < dtol, f
    if prec == "fp64":
        assert np.array_equal(out["np"], ref["np"]) and np.array_equal(out["itr"], ref["itr"])
    else:
        assert np.abs(out["np"] - ref["np"]).max() <= 1


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i,n_j,guess,neighbours", [
    (1, 60, 1.0, 20.0), (3, 64, 1.0, 30.0), (32, 65, 1.0, 30.0), (33, 500, 1.0, 50.0),
    (7, 4096, 1.0, 50.0), (37, 4097, 1.0, 50.0),     # the last list of one warp, the first of a block
    (40, 4000, 1.0, 160.0), (40, 9000, 1.0, 160.0),   # rows beyond their capacity
    (40, 3000, 0.9, 50.0), (40, 3000, 1.25, 50.0),   # h leaves the row radius upwards and downwards
    (700, 5000, 1.0, 50.0),
])
def test_density_rows(prec, n_i, n_j, guess, neighbours):
    _check(prec, *_cloud(n_i, n_j, 11 * n_i + n_j, guess, neighbours))


@pytest.mark.parametrize("scale", [1.0e-20, 1.0e25])
def test_density_fp64_beyond_the_fp32_range(scale):
    _check("fp64", *_cloud(20, 600, 5, scale=scale))
