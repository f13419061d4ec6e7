"""GPU tests of the gravity lists cut into parts (several work units per
i-group of a small call) against the oracle: list lengths around the smallest
part (128 entries) and the tile (32), and group sizes that leave one and many
lanes per particle.  Tolerances as in test_gpu_functors.py: FP64 1e-11, FP32C
1e-5, floor 1e-3."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as orc
from research_codes_gb300 import abi, functors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i,n_j", [(1, 1), (3, 31), (5, 255), (1, 256), (33, 257), (40, 20000), (700, 1500)])
def test_gravity_parts(prec, n_i, n_j):
    rng = np.random.default_rng(n_i + n_j)
    epi, epj = np.zeros(n_i, abi.GravityEPI), np.zeros(n_j, abi.GravityEPJ)
    epj["pos"] = rng.normal(size=(n_j, 3)) * 50.0 + 3.0e3
    epj["mass"] = rng.uniform(0.5, 1.5, n_j)
    epj["eps2"] = rng.uniform(5.0, 10.0, n_j)
    epi["pos"] = rng.normal(size=(n_i, 3)) * 50.0 + 3.0e3
    epi["eps2"] = rng.uniform(5.0, 10.0, n_i)
    out = np.zeros(n_i, abi.Gravity)
    with functors.Context(precision=prec) as ctx:
        functors.calcGravity(ctx)(epi, n_i, epj, n_j, out)
    ref = orc.gravity(epi, epj)
    for f in ("acc", "pot", "eta"):
        assert rel_err(out[f], ref[f], 1e-3).max() < (1e-11 if prec == "fp64" else 1e-5), f
