"""GPU tests of a particle system whose context changes its precision between
evaluations (sph_context_set_precision): every buffer that depends on the
precision fits both, and the evaluation is the one of a system created in the
precision it runs in.

Tolerance: the two systems run the same kernels on the same inputs.  FP64 sums
run in list order, which a list build may change: 1e-12 (n eps for ~1e3 terms),
floor 1e-3 of the field's largest value.  FP32C: 1e-5, as every FP32C parity
test.
"""
import numpy as np
import pytest

from conftest import rel_err
from research_codes_gb300 import functors, ic
from research_codes_gb300.system import ParticleSystem, state_from_ic

pytestmark = pytest.mark.gpu

FIELDS = ("dens", "ksr", "acc", "accg2", "pot", "eta", "udot", "vsmx")


def _state(n):
    return state_from_ic(ic.polytrope(n, 1.0, 1.0, 1.5, seed=3, eta=1.18))


def _evaluate(sys, s):
    sys.upload(s)
    sys.compute_forces()
    sys.compute_forces()   # a replay, where graphs are used
    return {f: sys.download(f) for f in FIELDS}


# the FP64 gravity lists are cut into eight parts at 700 and 5003 particles, into four at 100003 (FP32C: whole)
@pytest.mark.parametrize("n,use_graph", [(700, 0), (700, 1), (5003, 0), (5003, 1), (100003, 1)])
@pytest.mark.parametrize("first,then", [("fp32c", "fp64"), ("fp64", "fp32c")])
def test_precision_changes_after_creation(first, then, n, use_graph):
    s = _state(n)
    with functors.Context(precision=then, eta=1.18) as ctx:
        sys = ParticleSystem(ctx, n, n_group=64, use_graph=use_graph, ksr_max_mode=0)
        ref = _evaluate(sys, s)
        sys.close()
    with functors.Context(precision=first, eta=1.18) as ctx:
        sys = ParticleSystem(ctx, n, n_group=64, use_graph=use_graph, ksr_max_mode=0)
        _evaluate(sys, s)
        ctx.set_precision(then)
        got = _evaluate(sys, s)
        ctx.set_precision(first)
        _evaluate(sys, s)
        sys.close()
    tol = 1e-12 if then == "fp64" else 1e-5
    for f in FIELDS:
        assert rel_err(got[f], ref[f], 1e-3).max() < tol, (f, rel_err(got[f], ref[f], 1e-3).max())
