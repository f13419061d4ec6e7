"""GPU tests of functor calls with values at the edges of what the row kernels
(csrc/rows.cuh, csrc/density_rows.cuh) hold in FP32: coincident particles,
sources far outside the FP32 range of a squared distance, values that are not
finite.

Expected values are the oracle's, on the list without the sources that add
nothing where the oracle's own arithmetic makes NaN of them.  Tolerances as in
test_gpu_functors.py (same quantities, same reasons): FP64 1e-11, FP32C 1e-5.
"""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as orc
from research_codes_gb300 import abi, functors

pytestmark = pytest.mark.gpu

ETA = 1.18
TOL = {"fp64": 1e-11, "fp32c": 1e-5}


def _ball(n_i, n_j, seed, centre=30.0, neighbours=40.0):
    """HydroEPI / HydroEPJ of a uniform ball: the n_i sources nearest to one of
    them as targets, sound speeds of order one, velocities of order one."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n_j, 3))
    x *= (rng.uniform(size=n_j) ** (1.0 / 3.0) / np.linalg.norm(x, axis=1))[:, None]
    epj = np.zeros(n_j, abi.HydroEPJ)
    epj["id"], epj["pos"], epj["vel"] = np.arange(n_j), x + centre, rng.normal(size=(n_j, 3))
    epj["mass"] = rng.uniform(0.5, 1.5, n_j) / n_j
    epj["ksr"] = (neighbours / n_j) ** (1.0 / 3.0) * rng.uniform(0.8, 1.2, n_j)
    epj["hinv"] = 1.0 / epj["ksr"]
    epj["dens"] = 0.3 + 0.1 * (x ** 2).sum(1)
    epj["pres"] = 1.0 - 0.5 * (x ** 2).sum(1)
    epj["presc"] = epj["pres"] / epj["dens"] ** 2
    epj["bswt"], epj["alph"], epj["alphu"] = rng.uniform(0.0, 0.5, n_j), 1.0, 0.05
    epj["vsnd"] = rng.uniform(1.0, 1.3, n_j)
    epj["thrm"], epj["eta"] = epj["pres"] / epj["dens"], 0.1 * epj["ksr"] ** 2
    near = np.argsort(((x - x[0]) ** 2).sum(1), kind="stable")[:n_i]
    epi = np.zeros(n_i, abi.HydroEPI)
    for f in epi.dtype.names:
        epi[f] = epj[f][near]
    return epi, epj, near


def _hydro(prec, epi, epj):
    out = np.zeros(len(epi), abi.Hydro)
    with functors.Context(precision=prec, eta=ETA) as ctx:
        functors.calcHydro(ctx)(epi, len(epi), epj, len(epj), out)
    return out


# one target (items of one particle) and groups; lists of one warp and of a block
SIZES = [(1, 700), (1, 4000), (40, 700), (40, 4000)]


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i,n_j", SIZES)
@pytest.mark.parametrize("where,speed", [(1e16, 50.0), (1e16, 1e4), (1e3, 1e17)])
def test_signal_velocity_of_far_and_fast_sources(prec, n_i, n_j, where, speed):
    """The largest signal velocity is that of a source beyond the range in
    which FP32 bounds it."""
    epi, epj, near = _ball(n_i, n_j, 17 * n_i + n_j)
    far = epj[~np.isin(epj["id"], near)][-1:].copy()
    far["pos"] = epi["pos"][0] + [where, 0.0, 0.0]
    far["vel"] = [-speed, 0.0, 0.0]
    far["id"] += 10 ** 6
    lst = np.concatenate([epj[: n_j // 2], far, epj[n_j // 2:]])
    out, ref = _hydro(prec, epi, lst), orc.hydro(epi, lst)
    assert (ref["vsmx"] > 2.0 * speed).all()
    assert rel_err(out["vsmx"], ref["vsmx"], 1e-3).max() < TOL[prec]


# (FP32C forms the square of the separation in FP32: 1e-18 at least; 6000 targets: items of several in FP64)
@pytest.mark.parametrize("prec,sep", [("fp32c", 1e-9), ("fp32c", 1e-18), ("fp64", 1e-9), ("fp64", 1e-18), ("fp64", 1e-22)])
@pytest.mark.parametrize("n_i,n_j", SIZES + [(6000, 6000)])
def test_signal_velocity_of_close_particles(prec, sep, n_i, n_j):
    """Two distinct particles that approach each other closer than the FP32
    frame of their group resolves, or than FP32 squares."""
    epi, epj, near = _ball(n_i, n_j, 19 * n_i + n_j, centre=0.0)
    t = n_i // 2
    epj["pos"] -= epi["pos"][t]
    epi["pos"] -= epi["pos"][t]
    far = np.flatnonzero(~np.isin(epj["id"], near))
    k = far[-1] if len(far) else near[-1]
    epj["id"][k] = 10 ** 6
    epj["pos"][k] = [sep, 0.0, 0.0]
    epj["vel"][k] = epi["vel"][t] - [40.0, 0.0, 0.0]
    out, ref = _hydro(prec, epi, epj), orc.hydro(epi, epj)
    assert ref["vsmx"][t] > 120.0
    assert rel_err(out["vsmx"], ref["vsmx"], 1e-3).max() < TOL[prec]


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i,n_j", SIZES)
def test_signal_velocity_ignores_nan_terms(prec, n_i, n_j):
    """Sources without a sound speed beyond every support, listed before the
    others, leave the maximum over the others as it is."""
    epi, epj, near = _ball(n_i, n_j, 23 * n_i + n_j)
    nan = epj[:33].copy()
    nan["id"] += 10 ** 6
    nan["pos"] += 50.0
    nan["vsnd"] = np.nan
    out, ref = _hydro(prec, epi, np.concatenate([nan, epj])), orc.hydro(epi, epj)
    assert rel_err(out["vsmx"], ref["vsmx"], 1e-3).max() < TOL[prec]


@pytest.mark.parametrize("n_i,n_j", [(1, 700), (1, 4000), (5, 2000), (40, 4000), (6000, 6000)])
@pytest.mark.parametrize("which", [0, -1])
def test_hydro_fp64_of_a_target_without_a_position(n_i, n_j, which):
    """NaN in one coordinate of a target: its sums are NaN, which the call
    reports, and the others' are what they are without it."""
    epi, epj, near = _ball(n_i, n_j, 29 * n_i + n_j)
    epi["pos"][which, 0] = np.nan
    out = np.zeros(n_i, abi.Hydro)
    with functors.Context(precision="fp64", eta=ETA) as ctx:
        with pytest.raises(abi.SPHError, match="NONFINITE"):
            functors.calcHydro(ctx)(epi, n_i, epj, n_j, out)
    ref = orc.hydro(epi, epj)
    ok = np.arange(n_i) != which % n_i
    for f in ("acch", "accg", "udot", "diffu"):
        assert np.isnan(out[f][which]).all(), f
        if ok.any():
            assert rel_err(out[f][ok], ref[f][ok], 1e-3).max() < 1e-11, f
    if ok.any():
        assert rel_err(out["vsmx"][ok], ref["vsmx"][ok], 1e-3).max() < 1e-11


def _density_inputs(epi, epj, guess=1.0):
    """DensityEPI / DensityEPJ of hydro inputs; guess: first h over theirs."""
    di, dj = np.zeros(len(epi), abi.DensityEPI), np.zeros(len(epj), abi.DensityEPJ)
    mass = dict(zip(epj["id"].tolist(), epj["mass"].tolist()))
    for f in ("id", "pos", "vel"):
        di[f], dj[f] = epi[f], epj[f]
    dj["mass"] = epj["mass"]
    di["mass"] = [mass[k] for k in epi["id"].tolist()]
    di["ksr"] = guess * epi["ksr"]
    di["rs"] = 1.1 * di["ksr"]
    return di, dj


def _density(prec, di, dj):
    out = np.zeros(len(di), abi.Density)
    with functors.Context(precision=prec, eta=ETA) as ctx:
        functors.calcDensity(ctx)(di, len(di), dj, len(dj), out)
    return out


# the first guess of h near (rows) and far below the final one (sweeps)
@pytest.mark.parametrize("guess", [1.0, 0.5])
@pytest.mark.parametrize("far", [1e39, 1e200, np.inf, -np.inf])
@pytest.mark.parametrize("n_i,n_j", [(1, 40), (1, 700), (5, 4000), (40, 700)])
def test_fp64_sources_at_infinite_distance(n_i, n_j, far, guess):
    """Sources whose coordinates, or their squares, leave the FP32 or FP64
    range add nothing to FP64 sums."""
    epi, epj, near = _ball(n_i, n_j, 31 * n_i + n_j, neighbours=min(40.0, n_j))
    out_of = epj[:3].copy()
    out_of["id"] += 10 ** 6
    out_of["pos"][:, 1] = far
    lst = np.concatenate([epj[: n_j // 2], out_of, epj[n_j // 2:]])
    di, dj = _density_inputs(epi, epj, guess)
    out = _density("fp64", di, _density_inputs(epi, lst, guess)[1])
    ref = orc.density(di, dj, eta=ETA, ksr_max=0.0)
    for f in ("dens", "ksr", "grdh", "divv", "rotv"):
        assert rel_err(out[f], ref[f], 1e-2).max() < 1e-11, f
    assert np.array_equal(out["np"], ref["np"]) and np.array_equal(out["itr"], ref["itr"])
    h, href = _hydro("fp64", epi, lst), orc.hydro(epi, epj)
    for f in ("acch", "accg", "udot", "diffu"):
        assert rel_err(h[f], href[f], 1e-3).max() < 1e-11, f


@pytest.mark.parametrize("n_j", [40, 700])
@pytest.mark.parametrize("n_i", [1, 5])
def test_fp64_target_at_infinite_distance(n_i, n_j):
    """A target whose squared distances leave the FP64 range: no force, and its
    neighbours in the call keep theirs."""
    epi, epj, near = _ball(n_i, n_j, 37 * n_i + n_j)
    ref = orc.hydro(epi, epj)
    epi["pos"][0, 0] = 1e200
    out = _hydro("fp64", epi, epj)
    for f in ("acch", "accg", "udot", "diffu"):
        assert not out[f][0].any(), f
        if n_i > 1:
            assert rel_err(out[f][1:], ref[f][1:], 1e-3).max() < 1e-11, f


@pytest.mark.parametrize("guess", [1.0, 0.5])
@pytest.mark.parametrize("n_i,n_j", [(1, 40), (1, 700), (5, 4000), (40, 700)])
def test_fp32c_sources_beyond_the_range_of_a_square(n_i, n_j, guess):
    """FP32C density: sources whose squared distance is infinite in FP32 add
    nothing, also to particles that sweep the whole list (first guess of h far
    below the final one)."""
    epi, epj, near = _ball(n_i, n_j, 41 * n_i + n_j, neighbours=min(40.0, n_j))
    out_of = epj[:3].copy()
    out_of["id"] += 10 ** 6
    out_of["pos"][:, 1] = 1e20
    lst = np.concatenate([epj[: n_j // 2], out_of, epj[n_j // 2:]])
    di, dj = _density_inputs(epi, epj, guess)
    out = _density("fp32c", di, _density_inputs(epi, lst, guess)[1])
    ref = orc.density(di, dj, eta=ETA, ksr_max=0.0)
    for f in ("dens", "ksr", "grdh"):
        assert rel_err(out[f], ref[f], 1e-3).max() < 1e-5, f
    for f in ("divv", "rotv"):
        assert rel_err(out[f], ref[f], 1e-2).max() < 1e-4, f


# first guesses of h above the final one (rows) and far below it (sweeps)
@pytest.mark.parametrize("prec,guess", [("fp32c", 1.2), ("fp32c", 0.5), ("fp64", 1.2), ("fp64", 0.5)])
@pytest.mark.parametrize("field,value", [("mass", 1e39), ("mass", np.inf), ("mass", np.nan), ("pos", np.nan)])
@pytest.mark.parametrize("n_i,n_j", [(1, 40), (1, 700), (40, 700), (5, 4000)])
def test_density_of_unusable_sources_beyond_the_support(n_i, n_j, field, value, prec, guess):
    """Sources beyond the support add nothing, whatever their mass (1e39: infinite
    in FP32), nor does one that has no x but lies beyond it in y and z.  One
    target has such a source in its row (at 1.02 times the first guess of h)."""
    epi, epj, near = _ball(n_i, n_j, 47 * n_i + n_j, neighbours=min(40.0, n_j))
    di, dj = _density_inputs(epi, epj)
    di["ksr"] = guess * orc.density(di, dj, eta=ETA, ksr_max=0.0)["ksr"]
    di["rs"] = 1.1 * di["ksr"]
    bad = np.zeros(4, abi.DensityEPJ)
    bad["id"] = 10 ** 6 + np.arange(4)
    bad["mass"] = value if field == "mass" else 1.0
    bad["pos"] = di["pos"][0] + np.array([0.0, 6.0, 8.0])
    if n_i == 1 and guess > 1.0 and field == "mass":
        bad["pos"][0] = di["pos"][0] + 1.02 * di["ksr"][0] * np.array([0.0, 0.6, 0.8])
    if field == "pos":
        bad["pos"][:, 0] = value
    ref = orc.density(di, dj, eta=ETA, ksr_max=0.0)
    out = _density(prec, di, np.concatenate([dj[: n_j // 2], bad, dj[n_j // 2:]]))
    for f in ("dens", "ksr", "grdh"):
        assert rel_err(out[f], ref[f], 1e-3).max() < TOL[prec], f
    for f in ("divv", "rotv"):
        assert rel_err(out[f], ref[f], 1e-2).max() < 10 * TOL[prec], f


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i,n_j", [(1, 40), (1, 700), (40, 700), (5, 4000)])
@pytest.mark.parametrize("h", [1e-16, 1e-39])
def test_hydro_sources_with_a_tiny_support(n_i, n_j, h, prec):
    """Sources whose h lies below the range of the row tests reach no target
    but those in whose supports they are (h^-4 is infinite in FP32)."""
    epi, epj, near = _ball(n_i, n_j, 53 * n_i + n_j)
    tiny = epj[:3].copy()
    tiny["id"] += 10 ** 6
    tiny["pos"] = epi["pos"][0] + np.array([0.0, 6.0, 8.0])
    tiny["ksr"], tiny["hinv"] = h, 1.0 / h
    out, ref = _hydro(prec, epi, np.concatenate([epj[: n_j // 2], tiny, epj[n_j // 2:]])), orc.hydro(epi, epj)
    for f in ("acch", "accg", "udot"):
        assert rel_err(out[f], ref[f], 1e-3).max() < TOL[prec], f
    assert rel_err(out["diffu"], ref["diffu"], 1e-2).max() < 10 * TOL[prec]


@pytest.mark.parametrize("n_i,n_j", SIZES)
@pytest.mark.parametrize("speed", [1e39, 1e200, np.inf])
@pytest.mark.parametrize("who", ["source", "target"])
def test_fp32c_velocities_beyond_the_fp32_range(n_i, n_j, speed, who):
    """An approach faster than FP32 holds is an infinite signal velocity, which
    the call reports."""
    epi, epj, near = _ball(n_i, n_j, 59 * n_i + n_j)
    far = epj[~np.isin(epj["id"], near)][-1:].copy()
    far["id"] += 10 ** 6
    far["pos"] = epi["pos"][0] + [20.0, 1.0, 1.0]
    lst = np.concatenate([epj[: n_j // 2], far, epj[n_j // 2:]])
    if who == "source":
        lst["vel"][n_j // 2] = [-speed, 0.0, 0.0]
    else:
        epi["vel"][0] = [speed, 0.0, 0.0]
    out = np.zeros(n_i, abi.Hydro)
    with functors.Context(precision="fp32c", eta=ETA) as ctx:
        with pytest.raises(abi.SPHError, match="NONFINITE"):
            functors.calcHydro(ctx)(epi, n_i, lst, len(lst), out)
    assert np.isinf(out["vsmx"] if who == "source" else out["vsmx"][0]).all()


@pytest.mark.parametrize("n_i,n_j", [(1, 40), (1, 700), (5, 900)])
def test_fp64_density_of_a_negative_sum(n_i, n_j):
    """Sources of negative mass that outweigh the others make a negative h,
    which no row radius covers: the particle sweeps the list.  The same with 200
    massless sources beside the target, whose row overflows (FP64 sums in
    another order: 1e-9 of what they grow to)."""
    epi, epj, near = _ball(n_i, n_j, 43 * n_i + n_j, neighbours=min(40.0, n_j))
    di, dj = _density_inputs(epi, epj)
    dj["mass"][near] *= -50.0
    extra = np.repeat(dj[near[:1]], 200)
    extra["id"] = 10 ** 6 + np.arange(200)
    extra["mass"] = 0.0
    extra["pos"] += 1e-3 * np.random.default_rng(1).normal(size=(200, 3))
    out, ref = _density("fp64", di, dj), _density("fp64", di, np.concatenate([dj, extra]))
    assert (ref["ksr"] < 0.0).any()
    for f in ("dens", "ksr"):
        assert rel_err(out[f], ref[f], 1e-3).max() < 1e-9, f


@pytest.mark.parametrize("n_i,n_j", SIZES)
def test_fp64_squares_below_the_normal_range(n_i, n_j):
    """FP64 mode: 1/sqrt of squares that are subnormal (a separation of 1e-160,
    a softening of 1e-155) is finite."""
    epi, epj, near = _ball(n_i, n_j, 61 * n_i + n_j, centre=0.0)
    epj["pos"] -= epi["pos"][0]
    epi["pos"] -= epi["pos"][0]
    k = np.flatnonzero(~np.isin(epj["id"], near))[-1]
    epj["pos"][k] = [1e-160, 0.0, 0.0]
    epj["vel"][k] = epi["vel"][0]
    epj["vel"][k, 0] -= 40.0
    # (subnormal squares have few digits: 1e-4 where they set the value)
    out, ref = _hydro("fp64", epi, epj), orc.hydro(epi, epj)
    assert ref["vsmx"][0] > 100.0
    assert rel_err(out["vsmx"], ref["vsmx"], 1e-3).max() < 1e-4
    di, dj = _density_inputs(epi, epj)
    out, ref = _density("fp64", di, dj), orc.density(di, dj, eta=ETA, ksr_max=0.0)
    for f in ("dens", "ksr", "grdh", "divv", "rotv"):
        assert rel_err(out[f], ref[f], 1e-2).max() < 1e-10, f
    gi, gj = np.zeros(n_i, abi.GravityEPI), np.zeros(n_j, abi.GravityEPJ)
    gi["pos"], gi["eps2"] = epi["pos"], 1e-310
    gj["pos"], gj["mass"], gj["eps2"] = epj["pos"], epj["mass"], 1e-310
    gj["pos"][k] = 0.5
    got = np.zeros(n_i, abi.Gravity)
    with functors.Context(precision="fp64", eta=ETA) as ctx:
        try:
            functors.calcGravity(ctx)(gi, n_i, gj, n_j, got)
        except abi.SPHError:   # (the cube in the accelerations is infinite)
            pass
    pot = orc.gravity(gi, gj)["pot"]
    assert np.isfinite(pot).all() and rel_err(got["pot"], pot, 1e-3).max() < 1e-10
