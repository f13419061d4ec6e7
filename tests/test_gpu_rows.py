"""GPU tests of the neighbour-row kernels (csrc/rows.cuh and the sums over rows)
at the sizes where they can go wrong, against the oracle: rows of 0 to more
than ROW_CAP entries, list lengths around a streaming step (64 entries) and
around the length that a whole block marks (1536), group sizes that
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
    (7, 1536, 1.0, 50.0), (37, 1537, 1.0, 50.0), (7, 4097, 1.0, 50.0),   # the last list of one warp, the first of a block
    (40, 4000, 1.0, 160.0), (40, 9000, 1.0, 160.0),   # rows beyond their capacity
    (40, 3000, 0.9, 50.0), (40, 3000, 1.25, 50.0),   # h leaves the row radius upwards and downwards
    (700, 5000, 1.0, 50.0),
])
def test_density_rows(prec, n_i, n_j, guess, neighbours):
    _check(prec, *_cloud(n_i, n_j, 11 * n_i + n_j, guess, neighbours))


@pytest.mark.parametrize("scale", [1.0e-20, 1.0e25])
def test_density_fp64_beyond_the_fp32_range(scale):
    _check("fp64", *_cloud(20, 600, 5, scale=scale))


def _hydro_cloud(n_i, n_j, seed, neighbours=50.0, scale=1.0, speed=1.0):
    """Hydro inputs on the same ball: a pressure gradient, sound speeds of
    order one and random velocities of `speed` times that."""
    rng = np.random.default_rng(seed + 1)
    den, src = _cloud(n_i, n_j, seed, neighbours=neighbours, scale=scale)
    out = []
    for d, dt in ((den, abi.HydroEPI), (src, abi.HydroEPJ)):
        a = np.zeros(len(d), dt)
        a["id"], a["pos"], a["vel"] = d["id"], d["pos"], speed * scale * d["vel"]
        if dt is abi.HydroEPJ:
            a["mass"] = d["mass"]
        r2 = ((a["pos"] / scale - 30.0) ** 2).sum(1)
        a["ksr"] = scale * (neighbours / n_j) ** (1.0 / 3.0) * (0.8 + 0.4 * ((a["id"] * 37) % 101) / 101.0)
        a["hinv"] = 1.0 / a["ksr"]
        a["dens"] = 0.3 + 0.1 * r2
        a["pres"] = scale ** 2 * (1.0 - 0.5 * r2)
        a["presc"] = a["pres"] / a["dens"] ** 2
        a["bswt"] = 0.5 * ((a["id"] * 13) % 7) / 7.0
        a["vsnd"] = scale * (1.0 + 0.3 * ((a["id"] * 29) % 53) / 53.0)
        a["alph"], a["alphu"] = 1.0, 0.05
        a["thrm"] = a["pres"] / a["dens"]
        a["eta"] = 0.1 * a["ksr"] ** 2
        out.append(a)
    return out


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i,n_j,neighbours,speed", [
    (1, 40, 20.0, 1.0), (5, 64, 20.0, 0.0), (33, 65, 20.0, 1.0), (33, 1000, 50.0, 1e-3),
    (7, 1536, 50.0, 1.0), (37, 1537, 50.0, 30.0), (7, 4097, 50.0, 1.0),   # the last list of one warp, the first of a block
    (40, 3000, 160.0, 1.0), (40, 9000, 160.0, 1.0),  # rows beyond their capacity
])
def test_hydro_rows(prec, n_i, n_j, neighbours, speed):
    epi, epj = _hydro_cloud(n_i, n_j, 7 * n_i + n_j, neighbours, speed=speed)
    out = np.zeros(n_i, abi.Hydro)
    with functors.Context(precision=prec, eta=ETA) as ctx:
        functors.calcHydro(ctx)(epi, n_i, epj, n_j, out)
    ref = orc.hydro(epi, epj)
    tol = 1e-11 if prec == "fp64" else 1e-5
    for f in ("acch", "accg", "udot", "vsmx"):
        assert rel_err(out[f], ref[f], 1e-3).max() < tol, f
    assert rel_err(out["diffu"], ref["diffu"], 1e-2).max() < (tol if prec == "fp64" else 1e-4)


@pytest.mark.parametrize("scale", [1.0e-20, 1.0e25])
def test_hydro_fp64_beyond_the_fp32_range(scale):
    epi, epj = _hydro_cloud(20, 600, 5, scale=scale)
    out = np.zeros(20, abi.Hydro)
    with functors.Context(precision="fp64", eta=ETA) as ctx:
        functors.calcHydro(ctx)(epi, 20, epj, 600, out)
    ref = orc.hydro(epi, epj)
    for f in ("acch", "accg", "udot", "vsmx", "diffu"):
        assert rel_err(out[f], ref[f], 1e-3).max() < 1e-11, f


@pytest.mark.parametrize("n_walk,n_j", [(3, 12), (2, 30000), (40, 9000)])
def test_staged_arrays_by_size(n_walk, n_j):
    """Walk arrays at odd addresses, from one short copy to several threads and
    segments (and arrays longer than one copying task): a batch gives what the
    walks give one by one (FP64 sums of the same rows: 1e-13)."""
    rng = np.random.default_rng(n_j)

    def odd(a):
        raw = np.empty(a.nbytes + 1, np.uint8)
        raw[1:] = a.view(np.uint8)
        return raw[1:].view(a.dtype)

    walks = [_cloud(7 + k, n_j + int(rng.integers(0, 50)), seed=k) for k in range(n_walk)]
    epi, epj = [odd(a) for a, _ in walks], [odd(b) for _, b in walks]
    n_i, n_js = [len(a) for a in epi], [len(b) for b in epj]
    got = [np.zeros(n, abi.Density) for n in n_i]
    with functors.Context(precision="fp64", eta=ETA) as ctx:
        functors.DispatchKernel_Dens(ctx, 0, n_walk, epi, n_i, epj, n_js)
        functors.RetrieveKernel_Dens(ctx, 0, n_walk, n_i, got)
        for k in range(n_walk):
            one = np.zeros(n_i[k], abi.Density)
            functors.calcDensity(ctx)(epi[k], n_i[k], epj[k], n_js[k], one)
            for f in ("dens", "ksr", "grdh", "divv", "rotv"):
                assert np.allclose(got[k][f], one[f], rtol=1e-13, atol=1e-13 * np.abs(one[f]).max()), (k, f)
            assert np.array_equal(got[k]["np"], one["np"])
    one = orc.density(*walks[-1], eta=ETA, ksr_max=0.0)
    assert rel_err(got[-1]["dens"], one["dens"], 1e-3).max() < 1e-11


@pytest.mark.parametrize("prec", ["fp32c", "fp64"])
@pytest.mark.parametrize("n_i", [1, 5, 9, 17, 32, 40])
def test_hydro_rows_of_a_block_equal_a_warps(prec, n_i):
    """A list one entry under and some over the length that a block marks: the
    added j-particles lie far away and raise no signal velocity, so the rows, and
    the sums in their order, are the same bit for bit."""
    epi, epj = _hydro_cloud(n_i, 1536, n_i, 50.0)
    far = np.repeat(epj[:200], 1)
    far["id"] += 10 ** 6
    far["pos"] += 500.0
    far["vsnd"] = 0.0
    far["vel"] = epj["vel"].mean(axis=0)
    keep = np.random.default_rng(n_i).permutation(1736)
    mixed = np.concatenate([epj, far])[keep]
    order = mixed[mixed["id"] < 10 ** 6]   # the same list without the far ones
    out = []
    with functors.Context(precision=prec, eta=ETA) as ctx:
        for lst in (order, mixed):
            o = np.zeros(n_i, abi.Hydro)
            functors.calcHydro(ctx)(epi, n_i, lst, len(lst), o)
            out.append(o)
    for f in ("acch", "accg", "udot", "diffu"):
        assert np.array_equal(out[0][f], out[1][f]), f
    assert (out[1]["vsmx"] >= out[0]["vsmx"]).all()
