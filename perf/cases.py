"""Performance cases: the work a user has this framework do, through its public
entry points, over the ranges it is used at.

Families (the "do" of a case):
  call     one functor call on one i-group of host arrays (functors.calcDensity,
           calcHydro, calcGravity): the drop-in call of an FDPS tree walk
  batch    one multiwalk Dispatch/Retrieve round trip over many i-groups
  device   the allocation-free gravity entry point on device buffers
  forces   a state uploaded from pinned host memory, one force evaluation of
           the particle system, its forces read back
  steps    a run started from its initial conditions: upload, first forces,
           leapfrog steps, the new state read back
  adjoint  the vector-Jacobian product of one force evaluation

Precision of the outputs: in FP32C mode the density and gravity fields and the
signal velocity are formed in single precision, and so is what a force
evaluation derives from them: a program keeps these as float32.  What the
framework forms in double or double-float arithmetic stays float64 (the hydro
functor's sums, the integrated state, everything in FP64 mode).
"""
import ctypes
import math

import numpy as np
import torch

from research_codes_gb300 import _lib, abi, functors, ic, units, walks
from research_codes_gb300.system import ParticleSystem, state_from_ic

ETA = 1.18          # ~50 neighbours: configurations 0 to 3
ETA_LARGE = 1.28    # ~64 neighbours: the large collision


def listed():
    return [
        # the smallest drop-in call: one i-group of the tests' size against its neighbour list; latency counts
        dict(name="density call 64", do="call", kind="density", precision="fp32c", n=20000, n_group=64),
        # a hydro call at the reference's group size (256), in the plain FP64 mode that parity runs use
        dict(name="hydro call 256 fp64", do="call", kind="hydro", precision="fp64", n=20000, n_group=256),
        # gravity of a caller that owns its device buffers: a few hundred targets, a direct sum over one small star
        dict(name="gravity device 500x20k", do="device", n_i=500, n_j=20000),
        # FDPS multiwalk batches at the reference's group size
        dict(name="density batch 40k", do="batch", kind="density", precision="fp32c", n=40000, n_group=256),
        dict(name="hydro batch 21k", do="batch", kind="hydro", precision="fp32c", n=21001, n_group=200),
        dict(name="gravity batch 40k", do="batch", kind="gravity", precision="fp32c", n=40000, n_group=256),
        # relaxation of one small star (configuration 0): launches and gaps count
        dict(name="forces star 10k", do="forces", config="c0", scale=1.0, precision="fp32c", n_group=64),
        # the head-on collision of two 100k stars (configuration 1), default parameters
        dict(name="steps head-on 200k", do="steps", config="c1", scale=1.0, precision="fp32c", n_group=256, steps=8),
        # the headline run: off-axis collision of 1M particles (configuration 2) at the parameters the autotuner picks
        dict(name="steps off-axis 1M", do="steps", config="c2", scale=1.0, precision="fp32c", n_group=96, steps=8),
        # the FP64 comparator run of the head-on collision, an odd size
        dict(name="steps head-on 50k fp64", do="steps", config="c1", scale=0.25003, precision="fp64", n_group=128,
             steps=2),
        # the large collision's setting (configuration 4): node quadrupoles, ~64 neighbours
        dict(name="forces quadrupole 500k", do="forces", config="c4", scale=0.125, precision="fp32c", n_group=128),
        # one backward pass of the differentiable step (configuration 3, 2 x 50k)
        dict(name="adjoint 100k", do="adjoint", config="c3", scale=1.0, precision="fp64", n_group=64),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["call", "batch", "device", "forces", "steps", "adjoint"])
    precision = rng.choice(["fp32c", "fp32c", "fp64"])
    kind = rng.choice(["density", "hydro", "gravity"])
    if do == "call":
        return dict(do=do, kind=kind, precision=precision, n=_log_uniform(rng, 1000, 50000),
                    n_group=_log_uniform(rng, 1, 256))
    if do == "batch":
        n_group = _log_uniform(rng, 16, 256)
        return dict(do=do, kind=kind, precision=precision, n=n_group * _log_uniform(rng, 8, 200), n_group=n_group)
    if do == "device":
        return dict(do=do, n_i=_log_uniform(rng, 1, 4096), n_j=_log_uniform(rng, 50, 65536))
    # particle systems: up to 1M particles in FP32C, less where a pass costs more per particle
    n_group = rng.choice([64, 96, 128, 256])
    if do == "adjoint":
        return dict(do=do, config="c3", scale=_log_uniform(rng, 3000, 100000) / 1.0e5, precision=precision,
                    n_group=64)
    config = rng.choice(["c0", "c1", "c2", "c4"])
    full = {"c0": 1.0e4, "c1": 2.0e5, "c2": 1.0e6, "c4": 4.0e6}[config]
    most = {"c0": 2.0e4, "c1": 2.0e5, "c2": 1.0e6, "c4": 5.0e5}[config]
    if precision == "fp64":
        most = min(most, 5.0e4)
    case = dict(do=do, config=config, scale=_log_uniform(rng, 2000, most) / full, precision=precision,
                n_group=n_group)
    if do == "steps":
        case["steps"] = rng.randint(1, 8)
    return case


# ---------------------------------------------------------------- inputs
def _star(n, seed):
    """A rotating, expanding n = 1.5 star with noise and the hydro fields of an
    evolved state (Balsara switch, viscosity and softening coefficients)."""
    rng = np.random.default_rng(seed)
    s = ic.polytrope(n, 1.0, 1.0, 1.5, seed=seed, eta=ETA)
    s["vel"] = np.cross([0.0, 0.0, 2e-3], s["pos"]) + 1e-4 * s["pos"] + rng.normal(scale=1.0, size=s["pos"].shape)
    s["id"] = rng.permutation(n)
    s["pres"] = s["dens"] * s["uene"] / units.EOS_N
    s["vsnd"] = np.sqrt(units.GAMMA * s["pres"] / s["dens"])
    s["grdh"] = rng.uniform(0.9, 1.1, n)
    s["bswt"] = rng.uniform(0.0, 1.0, n)
    s["alph"] = rng.uniform(0.1, 2.0, n)
    s["alphu"] = rng.uniform(0.0, 0.1, n)
    s["eta"] = 4.0 * (s["ksr"] / units.KSRH) ** 2 * s["grdh"]
    return s


def _groups(pos, n_group):
    """The i-groups of a tree walk: maximal octree cells of at most n_group particles."""
    keys = walks.morton_keys(pos)
    order = np.argsort(keys, kind="stable")
    keys = keys[order]
    groups, todo = [], [(0, len(keys), 0)]
    while todo:
        a, b, level = todo.pop()
        if b - a <= n_group or level == 21:
            groups.append(order[a:b])
            continue
        digit = (keys[a:b] >> np.uint64(60 - 3 * level)).astype(np.int64) & 7
        cut = a + np.searchsorted(digit, np.arange(9))
        todo += [(cut[k], cut[k + 1], level + 1) for k in reversed(range(8)) if cut[k] < cut[k + 1]]
    return groups


def _walks(kind, s, groups):
    """Per walk (epi, epj, spj or None) of the i-groups."""
    if kind == "density":
        rs = 1.1 * s["ksr"]
        lists = walks.gather_lists(s["pos"], rs, groups)
        return [(walks.density_epi(g, s, rs), walks.density_epj(j, s), None) for g, j in zip(groups, lists)]
    if kind == "hydro":
        lists = walks.symmetric_lists(s["pos"], s["ksr"], groups)
        return [(walks.hydro_epi(g, s), walks.hydro_epj(j, s), None) for g, j in zip(groups, lists)]
    eps2 = (s["ksr"] / units.KSRH) ** 2
    near, far = walks.gravity_lists(s["pos"], s["mass"], eps2, groups, near_factor=0.5, cell_frac=1.0 / 16.0)
    return [(walks.gravity_epi(g, s), walks.gravity_epj(j, s), sp) for g, j, sp in zip(groups, near, far)]


FORCE = {"density": abi.Density, "hydro": abi.Hydro, "gravity": abi.Gravity}


def _walk_inputs(case, seed):
    s = _star(case["n"], seed)
    if case["do"] == "call":   # one compact group inside the star
        centre = s["pos"][np.random.default_rng(seed + 1).integers(case["n"] // 2)]
        near = np.argsort(((s["pos"] - centre) ** 2).sum(1), kind="stable")
        return _walks(case["kind"], s, [near[:case["n_group"]]])
    return _walks(case["kind"], s, _groups(s["pos"], case["n_group"]))


def _device_inputs(case, seed):
    n = max(case["n_j"], case["n_i"])
    s = _star(n, seed)
    order = np.random.default_rng(seed + 1).permutation(n)
    return walks.gravity_epi(order[:case["n_i"]], s), walks.gravity_epj(order[:case["n_j"]], s)


def _system_inputs(case, seed):
    s, eta = ic.config_system(case["config"], scale=case["scale"], seed=seed)
    s = state_from_ic(s)
    rng = np.random.default_rng(seed + 7)
    v = np.sqrt((s["vel"] ** 2).sum(1).mean())
    if v > 0.0:   # collisions: the stars' own motions, 2% of the bulk speed
        s["vel"] = s["vel"] + rng.normal(scale=0.02 * v, size=s["vel"].shape)
    else:         # a star being relaxed: spin and noise
        s["vel"] = np.cross([0.0, 0.0, 2e-3], s["pos"]) + rng.normal(scale=1.0, size=s["pos"].shape)
    if case["do"] == "forces":
        # a settled state: the polytrope's guess of h diverges at the surface, a step's is the last evaluation's
        s["ksr"] = np.minimum(s["ksr"], np.quantile(s["ksr"], 0.999))
    s["istar"] = s["istar"].astype(np.int32)
    keep = ("id", "istar", "mass", "pos", "vel", "uene", "ksr", "alph", "alphu")
    return {k: np.ascontiguousarray(s[k]) for k in keep}, eta


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


# ---------------------------------------------------------------- passes
FORCE_FIELDS = ("acc", "udot", "pot", "dens", "ksr")
STATE_FIELDS = ("pos", "vel", "uene")


def prepare(case, seed):
    do = case["do"]
    if do == "device":
        epi, epj = _device_inputs(case, seed)
        fn = _lib.load().sph_calc_gravity_ep_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p,
                       ctypes.c_void_p]
        return dict(do=do, fn=fn, n_i=len(epi), n_j=len(epj),
                    epi=torch.from_numpy(epi.view(np.uint8).copy()).cuda(),
                    epj=torch.from_numpy(epj.view(np.uint8).copy()).cuda(),
                    force=torch.zeros((len(epi), 5), dtype=torch.float64, device="cuda"))
    if do in ("call", "batch"):
        w = _walk_inputs(case, seed)
        ctx = functors.Context(precision=case["precision"], eta=ETA, max_walks=max(1000, len(w)))
        n_i = [len(a) for a, _, _ in w]
        off = np.concatenate([[0], np.cumsum(n_i)])
        force = np.zeros(off[-1], FORCE[case["kind"]])
        return dict(do=do, kind=case["kind"], single=case["precision"] == "fp32c", ctx=ctx, n_walk=len(w),
                    epi=[a for a, _, _ in w], epj=[b for _, b, _ in w], spj=[c for _, _, c in w],
                    n_i=n_i, n_j=[len(b) for _, b, _ in w], n_s=[0 if c is None else len(c) for _, _, c in w],
                    force=force, parts=[force[off[k]:off[k + 1]] for k in range(len(w))])
    host, eta = _system_inputs(case, seed)
    host = {k: _pinned(v) for k, v in host.items()}
    n = len(host["mass"])
    ctx = functors.Context(precision=case["precision"], eta=eta)
    params = dict(n_group=case["n_group"])
    if case["config"] == "c4":
        params["quadrupole"] = 1
    if do == "adjoint":
        params["ksr_max_mode"] = 0   # the derivative has no clamp of h
    ps = ParticleSystem(ctx, n, **params)
    ps.upload(host)
    ps.compute_forces()              # sizes the lists, captures the force graph
    state = dict(do=do, single=case["precision"] == "fp32c", ctx=ctx, ps=ps, host=host)
    if do == "adjoint":
        for _ in range(8):           # from a settled h: the derivative covers evaluations of one density walk
            ps.compute_forces()
            if ps.stats()["density_iterations"] == 1:
                break
        rng = np.random.default_rng(seed + 3)
        acc, udot = ps.download("acc"), ps.download("udot")
        state["seed"] = {"acc": rng.normal(size=(n, 3)) / np.abs(acc).mean(),
                         "udot": rng.normal(size=n) / np.abs(udot).mean(),
                         "adot": rng.normal(size=n) / np.abs(ps.download("adot")).mean(),
                         "ksr": rng.normal(size=n) / host["ksr"].mean(),
                         "pot": rng.normal(size=n) / np.abs(ps.download("pot")).mean(),
                         "dens": rng.normal(size=n) / ps.download("dens").mean()}
        return state
    if do == "steps":
        state["steps"] = case["steps"]
        ps.set_graph(False)          # a trial run sizes the lists for the steps to come
        ps.step(case["steps"])
        ps.set_graph(True)
        ps.upload(host)
        ps.compute_forces()
        ps.step(1)                   # captures the step graph
    fields = STATE_FIELDS if do == "steps" else FORCE_FIELDS
    state["out"] = {k: _pinned(np.zeros((n, 3) if k in ("acc", "pos", "vel") else n)) for k in fields}
    return state


def run(state):
    return {"call": _run_call, "batch": _run_batch, "device": _run_device, "forces": _run_system,
            "steps": _run_system, "adjoint": _run_adjoint}[state["do"]](state)


def _fields(state, names):
    """The force structs' fields; `names` are the ones FP32C forms in single
    precision.  Its neighbour count is left out: a neighbour at the edge of the
    support is counted or not by the rounding of those fields."""
    f = state["force"]
    if not state["single"]:
        return {k: f[k] for k in f.dtype.names}
    return {k: f[k].astype(np.float32) if k in names else f[k] for k in f.dtype.names if k != "np"}


SINGLE = {"density": ("dens", "divv", "rotv", "grdh", "ksr"), "hydro": ("vsmx",), "gravity": ("acc", "pot", "eta")}


def _run_call(st):
    epi, epj, spj, force = st["epi"][0], st["epj"][0], st["spj"][0], st["force"]
    if st["kind"] == "density":
        functors.calcDensity(st["ctx"])(epi, len(epi), epj, len(epj), force)
    elif st["kind"] == "hydro":
        functors.calcHydro(st["ctx"])(epi, len(epi), epj, len(epj), force)
    else:   # accumulates: particles, then monopoles, into a cleared force
        force.view(np.float64)[:] = 0.0
        gravity = functors.calcGravity(st["ctx"])
        gravity(epi, len(epi), epj, len(epj), force)
        gravity(epi, len(epi), spj, len(spj), force)
    return _fields(st, SINGLE[st["kind"]])


def _run_batch(st):
    ctx, nw = st["ctx"], st["n_walk"]
    if st["kind"] == "density":
        functors.DispatchKernel_Dens(ctx, 0, nw, st["epi"], st["n_i"], st["epj"], st["n_j"])
        functors.RetrieveKernel_Dens(ctx, 0, nw, st["n_i"], st["parts"])
    elif st["kind"] == "hydro":
        functors.DispatchKernel_HydroForce(ctx, 0, nw, st["epi"], st["n_i"], st["epj"], st["n_j"])
        functors.RetrieveKernel_HydroForce(ctx, 0, nw, st["n_i"], st["parts"])
    else:
        functors.DispatchKernel_Gravity(ctx, 0, nw, st["epi"], st["n_i"], st["epj"], st["n_j"], st["spj"], st["n_s"])
        functors.RetrieveKernel_Gravity(ctx, 0, nw, st["n_i"], st["parts"])
    return _fields(st, SINGLE[st["kind"]])


def _run_device(st):
    st["force"].zero_()
    r = st["fn"](st["epi"].data_ptr(), st["n_i"], st["epj"].data_ptr(), st["n_j"], st["force"].data_ptr(),
                 torch.cuda.current_stream().cuda_stream)
    if r:
        raise abi.SPHError(r, "gravity on device buffers")
    return st["force"].float()


def _run_system(st):
    ps = st["ps"]
    ps.upload(st["host"])
    ps.compute_forces()
    if st["do"] == "steps":
        ps.step(st["steps"])
    for k, out in st["out"].items():
        ps.download(k, out=out)
    if st["do"] == "forces" and st["single"]:
        return {k: torch.from_numpy(v).float() for k, v in st["out"].items()}
    return dict(st["out"])


def _run_adjoint(st):
    return st["ps"].adjoint_forces(st["seed"])


# ---------------------------------------------------------------- work
def _system_size(case):
    full = {"c0": (1.0e4, ETA), "c1": (2.0e5, ETA), "c2": (1.0e6, ETA), "c3": (1.0e5, ETA), "c4": (4.0e6, ETA_LARGE)}
    n, eta = full[case["config"]]
    return n * case["scale"], eta


def work(case):
    """Pairs inside a support (gravity: the listed ones) x the flop per pair of
    the reference's kernels (density 132, hydro 109, gravity 29), inputs read
    once and outputs written once."""
    def neighbours(eta):
        return 4.0 / 3.0 * math.pi * (eta * units.KSRH) ** 3

    if case["do"] == "device":
        return {"bytes": 32 * case["n_i"] + 40 * case["n_j"] + 2 * 40 * case["n_i"],
                "flops": 29.0 * case["n_i"] * case["n_j"]}
    if case["do"] in ("call", "batch"):
        # octree cells of at most n_group particles hold about half of that; a density or hydro list holds the
        # particles within the search radius of the cell, a gravity list its vicinity and the cells beyond
        call = case["do"] == "call"
        g = min(case["n"], case["n_group"] * (1.0 if call else 0.5))
        n_walk = 1.0 if call else max(1.0, case["n"] / g)
        if case["kind"] == "gravity":
            n_list = min(case["n"], 2000.0)
            return {"bytes": n_walk * (72.0 * g + 40.0 * n_list), "flops": 29.0 * n_walk * g * n_list}
        n_list = min(case["n"], (g ** (1.0 / 3.0) + 2.0 * 1.1 * ETA * units.KSRH) ** 3)
        i, j, f = (80, 64, 56) if case["kind"] == "density" else (144, 152, 72)
        flop = 132.0 if case["kind"] == "density" else 109.0
        return {"bytes": n_walk * ((i + f) * g + j * n_list),
                "flops": flop * n_walk * g * min(case["n"], neighbours(ETA))}
    n, eta = _system_size(case)
    # theta = 0.5 tree lists hold ~130 log2(n) entries per particle
    pairs = neighbours(eta) * (132.0 + 109.0) + 29.0 * min(n, 130.0 * math.log2(n))
    if case["do"] == "adjoint":   # about three times the forward pair work
        return {"bytes": 8.0 * n * (8 + 9 + 20), "flops": 3.0 * n * pairs}
    evals = 1 + case.get("steps", 0)
    return {"bytes": n * (100.0 + 56.0), "flops": evals * n * pairs}


# ---------------------------------------------------------------- 64-bit values
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _separations(xi, xj):
    d = [xi[:, None, k] - xj[None, :, k] for k in range(3)]
    return d, d[0] * d[0] + d[1] * d[1] + d[2] * d[2]


def _w0(q):
    u = torch.clamp(1.0 - q, min=0.0)
    return u ** 4 * (1.0 + 4.0 * q)


def _w1(q):
    u = torch.clamp(1.0 - q, min=0.0)
    return u ** 4 - u ** 3 * (1.0 + 4.0 * q)


def _density64(ii, jj, eta):
    """Three h passes and the gradient pass (hdr_density.hpp:264-349)."""
    d, r2 = _separations(ii["pos"], jj["pos"])
    r = r2.sqrt()
    h = ii["ksr"]
    for _ in range(3):
        rho = units.CEFF0 / h ** 3 * (jj["mass"] * _w0(r / h[:, None])).sum(1)
        h = eta * units.KSRH * (ii["mass"] / rho) ** (1.0 / 3.0)
    other = ii["id"][:, None] != jj["id"][None, :]
    ri = torch.where(other, 1.0 / r, torch.zeros_like(r))
    q = r2 * ri / h[:, None]
    w1 = _w1(q)
    grdh = -(jj["mass"] * (3.0 * units.CEFF0 * _w0(q) + units.CEFF1 * q * w1)).sum(1) / h ** 4
    omega = 1.0 / (1.0 + h * grdh / (3.0 * rho))
    dw = jj["mass"] * w1 * ri
    u = [ii["vel"][:, None, k] - jj["vel"][None, :, k] for k in range(3)]
    c = units.CEFF1 / h ** 4 / rho * omega
    divv = -c * ((u[0] * d[0] + u[1] * d[1] + u[2] * d[2]) * dw).sum(1)
    rot = [((u[(k + 1) % 3] * d[(k + 2) % 3] - u[(k + 2) % 3] * d[(k + 1) % 3]) * dw).sum(1) for k in range(3)]
    rotv = c * (rot[0] ** 2 + rot[1] ** 2 + rot[2] ** 2).sqrt()
    return {"dens": rho, "divv": divv, "rotv": rotv, "grdh": omega, "ksr": h}


def _hydro64(ii, jj):
    """hdr_hydro.hpp:349-421."""
    d, r2 = _separations(ii["pos"], jj["pos"])
    other = ii["id"][:, None] != jj["id"][None, :]
    ri = torch.where(other, 1.0 / r2.sqrt(), torch.zeros_like(r2))
    r = r2 * ri
    u = [ii["vel"][:, None, k] - jj["vel"][None, :, k] for k in range(3)]
    dw_i = units.CEFF1 * (ii["hinv"] ** 4)[:, None] * _w1(r * ii["hinv"][:, None])
    dw_j = units.CEFF1 * jj["hinv"] ** 4 * _w1(r * jj["hinv"])
    ka = (dw_i + dw_j) * jj["mass"]
    w = (d[0] * u[0] + d[1] * u[1] + d[2] * u[2]) * ri
    wn = torch.clamp(w, max=0.0)
    vs = ii["vsnd"][:, None] + jj["vsnd"] - 3.0 * wn
    rhi = 1.0 / (ii["dens"][:, None] + jj["dens"])
    av = (ii["bswt"][:, None] + jj["bswt"]) * (ii["alph"][:, None] + jj["alph"]) * vs * wn
    ta = (ii["presc"][:, None] + jj["presc"] - 0.5 * av * rhi) * ka * ri
    du = ii["thrm"][:, None] - jj["thrm"]
    vsu = (2.0 * (ii["pres"][:, None] - jj["pres"]).abs() * rhi).sqrt()
    udot = ka * (ii["presc"][:, None] * w
                 - rhi * (0.25 * av * wn - (ii["alphu"][:, None] + jj["alphu"]) * vsu * du))
    dg = jj["mass"] * ri * (ii["eta"][:, None] * dw_i + jj["eta"] * dw_j)
    return {"acch": torch.stack([-0.5 * (ta * x).sum(1) for x in d], 1),
            "accg": torch.stack([0.5 * (dg * x).sum(1) for x in d], 1),
            "udot": 0.5 * udot.sum(1), "vsmx": torch.clamp(vs.max(1).values, min=0.0),
            "diffu": 2.0 * (rhi * du * ka * ri).sum(1)}


def _gravity64(ii, jj):
    """hdr_gravity.hpp:295-339."""
    d, r2 = _separations(ii["pos"], jj["pos"])
    a = 1.0 / (r2 + ii["eps2"][:, None]).sqrt()
    b = 1.0 / (r2 + jj["eps2"]).sqrt()
    g = jj["mass"] * (a ** 3 + b ** 3)
    return {"acc": torch.stack([-0.5 * (g * x).sum(1) for x in d], 1),
            "pot": -0.5 * (jj["mass"] * (a + b)).sum(1), "eta": (jj["mass"] * a ** 3).sum(1)}


def _fields64(a):
    return {k: _t(a[k]) for k in a.dtype.names}


def _exact_walks(case, seed):
    parts = []
    for epi, epj, spj in _walk_inputs(case, seed):
        if spj is not None:
            epj = np.concatenate([epj, spj])
        jj = _fields64(epj)
        for k in range(0, len(epi), 4096):
            ii = _fields64(epi[k:k + 4096])
            parts.append(_density64(ii, jj, ETA) if case["kind"] == "density" else
                         _hydro64(ii, jj) if case["kind"] == "hydro" else _gravity64(ii, jj))
    got = {k: torch.cat([p[k] for p in parts]).cpu() for k in parts[0]}
    return {k: got.get(k) for k in FORCE[case["kind"]].names}   # np and itr: none


def _exact_forces(case, seed):
    """Density, h and du/dt of a small system over all pairs; the tree's
    acceleration and potential have no such value."""
    s, eta = _system_inputs(case, seed)
    n = len(s["mass"])
    jj = {k: _t(s[k]) for k in ("id", "mass", "pos", "vel", "ksr")}
    rows = max(1, 20_000_000 // n)

    def over_rows(f, names):
        parts = [f({k: v[a:a + rows] for k, v in names.items()}) for a in range(0, n, rows)]
        return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}

    den = over_rows(lambda ii: _density64(ii, jj, eta), jj)
    u, rho, h = _t(s["uene"]), den["dens"], den["ksr"]
    pres = rho * u / units.EOS_N
    c = (units.GAMMA * pres / rho).sqrt()
    ad = den["divv"].abs()
    bswt = ad / (ad + den["rotv"] + 1e-4 * c * units.KSRH / h)
    jj.update(ksr=h, hinv=1.0 / h, pres=pres, presc=pres * den["grdh"] / rho ** 2, bswt=0.5 * bswt, dens=rho, vsnd=c,
              alph=_t(s["alph"]), alphu=_t(s["alphu"]), thrm=u, eta=torch.zeros_like(h))
    udot = over_rows(lambda ii: _hydro64(ii, jj), jj)["udot"]
    return {"acc": None, "udot": udot.cpu(), "pot": None, "dens": rho.cpu(), "ksr": h.cpu()}


def exact(case, seed):
    if case["do"] in ("call", "batch"):
        return _exact_walks(case, seed)
    if case["do"] == "device":
        epi, epj = _device_inputs(case, seed)
        jj = _fields64(epj)
        got = [_gravity64(_fields64(epi[k:k + 256]), jj) for k in range(0, len(epi), 256)]
        return torch.cat([torch.cat([g["acc"], g["pot"][:, None], g["eta"][:, None]], 1) for g in got]).cpu()
    if case["do"] == "forces" and _system_size(case)[0] <= 30000:
        return _exact_forces(case, seed)
    return None
