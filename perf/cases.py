"""Timed cases of the framework's entry points, from the smallest calls to
the largest workloads.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones of the
same ranges, ``prepare`` builds what a program holds on the GPU before the
call, ``run`` is one pass through the public entry points, ``work`` counts
the bytes and operations a pass cannot do without, and ``exact`` restates the
pass in 64 bits with plain torch.

Particle sets are dam breaks and rolled sloshing tanks on the lattices of the
repository's own configurations: the fluid moves, is slightly compressed,
sheared and jittered off the lattice, and lies in memory in the order that the previous
step's sort left (a few particles have changed cell since).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from aquagpusph_gb300 import _lib, case as cases, learned
from aquagpusph_gb300.solver import Solver

REFD, NU, DELTA, G = 998.0, 1.0e-6, 0.1, 9.81
STATE_OUT = ("id", "r", "u", "dudt", "rho", "drhodt", "p", "shepard")
K_STEPS = 8          # plain steps one proposal stands for
MODEL_SCALES = (0.5, 2.0, 5.0, 50.0)   # u, rho, dudt, drhodt of the features
OUT_SCALE = (0.02, 0.2)


# ------------------------------------------------------------------ cases ----

def _dam(name, dims, dx, block, tank, fast, steps, bi=False):
    """Dam break: `block` fluid cells in a tank of `tank` cells."""
    b, t = tuple(block) + (1,), tuple(tank) + (1,)
    return {"name": name, "kind": "dam", "dims": dims, "dx": dx,
            "bx": b[0], "by": b[1], "bz": b[2] if dims == 3 else 1,
            "tx": t[0], "ty": t[1], "tz": t[2] if dims == 3 else 1,
            "fast": fast, "steps": steps, "bi": bi}


def listed():
    return [
        # the 2-D dam break of the smoke test, in the default arithmetic: a
        # short burst of steps between two reports, where latency counts
        _dam("dam2d_8k_exact", 2, 0.01, (120, 60), (322, 180), False, 8),
        # a small 3-D tank (the size of the history test), default arithmetic
        _dam("dam3d_16k_exact", 3, 0.01, (20, 20, 20), (60, 20, 40), False, 4),
        # the slab the CPU oracle is timed on, in both arithmetics
        _dam("dam3d_406k_exact", 3, 0.005, (80, 40, 110), (160, 40, 120), False, 1),
        _dam("dam3d_406k_fast", 3, 0.005, (80, 40, 110), (160, 40, 120), True, 1),
        # the benchmark's default workload
        _dam("dam3d_5.9M_fast", 3, 0.005, (246, 200, 110), (644, 200, 200), True, 1),
        # the largest configuration
        _dam("dam3d_26M_fast", 3, 0.003, (409, 333, 183), (1073, 333, 333), True, 1),
        # analytic boundary integrals with the improved Euler scheme
        _dam("dam3d_60k_bi", 3, 0.01, (40, 30, 35), (90, 30, 50), False, 1, True),
        # the batched configuration: 64 uneven tanks rolled on their own
        {"name": "slosh_64_fast", "kind": "slosh", "n_cases": 64, "dx": 0.004,
         "fast": True, "steps": 1},
        # a few tanks in the default arithmetic
        {"name": "slosh_5_exact", "kind": "slosh", "n_cases": 5, "dx": 0.005,
         "fast": False, "steps": 2},
        # the link-list tool on a caller's own positions
        {"name": "linklist_1.9M", "kind": "linklist", "dims": 3, "dx": 0.005,
         "bx": 160, "by": 100, "bz": 110, "tx": 320, "ty": 100, "tz": 120},
        # one learned proposal for the batch: neighbour graph, network, update
        {"name": "propose_64", "kind": "propose", "n_cases": 64, "dx": 0.004},
        # one training step's loss and gradients on 16 tanks
        {"name": "train_16", "kind": "train", "n_cases": 16, "dx": 0.004},
    ]


def draw(rng):
    kind = rng.choice(["dam"] * 6 + ["slosh"] * 3 + ["linklist", "propose", "train"])
    if kind in ("propose", "train"):
        return {"kind": kind, "n_cases": rng.randint(1, 64 if kind == "propose" else 16),
                "dx": round(rng.uniform(0.004, 0.008), 5)}
    if kind == "slosh":
        fast = rng.random() < 0.6
        return {"kind": kind, "n_cases": int(round(math.exp(rng.uniform(0, math.log(96))))),
                "dx": round(rng.uniform(0.004, 0.01), 5), "fast": fast,
                "steps": 1 if fast else rng.choice([1, 2, 3])}
    dims = 3 if kind == "linklist" else rng.choice([2, 3, 3])
    fast = rng.random() < 0.5
    bi = kind == "dam" and rng.random() < 0.15
    most = 2.0e5 if bi else 1.5e6 if (not fast or dims == 2) else 1.2e7
    n = math.exp(rng.uniform(math.log(800.0), math.log(most)))
    ax, az = rng.uniform(0.7, 1.6), rng.uniform(0.5, 1.4)
    if dims == 2:
        b = [max(4, round(math.sqrt(n * ax))), max(3, round(math.sqrt(n / ax)))]
        t = [b[0] + max(4, int(b[0] * rng.uniform(0.3, 1.6))),
             b[1] + max(4, int(b[1] * rng.uniform(0.2, 1.5)))]
    else:
        e = (n / (ax * az)) ** (1.0 / 3.0)
        b = [max(4, round(e * ax)), max(4, round(e)), max(3, round(e * az))]
        t = [b[0] + max(4, int(b[0] * rng.uniform(0.3, 1.6))), b[1],
             b[2] + max(4, int(b[2] * rng.uniform(0.1, 0.8)))]
    c = _dam("", dims, round(rng.uniform(0.003, 0.02), 5), b, t, fast,
             rng.choice([1, 1, 2, 4]) if not fast else 1, bi)
    del c["name"]
    if kind == "linklist":
        for k in ("fast", "steps", "bi"):
            del c[k]
        c["kind"] = kind
    return c


# -------------------------------------------------------------- particles ----

def _params(case):
    """Scalar Variables and Definitions of a dam-break case."""
    dims, dx = case["dims"], case["dx"]
    h = 2.0 * dx
    ext = (case["tx"] * dx, case["ty"] * dx, case["tz"] * dx)[:dims]
    m = 4 * h
    up = dims - 1
    g = [0.0] * 4
    g[up] = -G
    return cases.Params(
        dims=dims, h=h, cs=45.0 if dims == 2 else 40.0, g=tuple(g),
        refd=(REFD, REFD), visc_dyn=(NU * REFD,) * 2, delta=(DELTA, DELTA),
        domain_min=tuple([-m] * dims + [0.0] * (4 - dims)),
        domain_max=tuple([e + m for e in ext] + [0.0] * (4 - dims)),
        boundary=1 if case.get("bi") else 0, scheme=1 if case.get("bi") else 0)


def _lattice(*counts):
    """Centres ((i + 1/2), ...) of a lattice, the last axis fastest (f64)."""
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") + 0.5 for n in counts]
    return torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, len(counts))


def _dam_geometry(case):
    """Positions, kinds, normals and tangents of fluid, walls and probes."""
    dims, dx = case["dims"], case["dx"]
    bl = (case["bx"], case["by"], case["bz"])[:dims]
    tk = (case["tx"], case["ty"], case["tz"])[:dims]
    up = dims - 1
    r, im, nr, tg = [_lattice(*bl)], [], [], []
    n_fl = r[0].shape[0]
    im.append(torch.full((n_fl,), cases.FLUID, dtype=torch.int32, device="cuda"))
    nr.append(torch.zeros_like(r[0]))
    tg.append(torch.zeros_like(r[0]))
    for a in range(dims):
        for side in (0, 1):
            if dims == 3 and a == up and side == 1:
                continue  # open top
            rest = [k for k in range(dims) if k != a]
            f = _lattice(*[tk[k] for k in rest])
            p = torch.zeros((f.shape[0], dims), dtype=torch.float64, device="cuda")
            p[:, rest] = f
            p[:, a] = side * tk[a]
            n = torch.zeros_like(p)
            n[:, a] = 1.0 if side else -1.0
            t = torch.zeros_like(p)
            t[:, rest[0]] = 1.0
            r.append(p)
            nr.append(n)
            tg.append(t)
            im.append(torch.full((f.shape[0],), cases.WALL, dtype=torch.int32, device="cuda"))
    pr = torch.zeros((2, dims), dtype=torch.float64, device="cuda")  # two probes on the far wall
    pr[:, 0] = tk[0]
    if dims == 3:
        pr[:, 1] = 0.5 * tk[1]
    pr[:, up] = torch.tensor([2.0, 6.0], dtype=torch.float64, device="cuda")
    r.append(pr)
    nr.append(torch.zeros_like(pr))
    tg.append(torch.zeros_like(pr))
    im.append(torch.full((2,), cases.SENSOR, dtype=torch.int32, device="cuda"))
    return torch.cat(r) * dx, torch.cat(im), torch.cat(nr), torch.cat(tg)


def _fill(r, im, nr, tg, dx, dims, cs, hf, seed):
    """Moving, slightly compressed fluid on a sheared lattice; the walls and
    probes at rest.  `hf` = still-water height of each particle's case."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n, vs, up = r.shape[0], 4 if dims == 3 else 2, dims - 1
    fl = im == cases.FLUID
    f1 = fl[:, None].double()
    uni = lambda *s: torch.rand(*s, generator=gen, device="cuda", dtype=torch.float32).double() * 2 - 1  # noqa: E731
    press = REFD * G * (hf - r[:, up]).clamp_min(0.0)
    rho = torch.where(fl, REFD + press / cs ** 2, torch.full_like(press, REFD))
    m = torch.where(fl, rho * dx ** dims,
                    torch.where(im == cases.WALL, torch.full_like(rho, dx ** (dims - 1)),
                                torch.zeros_like(rho)))
    rho = rho * (1.0 + 2.0e-4 * uni(n) * fl)
    x = r[:, 0] / (r[:, 0].max() + dx)
    u = torch.zeros((n, dims), dtype=torch.float64, device="cuda")
    u[:, 0] = 1.2 * x
    u[:, up] = -0.6 * (r[:, up] / (hf + dx))
    u = (u + 0.03 * uni(n, dims)) * f1
    a = torch.zeros_like(u)
    a[:, 0] = 3.0 * x
    a[:, up] = -2.0
    a = (a + 0.5 * uni(n, dims)) * f1
    # the flow has sheared the lattice: cells cut it anywhere (nothing near
    # the walls and the surface)
    hi = torch.where(fl[:, None], r, torch.zeros_like(r)).amax(0) + 0.5 * dx
    win = (r / (4 * dx)).clamp(0, 1) * ((hi - r) / (4 * dx)).clamp(0, 1)
    phase = 2 * math.pi * torch.rand(dims, generator=gen, device="cuda", dtype=torch.float32).double()
    wave = torch.sin(2 * math.pi / (23.7 * dx) * r.roll(-1, 1) + phase)
    r = r + (0.8 * dx * win * wave + 0.1 * dx * uni(n, dims)) * f1

    def vec(v):
        out = torch.zeros((n, vs), dtype=torch.float32, device="cuda")
        out[:, :dims] = v.float()
        return out

    return {"id": torch.arange(n, dtype=torch.int32, device="cuda"),
            "iset": (~fl).int(), "imove": im, "r": vec(r), "normal": vec(nr),
            "tangent": vec(tg), "binormal": vec(torch.zeros_like(u)), "u": vec(u),
            "dudt": vec(a), "rho": rho.float(),
            "drhodt": (40.0 * uni(n) * fl).float(), "m": m.float(),
            "p": torch.where(fl, press, torch.zeros_like(press)).float()}


def _keys(r, dims, cell, cid=None):
    """Cell keys in the tool's float arithmetic: per case, x fastest."""
    c32 = torch.tensor(cell, dtype=torch.float32, device="cuda")
    inv = torch.tensor(1.0, dtype=torch.float32, device="cuda") / c32
    n_cases = 1 if cid is None else int(cid.max().item()) + 1
    keys = torch.zeros(r.shape[0], dtype=torch.int64, device="cuda")
    nxs = torch.zeros((n_cases, 3), dtype=torch.int64, device="cuda")
    base = 0
    for k in range(n_cases):
        at = slice(None) if cid is None else cid == k
        x = r[at, :dims]
        lo, hi = x.amin(0), x.amax(0)
        nc = torch.floor((hi - lo) / c32).long() + 6
        ic = torch.floor((x - lo) * inv).long() + 2
        key = torch.full((x.shape[0],), base, dtype=torch.int64, device="cuda")
        mul = 1
        for d in range(dims):
            key += ic[:, d] * mul
            nxs[k, d] = mul
            mul *= int(nc[d].item())
        keys[at] = key
        base += mul
    return keys, nxs


def _previous_order(s, dims, cell, dt, cid=None):
    """The order the last step's sort left: by the cells of r - u dt."""
    keys, _ = _keys(s["r"] - float(dt) * s["u"], dims, cell, cid)
    o = torch.argsort(keys, stable=True)
    return {k: v[o].contiguous() for k, v in s.items()}


def _dam_state(case, seed):
    p = _params(case)
    r, im, nr, tg = _dam_geometry(case)
    hf = torch.full((r.shape[0],), (case["by"] if p.dims == 2 else case["bz"]) * case["dx"],
                    dtype=torch.float64, device="cuda")
    s = _fill(r, im, nr, tg, case["dx"], p.dims, p.cs, hf, seed)
    return p, _previous_order(s, p.dims, p.cell_length, p.dt_fixed)


def _slosh_batch(case):
    return cases.sloshing_batch_2d(n_cases=case["n_cases"], seed=2026, dx=case["dx"])


def _slosh_state(case, seed):
    """Batch, params, state (case by case) and the case of each particle."""
    b = _slosh_batch(case)
    c, p = b.case, b.case.params
    cid = learned.case_ids(b)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    im = t(c.imove)
    r = t(c.r[:, :2].astype(np.float64))
    top = torch.full((b.n_cases,), 0.0, dtype=torch.float64, device="cuda")
    top.scatter_reduce_(0, cid.long(), torch.where(im == 1, r[:, 1], torch.zeros_like(r[:, 1])), "amax")
    hf = (top + 0.5 * case["dx"])[cid.long()]
    s = _fill(r, im, t(c.normal).double(), t(c.tangent).double(), case["dx"], 2, p.cs, hf, seed)
    s["iset"] = t(c.iset).int()
    s = _previous_order(s, 2, p.cell_length, p.dt_fixed, cid)
    return b, p, s, cid


def _ptrs(d, names=None):
    return {k: d[k].data_ptr() for k in (names or d)}


def _outputs(n, dims):
    vs = 4 if dims == 3 else 2
    return {k: torch.zeros((n, vs) if k in ("r", "u", "dudt") else (n,),
                           dtype=torch.int32 if k == "id" else torch.float32, device="cuda")
            for k in STATE_OUT}


# ----------------------------------------------------------------- passes ----

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("propose", "train"):
        return _prepare_learned(case, seed)
    if kind == "slosh":
        b, p, s, _ = _slosh_state(case, seed)
        n = s["r"].shape[0]
        sv = Solver(p, capacity=n, ihoc_capacity=b.n_cases * p.max_cells())
        b.case.dt = p.dt_fixed
    else:
        b = None
        p, s = _dam_state(case, seed)
        n = s["r"].shape[0]
        sv = Solver(p, capacity=n)
    st = {"kind": kind, "sv": sv, "n": n, "in": s, "dt": p.dt_fixed, "batch": b}
    if kind == "linklist":
        st["ihoc_capacity"] = sv.ncap
        st["out"] = {k: torch.zeros(n, dtype=torch.int32, device="cuda")
                     for k in ("icell", "id_sorted", "id_unsorted")}
        st["out"]["ihoc"] = torch.zeros(sv.ncap, dtype=torch.int32, device="cuda")
        return st
    sv.set_precision(case["fast"])
    st["steps"] = case["steps"]
    st["in_ptrs"] = _ptrs(s)
    st["out"] = _outputs(n, p.dims)
    st["out_ptrs"] = _ptrs(st["out"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "linklist":
        o = st["out"]
        got = st["sv"].linklist(st["in"]["r"].data_ptr(), st["n"], o["icell"].data_ptr(),
                                o["id_sorted"].data_ptr(), o["id_unsorted"].data_ptr(),
                                o["ihoc"].data_ptr(), st["ihoc_capacity"])
        return {**o, **got}
    if kind == "propose":
        return _propose(st)
    if kind == "train":
        return _train(st)
    # a snapshot becomes the resident state, advances, and is read back
    sv = st["sv"]
    sv.set_state_raw(st["n"], st["in_ptrs"], False, 0.0, st["dt"], 0)
    if st["batch"] is not None:
        sv.set_cases(st["batch"])
    sv.step(st["steps"], graph=True)
    sv.get_state_raw(st["out_ptrs"], False)
    return st["out"]


def _prepare_learned(case, seed):
    b, p, s, cid = _slosh_state(case, seed)
    n = s["r"].shape[0]
    sv = Solver(p, capacity=n, ihoc_capacity=b.n_cases * p.max_cells())
    model = learned.Model(2, seed=int(seed))
    model.scales.copy_(torch.tensor([p.h, *MODEL_SCALES, REFD], dtype=torch.float32))
    model.out_scale = OUT_SCALE
    dt = torch.full((b.n_cases,), p.dt_fixed, dtype=torch.float32, device="cuda")
    st = {"kind": case["kind"], "sv": sv, "n": n, "in": s, "cid": cid, "model": model,
          "dt": dt, "radius": float(p.support * p.h)}
    if case["kind"] == "train":
        s0, s1 = learned.Snapshot(n, 2), learned.Snapshot(n, 2)
        for k, v in s.items():
            s0[k].copy_(v)
        for k, v in _later(s, p.dt_fixed, seed).items():
            s1[k].copy_(v)
        st["pair"] = (s0, s1)
        st["trainer"] = learned.Trainer(model, sv, b, K_STEPS, cases_per_step=b.n_cases)
    return st


def _later(s, dt, seed):
    """A state K_STEPS later: the extrapolation plus a smooth residual."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 7)
    T = K_STEPS * float(dt)
    fl = (s["imove"] == 1).float()
    z = lambda *k: torch.randn(*k, generator=gen, device="cuda")  # noqa: E731
    n = fl.shape[0]
    out = dict(s)
    out["u"] = s["u"] + (T * s["dudt"] + OUT_SCALE[0] * z(n, 2)) * fl[:, None]
    out["rho"] = s["rho"] + (T * s["drhodt"] + OUT_SCALE[1] * z(n)) * fl
    return out


def _propose(st):
    s, n = st["in"], st["n"]
    g = learned.Graph(st["sv"], 2, s["r"], s["imove"], st["cid"], n, st["radius"])
    x = learned.Inputs(g, s["r"], s["u"], s["rho"], s["dudt"], s["drhodt"], s["imove"],
                       s["normal"])
    out = learned.Network(st["model"], g, x).forward(train=False)
    new = {k: s[k].clone() for k in ("r", "u", "rho")}
    su, srho = st["model"].out_scale
    _lib.check("aqua_gnn_apply", learned.lib().aqua_gnn_apply(
        g.n_nodes, 2, g.perm.data_ptr(), out.data_ptr(), st["cid"].data_ptr(),
        st["dt"].data_ptr(), K_STEPS, su, srho, new["r"].data_ptr(), new["u"].data_ptr(),
        new["rho"].data_ptr(), s["dudt"].data_ptr(), s["drhodt"].data_ptr(),
        s["imove"].data_ptr(), 0))
    return {"out": out, **new}


def _train(st):
    tr = st["trainer"]
    net, loss, dout, _ = tr.batch_loss(st["pair"], st["dt"], 0, len(tr.offsets) - 1)
    st["model"].grad.zero_()
    net.backward(dout)
    return {"loss": loss, "grad": st["model"].grad, "out": net.out}


# ------------------------------------------------------------------- work ----

def _counts(case):
    """(particles, fluid particles, dims)"""
    if case["kind"] in ("slosh", "propose", "train"):
        c = _slosh_batch(case).case
        return c.N, c.n_fluid, 2
    b = [case["bx"], case["by"], case["bz"]][:case["dims"]]
    t = [case["tx"], case["ty"], case["tz"]][:case["dims"]]
    nf = math.prod(b)
    if case["dims"] == 2:
        return nf + 2 * (t[0] + t[1]) + 2, nf, 2
    return nf + t[0] * t[1] + 2 * t[1] * t[2] + 2 * t[0] * t[2] + 2, nf, 3


# neighbours of a fluid particle in the support (h = 2 dx), FP32 operations
# of one pair's sums
NEIGHBOURS = {2: 48, 3: 260}
PAIR_FLOPS = {2: 42, 3: 52}
# network: multiply-adds x 2 of one edge (both rounds) and of one node
EDGE_FLOPS = 2 * (16 * 64 + 144 * 64 + 4 * 64 * 64)
NODE_FLOPS = 2 * (80 * 64 + 144 * 64 + 3 * 64 * 64 + 64 * 16)


def work(case):
    n, nf, dims = _counts(case)
    V = 16 if dims == 3 else 8
    kind = case["kind"]
    if kind == "linklist":
        return {"bytes": n * (V + 12), "flops": 6 * n}
    if kind in ("propose", "train"):
        edges = NEIGHBOURS[2] * nf
        times = 1 if kind == "propose" else 3
        return {"bytes": n * (5 * V + 16) * times,
                "flops": times * (edges * EDGE_FLOPS + n * NODE_FLOPS)}
    # the state in (12 integers' bytes, five vectors, four scalars) and the
    # results out (three vectors, five scalars)
    return {"bytes": n * (12 + 5 * V + 16) + n * (3 * V + 20),
            "flops": case["steps"] * nf * (NEIGHBOURS[dims] * PAIR_FLOPS[dims] + 150)}


# ------------------------------------------------------------------ exact ----

def exact(case, seed):
    if case["kind"] == "linklist":
        return None  # whole numbers
    if case["kind"] in ("propose", "train"):
        return _exact_learned(case, seed)
    n, nf, dims = _counts(case)
    if case.get("bi") or nf * NEIGHBOURS[dims] * case["steps"] > 2.0e9:
        return None
    if case["kind"] == "slosh":
        b, p, s, cid = _slosh_state(case, seed)
        motions = b.motions
    else:
        p, s = _dam_state(case, seed)
        cid, motions = torch.zeros(n, dtype=torch.int32, device="cuda"), [None]
    f = ("r", "normal", "tangent", "binormal", "u", "dudt", "rho", "drhodt", "m", "p")
    x = {k: v.double() if k in f else v.long() for k, v in s.items()}
    x["cid"] = cid.long()
    nc = len(motions)
    dt = torch.full((nc,), p.dt_fixed, dtype=torch.float64, device="cuda")
    t = torch.zeros_like(dt)
    for _ in range(case["steps"]):
        x, dt_new = _step64(x, p, dt, t, motions)
        t, dt = t + dt_new, dt_new
    return {k: None if k == "id" else x[k] for k in STATE_OUT}


def _neighbour_pairs(keys, nxs, cid, dims, lo, hi):
    """(i, j) index pairs of sorted particles lo..hi-1 with everything in
    their 3^D cells (j in the order of the rows)."""
    k, nx = keys[lo:hi], nxs[cid[lo:hi]]
    ii, jj = [], []
    for dz in ((-1, 0, 1) if dims == 3 else (0,)):
        for dy in (-1, 0, 1):
            row = k + dy * nx[:, 1] + (dz * nx[:, 2] if dims == 3 else 0)
            a = torch.searchsorted(keys, row - 1)
            b = torch.searchsorted(keys, row + 1, right=True)
            cnt = b - a
            i = torch.repeat_interleave(torch.arange(lo, hi, device="cuda"), cnt)
            off = torch.cumsum(cnt, 0) - cnt
            ii.append(i)
            jj.append(torch.arange(i.shape[0], device="cuda") - off[i - lo] + a[i - lo])
    return torch.cat(ii), torch.cat(jj)


def _step64(x, p, dt_case, t_case, motions):
    """One canonical step (midpoint, BIe walls) in 64 bits, sorted."""
    D = p.dims
    keys, nxs = _keys(x["r"].float(), D, p.cell_length, x["cid"])
    order = torch.argsort(keys, stable=True)
    p_old = x["p"]
    keys = keys[order]
    x = {k: v[order] for k, v in x.items()}
    n = keys.shape[0]
    im, cid = x["imove"], x["cid"]
    dt = dt_case[cid]
    fl, wall, probe = im == 1, im == -3, im == 0
    f1 = fl.double()
    r = x["r"][:, :D]
    uin, ain, rin, rhoin, din = x["u"][:, :D], x["dudt"][:, :D], r, x["rho"], x["drhodt"]
    nrm = x["normal"][:, :D]
    u = uin + 0.5 * dt[:, None] * ain * f1[:, None]
    rho = rhoin + 0.5 * dt * din * f1
    refd = torch.tensor(p.refd, dtype=torch.float64, device="cuda")[x["iset"]]
    pr = torch.where(fl, p.p0 + p.cs ** 2 * (rho - refd), p_old)
    H, CW, CF = p.H, p.CONW, p.CONF
    wc, fc = ((0.08203125, 0.8203125) if D == 3 else (0.109375, 1.09375))
    wc, fc = wc / math.pi, fc / math.pi
    shep, du, lp, dbi, srho, sp = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(6))
    gp, lu, gw, su = (torch.zeros((n, D), dtype=torch.float64, device="cuda") for _ in range(4))
    reach_i, reach_j = [], []
    step = 60000 if D == 3 else 400000
    dr_w = x["m"].clamp_min(0).sqrt() if D == 3 else x["m"]
    for lo in range(0, n, step):
        i, j = _neighbour_pairs(keys, nxs, cid, D, lo, min(n, lo + step))
        d = r[j] - r[i]
        q = (d * d).sum(1).sqrt() / H
        ok = q < 2.0
        i, j, d, q = i[ok], j[ok], d[ok], q[ok]
        w = wc * CW * (1 + 2 * q) * (2 - q) ** 4
        a = fl[j]
        wj = torch.where(a, w * x["m"][j] / rho[j], torch.zeros_like(w))
        shep.index_add_(0, i, wj)
        pb = a & probe[i]
        ip, jp, wp = i[pb], j[pb], wj[pb]
        su.index_add_(0, ip, u[jp] * wp[:, None])
        srho.index_add_(0, ip, rho[jp] * wp)
        sp.index_add_(0, ip, pr[jp] * wp)
        b = a & fl[i]
        i2, j2, d2 = i[b], j[b], d[b]
        f = fc * CF * (2 - q[b]) ** 3 * x["m"][j2]
        dv = u[j2] - u[i2]
        rr = rho[i2] * rho[j2]
        gp.index_add_(0, i2, ((pr[i2] + pr[j2]) / rr * f)[:, None] * d2)
        lu.index_add_(0, i2, (2 * f / rr)[:, None] * dv)
        du.index_add_(0, i2, (dv * d2).sum(1) * f * rho[i2] / rho[j2])
        lp.index_add_(0, i2, (pr[j2] - pr[i2]) * f / rho[j2])
        b = wall[j] & fl[i]
        i3, j3 = i[b], j[b]
        g = nrm[j3] * (w[b] * x["m"][j3])[:, None]
        gw.index_add_(0, i3, g)
        dbi.index_add_(0, i3, -(u[j3] * g).sum(1))
        near = (d[b] * d[b]).sum(1) < (4 * dr_w[j3]) ** 2
        reach_i.append(i3[near])
        reach_j.append(j3[near])
    gp = gp + (2 * pr / rho)[:, None] * gw
    du = du - 2 * rho * ((u * gw).sum(1) + dbi)
    sets = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")[x["iset"]]  # noqa: E731
    grav = torch.tensor(p.g[:D], dtype=torch.float64, device="cuda")
    acc = -gp + sets(p.visc_dyn)[:, None] * lu + grav
    drho = -du + sets(p.delta) * dt * rho / refd * lp
    # elastic bounce, then the corrector and the shifting, wall by wall in the
    # order the cells are visited (x offset outermost)
    ri, rj = torch.cat(reach_i), torch.cat(reach_j)
    cell = keys[rj] - keys[ri]
    nx1 = nxs[cid[ri], 1]
    nx2 = nxs[cid[ri], 2] if D == 3 else torch.ones_like(nx1)
    if D == 3:
        dz = torch.round(cell.double() / nx2).long()
        dy = torch.round((cell - dz * nx2).double() / nx1).long()
    else:
        dz = torch.zeros_like(cell)
        dy = torch.round(cell.double() / nx1).long()
    dxc = cell - dz * nx2 - dy * nx1 if D == 3 else cell - dy * nx1
    rank = ((dxc + 1) * 9 + (dy + 1) * 3 + (dz + 1)) * n + rj
    o = torch.argsort(rank, stable=True)
    o = o[torch.argsort(ri[o], stable=True)]
    ri, rj = ri[o], rj[o]
    if ri.numel():
        cnt = torch.bincount(ri, minlength=n)
        first = torch.cumsum(cnt, 0) - cnt
        turn = torch.arange(ri.shape[0], device="cuda") - first[ri]
        rounds = [(ri[turn == k], rj[turn == k]) for k in range(int(turn.max().item()) + 1)]
    else:
        rounds = []
    acc = torch.where(fl[:, None], acc, ain)
    for i, j in rounds:
        nj, dti = nrm[j], dt[i]
        vh = uin[i] + 0.5 * dti[:, None] * acc[i]
        d = rin[j] - rin[i]
        rn = (d * nj).sum(1)
        tt = d - rn[:, None] * nj
        drn = dti * (vh * nj).sum(1)
        hit = ((rn >= 0) & ((tt * tt).sum(1) < (p.dr_factor * dr_w[j]) ** 2) & (drn >= 0)
               & (rn - drn <= p.min_bound_dist * dr_w[j]))
        v = uin[i] + dti[:, None] * acc[i]
        vr = v - 2 * (v * nj).sum(1)[:, None] * nj
        acc[i] = torch.where(hit[:, None], (vr - uin[i]) / dti[:, None], acc[i])
    drho = torch.where(fl, drho, din)
    rn_ = torch.where(fl[:, None], rin + dt[:, None] * uin + 0.5 * dt[:, None] ** 2 * acc, rin)
    un = torch.where(fl[:, None], uin + dt[:, None] * acc, u)
    rho_n = torch.where(fl, rhoin + dt * drho, rho)
    Ri = 0.5 * (x["m"].clamp_min(0) / rho_n) ** (1.0 / D)
    for i, j in rounds:
        nj = nrm[j]
        d = rin[j] - rn_[i]
        rn = (d * nj).sum(1)
        tt = d - rn[:, None] * nj
        hit = (rn.abs() <= Ri[i]) & ((tt * tt).sum(1) < (p.dr_factor * dr_w[j]) ** 2)
        rn_[i] = torch.where(hit[:, None], rn_[i] + (rn - Ri[i])[:, None] * nj, rn_[i])
    sh = torch.where(shep < 1e-6, torch.ones_like(shep), shep)
    un = torch.where(probe[:, None], su / sh[:, None], un)
    rho_n = torch.where(probe, srho / sh, rho_n)
    pr = torch.where(probe, sp / sh, pr)
    dt_u = p.courant * p.dt_Ma * p.h / (un * un).sum(1).sqrt().clamp_min(1e-300)
    dt_v = torch.where(fl, dt_u.clamp_max(p.dt_fixed).clamp_min(p.dt_min), torch.full_like(dt_u, p.dt_fixed))
    dt_new = torch.full_like(dt_case, math.inf).scatter_reduce_(0, cid, dt_v, "amin")
    nrm = nrm.clone()
    for k, mo in enumerate(motions):
        if mo is None:
            continue
        at = (cid == k) & (x["iset"] == mo.iset) & ~fl
        t0, t1 = float(t_case[k]), float(t_case[k] + dt_new[k])
        psi = [mo.amplitude * math.sin(mo.angular_freq * v) for v in (t0, t1)]
        om = mo.amplitude * mo.angular_freq * math.cos(mo.angular_freq * t1)
        cen = torch.tensor(mo.center[:D], dtype=torch.float64, device="cuda")
        turn = lambda v, s: torch.stack([math.cos(s) * v[:, 0] - math.sin(s) * v[:, 1],  # noqa: E731
                                         math.sin(s) * v[:, 0] + math.cos(s) * v[:, 1]], 1)
        loc = turn(rn_[at] - cen, -psi[0])
        un[at] = turn(torch.stack([-om * loc[:, 1], om * loc[:, 0]], 1), psi[1])
        rn_[at] = turn(loc, psi[1]) + cen
        nn = turn(turn(nrm[at], -psi[0]), psi[1])
        nrm[at] = nn / (nn * nn).sum(1).sqrt().clamp_min(1e-300)[:, None]
    vs = x["r"].shape[1]

    def vec(v):
        return torch.nn.functional.pad(v, (0, vs - D))

    x.update(r=vec(rn_), u=vec(un), dudt=vec(acc), normal=vec(nrm), rho=rho_n, drhodt=drho,
             p=pr, shepard=torch.where((im >= -3) & (im <= 1), shep, torch.zeros_like(shep)))
    return x, dt_new


NET = [("e1_0", 64, 16, 1), ("e1_1", 64, 64, 1), ("e1_2", 64, 64, 0),
       ("n1_0", 64, 80, 1), ("n1_1", 64, 64, 1), ("n1_2", 64, 64, 0),
       ("e2_0", 64, 144, 1), ("e2_1", 64, 64, 1), ("e2_2", 64, 64, 0),
       ("n2_0", 64, 144, 1), ("n2_1", 64, 64, 1), ("n2_2", 16, 64, 0)]


def _exact_learned(case, seed):
    b, p, s, cid = _slosh_state(case, seed)
    rng = np.random.default_rng(int(seed))
    flat = []
    for name, n, k, act in NET:
        std = math.sqrt((2.0 if act else 1.0) / k) * (0.1 if name == "n2_2" else 1.0)
        w = torch.from_numpy(rng.normal(0, std, (n, k)).astype(np.float32)).cuda()
        flat += [w.bfloat16().double().reshape(-1), torch.zeros(n, dtype=torch.float64, device="cuda")]
    train = case["kind"] == "train"
    flat = torch.cat(flat).requires_grad_(train)
    W, o = {}, 0
    for name, n, k, act in NET:
        W[name] = (flat[o:o + n * k].reshape(n, k), flat[o + n * k:o + n * k + n], act)
        o += n * k + n

    def mlp(pre, v):
        for k in range(3):
            w, bias, act = W["%s_%d" % (pre, k)]
            v = v @ w.t() + bias
            v = torch.nn.functional.silu(v) if act else v
        return v

    # nodes in particle order (no probes), edges by the float distance test
    rad = np.float32(float(p.support * p.h))
    r2 = float(np.float32(rad * rad))
    node = torch.nonzero(s["imove"] != 0).reshape(-1)
    keys, nxs = _keys(s["r"], 2, float(rad), cid.long())
    order = node[torch.argsort(keys[node], stable=True)]
    ks, cs = keys[order], cid.long()[order]
    rs = s["r"][order]
    i, j = [], []
    for lo in range(0, order.shape[0], 200000):
        a, c = _neighbour_pairs(ks, nxs, cs, 2, lo, min(order.shape[0], lo + 200000))
        d = rs[c] - rs[a]
        ok = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] < r2) & (a != c)
        i.append(a[ok])
        j.append(c[ok])
    i, j = torch.cat(i), torch.cat(j)
    nn = order.shape[0]
    U, R, A, Rd = MODEL_SCALES
    h = float(np.float32(p.h))
    x = {k: v[order].double() if v.is_floating_point() else v[order] for k, v in s.items()}
    wall = (x["imove"] < 0).double()
    F = torch.zeros((nn, 16), dtype=torch.float64, device="cuda")
    F[:, 0:2], F[:, 2], F[:, 3:5] = x["u"] / U, (x["rho"] - REFD) / R, x["dudt"] / A
    F[:, 5], F[:, 6], F[:, 7] = x["drhodt"] / Rd, (x["imove"] == 1).double(), wall
    F[:, 8:10] = x["normal"] * wall[:, None]

    def edges(a, c):
        d = x["r"][c] - x["r"][a]
        E = torch.zeros((a.shape[0], 16), dtype=torch.float64, device="cuda")
        q = (d * d).sum(1).sqrt() / h
        E[:, 0:2], E[:, 2], E[:, 3:5] = d / h, q, (x["u"][c] - x["u"][a]) / U
        E[:, 5] = (x["rho"][c] - x["rho"][a]) / R
        E[:, 6] = torch.where(q < 2, (1 + 2 * q) * (1 - 0.5 * q) ** 4, torch.zeros_like(q))
        E[:, 7] = wall[c]
        E[:, 8:10] = x["normal"][c] * wall[c][:, None]
        return E

    def summed(pre, Hn=None):
        total = torch.zeros((nn, 64), dtype=torch.float64, device="cuda")
        for lo in range(0, i.shape[0], 2000000):
            a, c = i[lo:lo + 2000000], j[lo:lo + 2000000]
            E = edges(a, c)
            v = E if Hn is None else torch.cat([Hn[a], Hn[c], E], 1)
            total = total.index_add(0, a, mlp(pre, v))
        return total / 32.0

    with torch.set_grad_enabled(train):
        Hn = mlp("n1", torch.cat([summed("e1"), F], 1))
        out = mlp("n2", torch.cat([summed("e2", Hn), Hn, F], 1))
        T = K_STEPS * float(np.float32(p.dt_fixed))
        fl = x["imove"] == 1
        if train:
            y = _later(s, p.dt_fixed, seed)
            y = {k: y[k][order].double() for k in ("u", "rho")}
            tu = (y["u"] - x["u"] - T * x["dudt"]) / OUT_SCALE[0]
            tr = (y["rho"] - x["rho"] - T * x["drhodt"]) / OUT_SCALE[1]
            diff = out[:, :3] - torch.cat([tu, tr[:, None]], 1)
            loss = (diff[fl] ** 2).sum() / fl.sum()
            loss.backward()
            return {"loss": loss.detach().reshape(1), "grad": flat.grad, "out": None}
    new = {k: s[k].double() for k in ("r", "u", "rho")}
    f1 = fl.double()
    u1 = x["u"] + (T * x["dudt"] + OUT_SCALE[0] * out[:, :2]) * f1[:, None]
    new["u"][order] = u1
    new["r"][order] = x["r"] + 0.5 * T * (x["u"] + u1) * f1[:, None]
    new["rho"][order] = x["rho"] + (T * x["drhodt"] + OUT_SCALE[1] * out[:, 2]) * f1
    return {"out": None, **new}
