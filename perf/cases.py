"""The workloads this library's speed is judged on.

Every case is one call sequence of the Python package (``bfvm``), the way a
host simulation uses it: the microenvironment stays on the GPU, the host code
sends agents, advances a number of diffusion steps and reads back what it
needs.  A case is a dict of plain values; ``kind`` says which sequence:

``steps``     advance ``steps`` diffusion steps with the agents' sources, and
              read the densities at the agents when ``sample`` is set;
``interval``  one mechanics interval: the agents have moved, so the whole list
              is sent again from its rates, ten steps follow, and every
              agent's densities come back to the host;
``batch``     many solves of different shapes advanced together;
``gradients`` the gradient of every substrate at every voxel, on the device;
``field``     the field handed over in the reference's layout and taken back,
              both in device memory;
``plane``     the 2-D solver with its Dirichlet nodes on the rim;
``bulk``      per-voxel supply and uptake, then the substrates' totals.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "physicell-x_b200"))

from bfvm import Batch, Microenvironment  # noqa: E402

DT = 0.01  # min, the diffusion time step of every configuration
VOLUME = 2494.0  # um^3, a cell's volume


def listed():
    return [
        # A small tissue: 50^3 voxels, an oxygen-like and a secreted substrate,
        # one mechanics interval of ten steps; launches and latency count.
        _steps("small_tissue_fp64", 50, 50, 50, 2, "fp64", 2000, 10, medium="tissue", sample=True),
        # The usual benchmark grid, 200^3 with four substrates and 100,000
        # agents, in both precisions.
        _steps("cube200_fp64", 200, 200, 200, 4, "fp64", 100_000, 10),
        _steps("cube200_fp32", 200, 200, 200, 4, "fp32", 100_000, 10),
        # The largest domain, 640^3 with a million agents in a ball.
        _steps("cube640_fp64", 640, 640, 640, 2, "fp64", 1_000_000, 2, medium="tissue", ball=True),
        # The same in the FP32 form under the partitioned chain, the setting for
        # long lines.
        _steps("cube640_fp32_chain2", 640, 640, 640, 2, "fp32", 1_000_000, 2, medium="tissue", ball=True, chain=2),
        # A request to a serving loop: ragged extents, five substrates, faces
        # with their own values; enough steps for the library's graph replay.
        _steps("ragged_request_fp64", 97, 211, 143, 5, "fp64", 60_000, 32),
        # Agents that move: the list is rebuilt for every mechanics interval.
        {"name": "moving_agents_fp64", "kind": "interval", "nx": 200, "ny": 200, "nz": 200, "S": 4,
         "precision": "fp64", "agents": 100_000},
        # A parameter sweep: 24 uneven solves of edges 24-128 stepped together.
        {"name": "uneven_batch_fp32", "kind": "batch", "members": 24, "edge_hi": 128, "precision": "fp32", "steps": 16},
        # Chemotaxis needs every gradient.
        {"name": "gradients_fp64", "kind": "gradients", "nx": 200, "ny": 200, "nz": 200, "S": 4, "precision": "fp64"},
        # A coupled GPU code hands the field over and takes it back.
        {"name": "field_exchange_fp64", "kind": "field", "nx": 200, "ny": 200, "nz": 200, "S": 4, "precision": "fp64"},
        # A 2-D simulation (one layer of voxels).
        {"name": "plane_fp64", "kind": "plane", "nx": 300, "ny": 260, "S": 3, "precision": "fp64", "agents": 10_000,
         "steps": 10},
        # Perfusion by per-voxel supply rates, checked by the totals.
        {"name": "bulk_totals_fp64", "kind": "bulk", "nx": 160, "ny": 200, "nz": 120, "S": 3, "precision": "fp64"},
    ]


def _steps(name, nx, ny, nz, S, precision, agents, steps, medium="random", ball=False, chain=0, sample=False,
           track=False):
    c = {"kind": "steps", "nx": nx, "ny": ny, "nz": nz, "S": S, "precision": precision, "agents": agents,
         "steps": steps, "medium": medium, "ball": ball, "chain": chain, "sample": sample, "track": track}
    if name:
        c["name"] = name
    return c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["steps", "interval", "batch", "gradients", "field", "plane", "bulk"],
                       [10, 2, 1, 1, 1, 2, 1])[0]
    precision = rng.choice(["fp64", "fp64", "fp32"])
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(8, 24), "edge_hi": _log(rng, 40, 128), "precision": precision,
                "steps": rng.randint(4, 16)}
    if kind == "plane":
        return {"kind": kind, "nx": _log(rng, 60, 700), "ny": _log(rng, 60, 700), "S": rng.randint(1, 4),
                "precision": precision, "agents": _log(rng, 500, 20_000), "steps": rng.randint(1, 10)}
    S = rng.randint(1, 8)
    cap = 1 << 26 if kind == "steps" else 1 << 25  # values of the field
    while True:
        nx, ny, nz = (_log(rng, 24, 640 if kind == "steps" else 256) for _ in range(3))
        if nx * ny * nz * S <= cap:
            break
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "S": S, "precision": precision}
    agents = max(200, min(200_000, int(nx * ny * nz * math.exp(rng.uniform(math.log(0.002), math.log(0.1))))))
    if kind == "steps":
        steps = min(_log(rng, 1, 32), 2 * 640 ** 3 * 2 // (nx * ny * nz * S))  # no more than the largest listed case
        c = _steps(None, nx, ny, nz, S, precision, agents, steps, medium="random",
                   ball=rng.random() < 0.3, chain=rng.choice([0, 0, 0, 1, 2]), sample=rng.random() < 0.3,
                   track=rng.random() < 0.15)
    elif kind == "interval":
        c["agents"] = agents
    return c


# ---- inputs ----------------------------------------------------------------


def _medium(case, rng):
    """Diffusion coefficients, decay rates, Dirichlet activation and one value
    per face and substrate (faces in the order xmin, xmax, ymin, ...)."""
    S = case["S"]
    if case.get("medium") == "tissue":  # oxygen-like, and a secreted substrate
        return (np.array([1e5, 1e3]), np.array([0.1, 0.01]), np.array([1, 0], np.uint8),
                np.tile(np.array([38.0, 1.0]), (6, 1)))
    D = np.exp(rng.uniform(math.log(1e2), math.log(1e5), S))
    decay = np.exp(rng.uniform(math.log(1e-3), 0.0, S))
    active = (rng.uniform(0, 1, S) < 0.5).astype(np.uint8)
    active[0] = 1
    faces = np.ones((6, S))
    on = rng.uniform(0, 1, (6, S)) < 0.6
    faces[on] = rng.uniform(0.0, 50.0, int(on.sum()))
    return D, decay, active, faces


def _dx(case):
    return 20.0 if case["kind"] in ("plane", "batch") or case["nx"] <= 64 else 10.0


def _agents(case, rng, n):
    """Voxels and rates of n agents: uniform in the box, or a ball of cells."""
    nx, ny, nz, S = case["nx"], case["ny"], case.get("nz", 1), case["S"]
    ext = np.array([nx, ny, nz], np.float64)
    if case.get("ball"):
        pos = ext / 2 + rng.normal(0.0, 0.23 * ext.min(), (n, 3))
    else:
        pos = rng.uniform(0.0, 1.0, (n, 3)) * ext
    ijk = np.clip(np.floor(pos).astype(np.int64), 0, np.array([nx, ny, nz]) - 1)
    voxel = ((ijk[:, 0] * ny + ijk[:, 1]) * nz + ijk[:, 2]).astype(np.int32)
    if case.get("medium") == "tissue":
        uptake, secretion = np.zeros((n, 2)), np.zeros((n, 2))
        uptake[:, 0], secretion[:, 1] = 10.0, 1.0
    else:
        uptake, secretion = rng.uniform(0.0, 10.0, (n, S)), rng.uniform(0.0, 1.0, (n, S))
    export = rng.uniform(0.0, 5.0, (n, S)) * (rng.uniform(0, 1, (n, 1)) < 0.1)
    return {"voxel": voxel, "volume": np.full(n, VOLUME), "secretion": secretion, "uptake": uptake,
            "saturation": np.ones((n, S)), "net_export": export}


def _field(case, seed):
    """The initial field in the reference's layout [x][y][z][substrate]."""
    nx, ny, nz, S = case["nx"], case["ny"], case.get("nz", 1), case["S"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.rand((nx, ny, nz, S), dtype=torch.float64, device="cuda", generator=g)
    if case.get("medium") == "tissue":  # 38 everywhere with a little noise; traces of the secreted one
        f[..., 0].mul_(0.5).add_(37.5)
        f[..., 1].mul_(0.1)
    else:
        f.mul_(40.0)
    return f


def _planes(case, faces):
    """The six face planes; a shared edge has the value of the later face."""
    nx, ny, nz, S = case["nx"], case["ny"], case.get("nz", 1), case["S"]
    x = [np.broadcast_to(faces[q], (ny, nz, S)).copy() for q in (0, 1)]
    y = [np.broadcast_to(faces[q], (nx, nz, S)).copy() for q in (2, 3)]
    z = [np.broadcast_to(faces[q], (nx, ny, S)).copy() for q in (4, 5)]
    for p in x:
        p[0], p[-1] = faces[2], faces[3]
    for p in x + y:
        p[:, 0], p[:, -1] = faces[4], faces[5]
    return x + y + z


class _Buffer:
    """A solve's device field, [S][nz][ny][nx] inside padded rows.  A tensor on
    it keeps this object, and so the solve, alive."""

    def __init__(self, me):
        self.owner = me
        ptr, pitch, size = me.device_field()
        nx, ny, nz, S = me.shape
        self.__cuda_array_interface__ = {
            "data": (ptr, False), "typestr": "<f%d" % size, "version": 3, "shape": (S, nz, ny, nx),
            "strides": (nz * ny * pitch * size, ny * pitch * size, pitch * size, size)}


def _solve(case, seed, rng):
    D, decay, active, faces = _medium(case, rng)
    me = Microenvironment(case["nx"], case["ny"], case.get("nz", 1), _dx(case), DT, D, decay, case["precision"])
    me.set_dirichlet_activation(active)
    for q, p in enumerate(_planes(case, faces)):
        me.set_dirichlet_face(q, p)
    f = _field(case, seed)
    torch.cuda.synchronize()
    me.upload_field_device(f.data_ptr())
    me.synchronize()
    return me, f


def _rim(case, rng):
    """Dirichlet nodes of the 2-D solver: the rim, for one substrate in two."""
    nx, ny, S = case["nx"], case["ny"], case["S"]
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    v = (i * ny + j)[(i == 0) | (i == nx - 1) | (j == 0) | (j == ny - 1)].astype(np.int32)
    on = np.zeros(S, np.uint8)
    on[::2] = 1
    return v, np.broadcast_to(rng.uniform(0.0, 50.0, S), (v.size, S)).copy(), np.broadcast_to(on, (v.size, S)).copy()


def _shapes(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 5]))
    # the shapes belong to the case, the values to the seed
    fixed = np.random.Generator(np.random.PCG64([case["members"], case["edge_hi"]]))
    for q in range(case["members"]):
        nx, ny, nz = (int(v) for v in fixed.integers(24, case["edge_hi"] + 1, 3))
        yield {"kind": "batch", "nx": nx, "ny": ny, "nz": nz, "S": int(fixed.integers(1, 7)),
               "precision": case["precision"], "agents": int(fixed.integers(0, 20_001))}, seed * 1000 + q, rng


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        batch, members = Batch(case["precision"]), []
        batch.set_schedule(mode=2)  # the serving loop's
        for one, s, rng in _shapes(case, seed):
            me, _ = _solve(one, s, rng)
            if one["agents"]:
                me.set_agents_from_rates(**_agents(one, rng, one["agents"]))
            batch.add(me)
            members.append(me)
        batch.synchronize()
        return {"case": case, "batch": batch, "members": members,
                "fields": [torch.as_tensor(_Buffer(me), device="cuda") for me in members]}
    rng = np.random.Generator(np.random.PCG64(seed))
    me, f = _solve(case, seed, rng)
    st = {"case": case, "me": me, "field": torch.as_tensor(_Buffer(me), device="cuda")}
    nx, ny, nz, S = me.shape
    if kind in ("steps", "plane"):
        if case.get("chain"):
            me.set_fp64_chain(case["chain"])
        if case.get("track"):
            me.set_track_internalized_substrates(True)
        me.set_agents_from_rates(**_agents(case, rng, case["agents"]))
    if kind == "plane":
        me.set_dirichlet_nodes(*_rim(case, rng))
    elif kind == "interval":
        # where the agents were, and where they are now
        me.set_agents_from_rates(**_agents(case, rng, case["agents"]))
        st["agents"] = _agents(case, rng, case["agents"])
    elif kind == "gradients":
        st["out"] = torch.empty((nx * ny * nz, S, 3), dtype=torch.float64, device="cuda")
    elif kind == "field":
        st["in"] = f.flip(0).contiguous()
        st["out"] = torch.empty_like(f)
    elif kind == "bulk":
        me.set_bulk_rates(*_bulk(case, rng))
    me.synchronize()
    torch.cuda.synchronize()
    return st


def _bulk(case, rng):
    """Supply where vessels are (one voxel in fifty), uptake everywhere."""
    n = (case["nx"] * case["ny"] * case["nz"], case["S"])
    supply = 20.0 * (rng.random(n) < 0.02)
    return supply, np.full(n, 38.0), 5.0 * rng.random(n)


# ---- one pass --------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].step(case["steps"], sources=True)
        return state["fields"]
    me, field = state["me"], state["field"]
    if kind == "steps":
        me.simulate_diffusion_decay(case["steps"], sources=True)
        out = {"field": field}
        if case["track"]:
            out["internalized"] = me.internalized_substrates()
        if case["sample"]:
            out["densities"] = me.sample_agents()
        return out
    if kind == "interval":
        me.set_agents_from_rates(**state["agents"])
        me.simulate_diffusion_decay(10, sources=True)
        return {"field": field, "densities": me.sample_agents()}
    if kind == "gradients":
        me.compute_all_gradient_vectors_device(state["out"].data_ptr())
        return state["out"]
    if kind == "field":
        me.upload_field_device(state["in"].data_ptr())
        me.download_field_device(state["out"].data_ptr())
        return {"field": field, "out": state["out"]}
    if kind == "plane":
        me.simulate_diffusion_decay_2d(case["steps"], sources=True)
        return field
    me.simulate_bulk_sources_and_sinks()
    return {"field": field, "totals": me.field_sums()}


# ---- what a pass cannot do without -----------------------------------------


def _step_work(c, sweeps):
    """One diffusion step: each sweep reads and writes the field once; the
    agents' constants and voxels are read, their densities read and written.
    A value takes five operations forward (an FMA, a division's multiply and
    one correction counted as three) and two back."""
    n = c["nx"] * c["ny"] * c.get("nz", 1) * c["S"]
    w = 8 if c["precision"] == "fp64" else 4
    a = c["agents"] * c["S"]
    return sweeps * 2 * n * w + a * (24 + 2 * w) + 4 * c["agents"], sweeps * 7 * n + 3 * a


def work(case):
    kind = case["kind"]
    if kind == "batch":
        each = [_step_work(c, 3) for c, _, _ in _shapes(case, 0)]
        return {"bytes": case["steps"] * sum(b for b, _ in each), "flops": case["steps"] * sum(f for _, f in each)}
    n = case["nx"] * case["ny"] * case.get("nz", 1) * case["S"]
    w = 8 if case["precision"] == "fp64" else 4
    if kind in ("steps", "plane", "interval"):
        b, f = _step_work(case, 2 if kind == "plane" else 3)
        k = case.get("steps", 10)
        a = case["agents"] * case["S"]
        b, f = k * b, k * f
        if case.get("track"):
            b += 16 * a * k
        if kind == "interval":  # the rates in, the constants out
            b, f = b + a * (32 + 24) + 12 * case["agents"], f + 9 * a
        if case.get("sample") or kind == "interval":
            b += a * (8 + w)
        return {"bytes": b, "flops": f}
    if kind == "gradients":
        return {"bytes": n * (w + 24), "flops": 6 * n}
    if kind == "field":
        return {"bytes": n * 2 * (8 + w), "flops": 0}
    return {"bytes": n * (24 + 2 * w), "flops": 8 * n}


# ---- the same in plain 64-bit torch ----------------------------------------


def _thomas(n, k1, k2):
    """Factors of one axis: the constant tridiagonal system with zero flux."""
    d = np.empty((n, k1.size))
    c = np.empty_like(d)
    for i in range(n):
        d[i] = 1.0 + k2 + (0.0 if n == 1 else k1 if i in (0, n - 1) else 2.0 * k1)
        if i:
            d[i] += k1 * c[i - 1]
        c[i] = -k1 / d[i]
    return torch.from_numpy(d).cuda(), torch.from_numpy(c).cuda()


def _sweep(f, axis, k1, factors):
    """Solve along one axis of f [nx][ny][nz][S] in place."""
    d, c = factors
    k = torch.from_numpy(k1).cuda()
    rows = f.unbind(axis)
    rows[0].div_(d[0])
    for i in range(1, len(rows)):
        rows[i].add_(rows[i - 1] * k).div_(d[i])
    for i in range(len(rows) - 2, -1, -1):
        rows[i].sub_(rows[i + 1] * c[i])


def _pin(f, active, planes):
    for s in np.flatnonzero(active):
        for q, p in enumerate(planes):
            p = torch.from_numpy(p[..., s]).cuda()
            f.select(q // 2, 0 if q % 2 == 0 else f.shape[q // 2] - 1)[..., s] = p


class _Sources:
    """The agents in list order: agents that share a voxel follow each other."""

    def __init__(self, case, a, dx):
        v3 = dx * dx * dx
        k = (DT * a["volume"] / v3)[:, None]
        c = (a["secretion"] * a["saturation"] * k, 1.0 + k * (a["secretion"] + a["uptake"]),
             a["net_export"] * DT / v3)
        order = np.argsort(a["voxel"], kind="stable")
        v = a["voxel"][order]
        first = np.r_[0, np.flatnonzero(v[1:] != v[:-1]) + 1] if v.size else np.zeros(0, np.int64)
        rank = np.arange(v.size) - np.repeat(first, np.diff(np.r_[first, v.size]))
        self.rounds = []
        for r in range(int(rank.max()) + 1 if v.size else 0):
            at = order[rank == r]
            self.rounds.append([torch.from_numpy(x).cuda() for x in (at, a["voxel"][at].astype(np.int64), *(y[at] for y in c))])
        self.export = torch.from_numpy(a["net_export"] * DT).cuda()
        self.internal = torch.zeros((a["voxel"].size, case["S"]), dtype=torch.float64, device="cuda")
        self.voxel, self.v3 = torch.from_numpy(a["voxel"].astype(np.int64)).cuda(), v3

    def __call__(self, f):
        flat = f.view(-1, f.shape[-1])
        for at, v, c1, c2, e2 in self.rounds:
            r = flat[v]
            self.internal[at] -= (((1.0 - c2) * r + c1) / c2) * self.v3 + self.export[at]
            flat[v] = (r + c1) / c2 + e2

    def sample(self, f):
        return f.view(-1, f.shape[-1])[self.voxel]


def _exact_solve(case, seed, rng, agents, steps):
    """The field after `steps` steps, in the reference's layout, and the agents."""
    D, decay, active, faces = _medium(case, rng)
    planes, f, dx = _planes(case, faces), _field(case, seed), _dx(case)
    src = [_Sources(case, a, dx) for a in agents(rng)]
    k1, k2 = D * DT / dx / dx, decay * DT / 3.0
    fac = [_thomas(n, k1, k2) for n in f.shape[:3]]
    for _ in range(steps):
        if src:
            src[-1](f)
        _pin(f, active, planes)
        for axis in range(3):
            _sweep(f, axis, k1, fac[axis])
            _pin(f, active, planes)
    return f, src, (active, planes)


def _stored(f, case, active, planes):
    """The device's layout; an FP32 solve stores differences from the mean
    boundary value of each activated substrate."""
    f = f.permute(3, 2, 1, 0)
    if case["precision"] == "fp64":
        return f
    off = [sum(p[..., s].sum() for p in planes) / sum(p[..., s].size for p in planes) if active[s] else 0.0
           for s in range(case["S"])]
    return f - torch.tensor(off, dtype=torch.float64, device="cuda").view(-1, 1, 1, 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for one, s, rng in _shapes(case, seed):
            n = one["agents"]
            f, _, bc = _exact_solve(one, s, rng, lambda r: [_agents(one, r, n)] if n else [], case["steps"])
            out.append(_stored(f, one, *bc))
        return out
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind in ("steps", "interval"):
        lists = 2 if kind == "interval" else 1
        f, src, bc = _exact_solve(case, seed, rng, lambda r: [_agents(case, r, case["agents"]) for _ in range(lists)],
                                  case.get("steps", 10))
        out = {"field": _stored(f, case, *bc)}
        if case.get("track"):
            out["internalized"] = src[-1].internal
        if case.get("sample") or kind == "interval":
            out["densities"] = src[-1].sample(f)
        return out
    if kind == "plane":
        D, decay, active, faces = _medium(case, rng)
        planes, f, dx = _planes(case, faces), _field(case, seed), _dx(case)
        src = _Sources(case, _agents(case, rng, case["agents"]), dx)
        v, val, on = (torch.from_numpy(x).cuda() for x in _rim(case, rng))
        k1, k2 = D * DT / dx / dx, decay * DT * 0.5
        fac = [_thomas(n, k1, k2) for n in f.shape[:2]]

        def nodes():
            flat = f.view(-1, case["S"])
            flat[v.long()] = torch.where(on.bool(), val, flat[v.long()])

        for _ in range(case["steps"]):
            src(f)
            nodes()
            for axis in range(2):
                _sweep(f, axis, k1, fac[axis])
                nodes()
        return _stored(f, case, active, planes)
    _, _, active, faces = _medium(case, rng)
    planes, f = _planes(case, faces), _field(case, seed)
    if kind == "gradients":
        g, dx = torch.zeros((*f.shape, 3), dtype=torch.float64, device="cuda"), _dx(case)
        for a in range(3):
            n = f.shape[a]
            if n < 2:
                continue
            lo = torch.arange(n, device="cuda").sub_(1).clamp_(min=0)
            hi = torch.arange(n, device="cuda").add_(1).clamp_(max=n - 1)
            h = ((hi - lo).double() * dx).view([-1 if q == a else 1 for q in range(4)])
            g[..., a] = (f.index_select(a, hi) - f.index_select(a, lo)) / h
        return g.view(-1, case["S"], 3)
    if kind == "field":
        f = f.flip(0).contiguous()
        return {"field": _stored(f, case, active, planes), "out": f}
    supply, target, uptake = (torch.from_numpy(x).cuda().view(f.shape) for x in _bulk(case, rng))
    f = (f + DT * supply * target) / (1.0 + DT * (supply + uptake))
    return {"field": _stored(f, case, active, planes), "totals": f.sum((0, 1, 2))}
