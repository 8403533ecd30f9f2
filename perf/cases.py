"""Timing cases of the force path: what a program that uses this framework has it do.

Every case goes through the package's own entry points (the solver classes, the server, the device
pointer calls of include/nbody_gpu.h) on seeded synthetic bodies of the shapes the configurations
use: a uniform ball, Plummer spheres, two colliding Hernquist spheres. Kinds of case:

  forces    one force evaluation in a host program: bodies in, accelerations out
  scenario  a short run in a host program: bodies in, a few steps, bodies out
  step      device-resident stepping of one body set
  dual      device-resident stepping with the dual-tree solver
  batch     device-resident stepping of many independent instances, graph-captured
  serve     requests through the continuous-batching server until all are done
  sort      the allocation-free Morton-code sort
  direct64  FP64 direct sum over a sample of targets (the accuracy check beside a run)
  energy    FP64 energy diagnostics of a body set
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "n-body_b200"))
import nbody_b200 as nb  # noqa: E402


def listed():
    return [
        # a small interactive scene on the drop-in boundary: the caller's program owns the bodies and
        # asks for accelerations each frame; latency and launches count
        {"name": "forces-1k", "kind": "forces", "solver": "quadrupole", "dist": "plummer", "n": 1023, "theta": 0.5,
         "leaf": 16, "epsilon": 1e-4},
        # the 10,000-body scenario of the configurations, whole: monopole tree, ten steps, host in and out
        {"name": "scenario-10k", "kind": "scenario", "solver": "monopole", "dist": "ball", "n": 10000, "theta": 0.5,
         "leaf": 16, "epsilon": 1e-4, "steps": 10, "dt": 1e-3},
        # the drop-in solver at the reference's own defaults (theta 0.3, leaf 64, epsilon 1e-5), ragged size
        {"name": "forces-100k", "kind": "forces", "solver": "monopole", "dist": "plummer", "n": 100003, "theta": 0.3,
         "leaf": 64, "epsilon": 1e-5},
        # the headline run: 2^20-body Plummer sphere, quadrupoles, device-resident steps
        {"name": "step-1m", "kind": "step", "solver": "quadrupole", "dist": "plummer", "n": 1 << 20, "theta": 0.5,
         "leaf": 16, "epsilon": 2.5e-5, "steps": 1, "dt": 5e-4},
        # the direct-sum solver on a set where a tree is not worth it, ragged size
        {"name": "forces-naive-30k", "kind": "forces", "solver": "naive", "dist": "plummer", "n": 30011, "theta": 0.5,
         "leaf": 16, "epsilon": 1e-4},
        # the dual-tree solver on a laptop-sized pair of galaxies
        {"name": "dual-60k", "kind": "dual", "n": 60001, "theta": 0.5, "leaf": 32, "epsilon": 2.5e-5, "dt": 1e-3},
        # the precision study: two colliding spheres of 2^21 bodies each
        {"name": "dual-4m", "kind": "dual", "n": 1 << 22, "theta": 0.4, "leaf": 64, "epsilon": 2.5e-5, "dt": 1e-3},
        # the batch configuration: 256 uneven instances, two graph-captured steps per call
        {"name": "batch-256", "kind": "batch", "mix": 44, "count": 256, "n_min": 1024, "n_max": 200000, "leaf": 16,
         "epsilon": 1e-4, "steps": 2, "dt": 1e-3},
        # a burst of served requests, from admission to results
        {"name": "serve-12", "kind": "serve", "mix": 47, "count": 12, "n_min": 2048, "n_max": 65536, "leaf": 16,
         "epsilon": 1e-4, "steps": 8, "dt": 1e-3},
        # Morton codes of a snapshot sorted for a caller that may not allocate
        {"name": "sort-1m", "kind": "sort", "n": 1000003},
        # the accuracy check of a run: 4096 sampled targets against all bodies in FP64
        {"name": "direct64-4k", "kind": "direct64", "n": 1 << 18, "targets": 4096, "epsilon": 2.5e-5},
        # energy diagnostics of a 40,000-body set
        {"name": "energy-40k", "kind": "energy", "n": 40009, "epsilon": 1e-4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forces", "forces", "forces", "scenario", "scenario", "step", "step", "step", "dual", "dual",
                       "batch", "serve", "sort", "direct64", "energy"])
    solver = rng.choice(["quadrupole", "quadrupole", "monopole"])
    theta = round(rng.uniform(0.3, 0.7), 3)
    leaf = rng.choice([8, 16, 16, 32, 64])
    epsilon = rng.choice([1e-5, 2.5e-5, 1e-4])
    dist = rng.choice(["ball", "plummer"])
    dt = rng.choice([5e-4, 1e-3])
    if kind == "forces":
        if rng.random() < 0.25:
            return {"kind": kind, "solver": "naive", "dist": dist, "n": _log(rng, 500, 65536), "theta": 0.5,
                    "leaf": 16, "epsilon": epsilon}
        return {"kind": kind, "solver": solver, "dist": dist, "n": _log(rng, 500, 400000), "theta": theta,
                "leaf": leaf, "epsilon": epsilon}
    if kind == "scenario":
        return {"kind": kind, "solver": solver, "dist": dist, "n": _log(rng, 500, 100000), "theta": theta,
                "leaf": leaf, "epsilon": epsilon, "steps": rng.randint(2, 16), "dt": dt}
    if kind == "step":
        return {"kind": kind, "solver": solver, "dist": "plummer", "n": _log(rng, 2000, 1500000),
                "theta": round(rng.uniform(0.4, 0.7), 3), "leaf": leaf, "epsilon": epsilon,
                "steps": rng.randint(1, 3), "dt": dt}
    if kind == "dual":
        return {"kind": kind, "n": _log(rng, 4000, 1000000), "theta": round(rng.uniform(0.4, 0.6), 3),
                "leaf": rng.choice([32, 64]), "epsilon": epsilon, "dt": dt}
    if kind == "batch":
        return {"kind": kind, "mix": rng.randrange(1000), "count": rng.randint(8, 200), "n_min": 1024,
                "n_max": _log(rng, 8192, 100000), "leaf": rng.choice([8, 16]), "epsilon": epsilon, "steps": 2 * rng.randint(1, 2), "dt": dt}
    if kind == "serve":
        return {"kind": kind, "mix": rng.randrange(1000), "count": rng.randint(4, 24), "n_min": 2048,
                "n_max": _log(rng, 8192, 131072), "leaf": 16, "epsilon": epsilon, "steps": rng.randint(3, 12), "dt": dt}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 1000, 1 << 20)}
    if kind == "direct64":
        return {"kind": kind, "n": _log(rng, 10000, 1 << 20), "targets": _log(rng, 500, 8192), "epsilon": epsilon}
    return {"kind": kind, "n": _log(rng, 1000, 65536), "epsilon": epsilon}


# ---- seeded inputs, made on the GPU ----

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=g.device, dtype=torch.float64)


def _directions(g, n):
    z = 2.0 * _rand(g, n) - 1.0
    phi = 2.0 * math.pi * _rand(g, n)
    s = torch.sqrt(1.0 - z * z)
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _accepted(n, sample):
    """n values of a rejection sampler: sample(k) gives the accepted ones of k trials."""
    got = sample(2 * n + 64)
    while len(got) < n:
        got = torch.cat([got, sample(2 * n + 64)])
    return got[:n]


def _pack(pos, mass, vel):
    bodies = torch.zeros(len(pos), 4, dtype=torch.float32, device=pos.device)
    bodies[:, :3] = pos.float()
    bodies[:, 3] = mass.float()
    velocities = torch.zeros_like(bodies)
    velocities[:, :3] = vel.float()
    return bodies, velocities


def _ball(g, n):
    # uniform in the unit ball, masses uniform in [0.5, 1.5] / n, at rest
    pos = _directions(g, n) * _rand(g, n, 1) ** (1.0 / 3.0)
    return _pack(pos, (0.5 + _rand(g, n)) / n, torch.zeros_like(pos))


def _plummer(g, n):
    # scale radius 1, mass 1, truncated at radius 100; speeds q v_esc with density q^2 (1 - q^2)^(7/2)
    x = _rand(g, n) * 0.9998
    r = 1.0 / torch.sqrt(x.clamp_min(1e-12) ** (-2.0 / 3.0) - 1.0)

    def speeds(k):
        q, y = _rand(g, k), 0.1 * _rand(g, k)
        return q[y < q * q * (1.0 - q * q) ** 3.5]

    q = _accepted(n, lambda k: speeds(5 * k))
    vel = (q * math.sqrt(2.0) * (1.0 + r * r) ** -0.25)[:, None] * _directions(g, n)
    pos = r[:, None] * _directions(g, n)
    pos, vel = pos - pos.mean(0), vel - vel.mean(0)
    return _pack(pos, torch.full((n,), 1.0 / n, dtype=torch.float64, device=pos.device), vel)


def _galaxies(g, n):
    # two Hernquist spheres (scale radius 1, mass 1 each) 20 apart, approaching at 0.5; each body
    # moves in a random direction at a fraction of its circular speed
    half = n // 2
    s = torch.sqrt(_rand(g, n) * 0.98)
    r = s / (1.0 - s)
    v = torch.sqrt(r) / (1.0 + r)
    pos, vel = r[:, None] * _directions(g, n), (v * _rand(g, n))[:, None] * _directions(g, n)
    pos[:half, 0] -= 10.0
    pos[half:, 0] += 10.0
    vel[:half, 0] += 0.25
    vel[half:, 0] -= 0.25
    return _pack(pos, torch.full((n,), 2.0 / n, dtype=torch.float64, device=pos.device), vel)


def _bodies(case, seed):
    g = _gen(seed)
    if case["kind"] == "dual":
        return _galaxies(g, case["n"])
    return (_ball if case.get("dist") == "ball" else _plummer)(g, case["n"])


def _codes(pos):
    """63-bit Morton codes of FP32 positions in their bounding cube (x, y, z interleaved)."""
    lo, hi = pos.amin(0), pos.amax(0)
    cell = ((pos - lo) / (hi - lo).amax() * 2097152.0).clamp(0.0, 2097151.0).to(torch.int64)
    code = torch.zeros(len(pos), dtype=torch.int64, device=pos.device)
    for axis in range(3):
        c = cell[:, axis]
        c = (c | c << 32) & 0x1F00000000FFFF
        c = (c | c << 16) & 0x1F0000FF0000FF
        c = (c | c << 8) & 0x100F00F00F00F00F
        c = (c | c << 4) & 0x10C30C30C30C30C3
        c = (c | c << 2) & 0x1249249249249249
        code |= c << (2 - axis)
    return code


def _instances(case):
    """Sizes (log-uniform), thetas (uniform in 0.4 .. 0.7) and step counts of a batch or a request burst."""
    rng = np.random.default_rng(case["mix"])
    sizes = np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["count"]))
    sizes = sizes.round().astype(np.int64)
    thetas = rng.uniform(0.4, 0.7, case["count"]).astype(np.float32)
    steps = rng.integers(max(1, case["steps"] // 2), case["steps"] + 1, case["count"])
    return sizes, thetas, steps


def _spheres(case, seed, sizes):
    # requests are Plummer spheres and uniform balls in turn, batches Plummer spheres
    g = _gen(seed)
    return [(_ball if case["kind"] == "serve" and k % 2 else _plummer)(g, int(n)) for k, n in enumerate(sizes)]


# ---- what a program has in hand ----

_SOLVERS = {"monopole": nb.LinearBVHSolver, "quadrupole": nb.QuadrupoleLinearBVHSolver, "naive": nb.NaiveSolver,
            "dual": nb.OctupoleImplicitLinearBVHFMMSolver}


def _solver(case, bodies=None, velocities=None):
    cls = _SOLVERS["dual" if case["kind"] == "dual" else case.get("solver", "quadrupole")]
    solver = cls(None, nb.Gravity(1.0, case["epsilon"]), theta=case.get("theta", 0.5),
                 max_leaf_size=case.get("leaf", 16), time_step=case.get("dt", 1e-3))
    if bodies is not None:
        torch.cuda.synchronize()
        solver.set_bodies_device(len(bodies), bodies.data_ptr(), velocities.data_ptr())
        solver.synchronize()
    return solver


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("forces", "scenario"):
        bodies, velocities = _bodies(case, seed)
        state.update(solver=_solver(case), bodies=bodies.cpu().numpy(), velocities=velocities.cpu().numpy())
    elif kind in ("step", "dual"):
        bodies, velocities = _bodies(case, seed)
        state.update(solver=_solver(case, bodies, velocities), bodies=bodies, velocities=velocities)
    elif kind == "batch":
        sizes, thetas, _ = _instances(case)
        sets = _spheres(case, seed, sizes)
        bodies, velocities = torch.cat([b for b, _ in sets]), torch.cat([v for _, v in sets])
        solver = _solver(case)
        solver.set_instances(sizes, bodies.cpu().numpy(), velocities.cpu().numpy(), thetas)
        solver.enable_graphs(True)
        solver.step(1)  # the first step is not captured
        state.update(solver=solver, bodies=bodies, velocities=velocities)
    elif kind == "serve":
        sizes, thetas, steps = _instances(case)
        requests = [(b.cpu().numpy(), v.cpu().numpy(), float(t), int(s))
                    for (b, v), t, s in zip(_spheres(case, seed, sizes), thetas, steps)]
        server = nb.Server(nb.Gravity(1.0, case["epsilon"]), order=2, max_leaf_size=case["leaf"], time_step=case["dt"])
        state.update(server=server, requests=requests)
    elif kind == "sort":
        codes = _codes(_plummer(_gen(seed), case["n"])[0][:, :3])
        state.update(codes=codes, sorted=torch.empty_like(codes),
                     ids=torch.empty(case["n"], dtype=torch.int32, device=codes.device))
    elif kind == "direct64":
        bodies, _ = _bodies(case, seed)
        targets = bodies[:: max(1, case["n"] // case["targets"])][: case["targets"]].contiguous()
        state.update(solver=_solver(case), bodies=bodies, targets=targets,
                     acc=torch.empty(len(targets), 3, dtype=torch.float64, device=bodies.device))
    else:
        bodies, velocities = _bodies(case, seed)
        state.update(solver=_solver(case, bodies, velocities))
    return state


def _check(rc):
    if rc != nb.NB_OK:
        raise RuntimeError("status %d" % rc)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forces":
        solver = state["solver"]
        solver.set_bodies(state["bodies"])
        return solver.update_accelerations()
    if kind == "scenario":
        solver = state["solver"]
        solver.set_bodies(state["bodies"], state["velocities"])
        solver.step(case["steps"])
        return solver.bodies()
    if kind in ("step", "dual", "batch"):
        solver, bodies, velocities = state["solver"], state["bodies"], state["velocities"]
        solver.step(case.get("steps", 1))
        _check(nb.lib().nb_get_bodies_device(solver.handle, bodies.data_ptr(), velocities.data_ptr()))
        return bodies, velocities
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(b, v, theta=t, steps=s) for b, v, t, s in state["requests"]]
        done = 0
        while done < len(ids):
            done += server.tick()
        return [server.take_result(i, len(r[0])) for i, r in zip(ids, state["requests"])]
    if kind == "sort":
        _check(nb.lib().nb_sort_codes_noalloc(*(ctypes.cast(t.data_ptr(), ctypes.c_void_p)
                                                for t in (state["codes"], state["sorted"], state["ids"])),
                                              case["n"], None))
        return state["sorted"], state["ids"]
    if kind == "direct64":
        bodies, targets = state["bodies"], state["targets"]
        state["solver"].direct_device(len(bodies), bodies.data_ptr(), len(targets), targets.data_ptr(),
                                      state["acc"].data_ptr(), 64)
        return state["acc"]
    return state["solver"].energy()


# ---- what a pass cannot do without ----

def _tree_flops(n, theta, leaf, order):
    # interactions per body, after the counts of Plummer spheres (225 nodes per tree level and 226
    # pairs per body of leaf capacity at theta 0.5, both as theta^-3), never more than all pairs;
    # 20 flops a pair or monopole term, 56 a quadrupole term
    k = (0.5 / theta) ** 3
    pairs = min(float(n), 226.0 * leaf * k)
    nodes = min(float(n) / leaf, 225.0 * k * max(1.0, math.log2(max(2.0, n / leaf))))
    return n * (20.0 * pairs + (56.0 if order == 2 else 20.0) * nodes)


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("forces", "scenario", "step"):
        steps = case.get("steps", 1)
        if case["solver"] == "naive":
            return {"bytes": 32.0 * n, "flops": 20.0 * n * n}
        flops = steps * _tree_flops(n, case["theta"], case["leaf"], 2 if case["solver"] == "quadrupole" else 1)
        return {"bytes": (32.0 if kind == "forces" else 64.0) * n, "flops": flops}
    if kind == "dual":
        # 1.6e6 flops per body (pairs, M2P, P2L, M2L) in 2^22 bodies at theta 0.4, leaf 64
        per = min(20.0 * n, 1.6e6 * (0.4 / case["theta"]) ** 3 * (case["leaf"] / 64.0) ** 0.5)
        return {"bytes": 64.0 * n, "flops": n * per}
    if kind in ("batch", "serve"):
        # mean size of the log-uniform range; thetas average 0.55, a request's steps 3/4 of the most
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        steps = case["steps"] if kind == "batch" else 0.75 * case["steps"]
        return {"bytes": 64.0 * mean * case["count"],
                "flops": case["count"] * steps * _tree_flops(mean, 0.55, case["leaf"], 2)}
    if kind == "sort":
        return {"bytes": 20.0 * n, "flops": 0.0}
    if kind == "direct64":
        return {"bytes": 16.0 * n + 40.0 * case["targets"], "flops": 20.0 * n * case["targets"]}
    return {"bytes": 32.0 * n, "flops": 14.0 * n * n}


# ---- the same values in FP64, written with torch alone ----

def _direct(bodies, targets, eps, potential=False):
    src, out = bodies.double(), []
    chunk = max(1, (1 << 26) // len(bodies))
    for t in targets.double().split(chunk):
        d = src[None, :, :3] - t[:, None, :3]
        r2 = (d * d).sum(-1)
        same = r2 == 0
        w = src[None, :, 3] * ((r2 + eps) ** (-0.5 if potential else -1.5))
        w = w.masked_fill(same, 0.0)
        out.append(w.sum(1) if potential else (d * w[..., None]).sum(1))
    return torch.cat(out)


def _tree(pos, mass, leaf):
    """Linear BVH over Morton-sorted bodies: ranges, children (-1: leaf), FP32 boxes, per node."""
    code = _codes(pos)
    code, perm = torch.sort(code, stable=True)
    pos, mass = pos[perm], mass[perm]
    dev = pos.device
    b, e = torch.zeros(1, dtype=torch.int64, device=dev), torch.full((1,), len(pos), dtype=torch.int64, device=dev)
    begins, ends, lefts, spans, total = [], [], [], [], 0
    while len(b):
        first, last = code[b], code[e - 1]
        split = (e - b > leaf) & (first != last)
        diff = first ^ last
        for s in (1, 2, 4, 8, 16, 32):
            diff = diff | (diff >> s)
        pivot = last & ~(diff >> 1)
        middle = torch.searchsorted(code, pivot)
        begins.append(b)
        ends.append(e)
        spans.append((total, total + len(b)))
        total += len(b)
        order = torch.cumsum(split.to(torch.int64), 0) - 1
        lefts.append(torch.where(split, total + 2 * order, torch.full_like(order, -1)))
        b, m, e = b[split], middle[split], e[split]
        b, e = torch.stack([b, m], 1).reshape(-1), torch.stack([m, e], 1).reshape(-1)
    begin, end, left = torch.cat(begins), torch.cat(ends), torch.cat(lefts)
    lo = torch.full((total, 3), math.inf, dtype=torch.float32, device=dev)
    hi = -lo
    leaves = torch.nonzero(left < 0).squeeze(1)
    owner = torch.repeat_interleave(leaves, end[leaves] - begin[leaves])
    body = torch.arange(len(owner), device=dev) - torch.repeat_interleave(
        torch.cumsum(end[leaves] - begin[leaves], 0) - end[leaves], end[leaves] - begin[leaves])
    index = owner[:, None].expand(-1, 3)
    lo.scatter_reduce_(0, index, pos[body], "amin")
    hi.scatter_reduce_(0, index, pos[body], "amax")
    for a, z in reversed(spans):
        inner = torch.nonzero(left[a:z] >= 0).squeeze(1) + a
        lo[inner] = torch.minimum(lo[left[inner]], lo[left[inner] + 1])
        hi[inner] = torch.maximum(hi[left[inner]], hi[left[inner] + 1])
    return perm, pos, mass, begin, end, left, lo, hi


def _tree_forces(bodies, theta, leaf, eps, order):
    """The Barnes-Hut sum: approximations decided in FP32 as the criterion states them (squared box
    diagonal over squared distance to the box centre, against theta squared), terms in FP64."""
    perm, pos, mass, begin, end, left, lo, hi = _tree(bodies[:, :3].contiguous(), bodies[:, 3], leaf)
    n, dev = len(pos), pos.device
    p64, m64 = pos.double(), mass.double()
    pairs = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
    second = torch.stack([p64[:, i] * p64[:, j] * m64 for i, j in pairs], 1)
    raw = torch.cat([m64[:, None], p64 * m64[:, None], second], 1)
    sums = torch.cat([torch.zeros(1, 10, dtype=torch.float64, device=dev), torch.cumsum(raw, 0)])
    raw = sums[end] - sums[begin]
    M = raw[:, 0]
    com = raw[:, 1:4] / M[:, None]
    Q = torch.stack([raw[:, 4 + k] - M * com[:, i] * com[:, j] for k, (i, j) in enumerate(pairs)], 1)
    centre = (hi + lo) / 2.0
    side = hi - lo
    diag2 = (side[:, 0] * side[:, 0] + side[:, 1] * side[:, 1]) + side[:, 2] * side[:, 2]
    theta2 = torch.tensor(theta, dtype=torch.float32, device=dev) ** 2
    out = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    for t0 in range(0, n, 16384):
        t = torch.arange(t0, min(n, t0 + 16384), device=dev)
        node = torch.zeros_like(t)
        while len(t):
            keep_t, keep_node = [], []
            for tc, nc in zip(t.split(1 << 23), node.split(1 << 23)):
                d = pos[tc] - centre[nc]
                d2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
                far = diag2[nc] / d2 < theta2
                a, k = tc[far], nc[far]
                R = p64[a] - com[k]
                r2 = (R * R).sum(1)
                inv = (r2 + eps) ** -0.5
                term = -R * (M[k] * inv ** 3)[:, None]
                if order == 2:
                    q = Q[k]
                    x, y, z = R[:, 0], R[:, 1], R[:, 2]
                    QR = torch.stack([q[:, 0] * x + q[:, 1] * y + q[:, 2] * z, q[:, 1] * x + q[:, 3] * y + q[:, 4] * z,
                                      q[:, 2] * x + q[:, 4] * y + q[:, 5] * z], 1)
                    trace = q[:, 0] + q[:, 3] + q[:, 5]
                    term += R * (1.5 * trace * inv ** 5 - 7.5 * (R * QR).sum(1) * inv ** 7)[:, None]
                    term += QR * (3.0 * inv ** 5)[:, None]
                out.index_add_(0, a, term.masked_fill((r2 == 0)[:, None], 0.0))
                a, k = tc[~far], nc[~far]
                inner = left[k] >= 0
                keep_t.append(a[inner].repeat_interleave(2))
                keep_node.append((left[k[inner]][:, None] + torch.arange(2, device=dev)).reshape(-1))
                for al, kl in zip(a[~inner].split(1 << 19), k[~inner].split(1 << 19)):
                    size = end[kl] - begin[kl]
                    who = al.repeat_interleave(size)
                    shift = torch.cumsum(size, 0) - size - begin[kl]
                    body = torch.arange(len(who), device=dev) - shift.repeat_interleave(size)
                    R = p64[who] - p64[body]
                    r2 = (R * R).sum(1)
                    term = -R * (m64[body] * (r2 + eps) ** -1.5)[:, None]
                    out.index_add_(0, who, term.masked_fill((r2 == 0)[:, None], 0.0))
            t, node = torch.cat(keep_t), torch.cat(keep_node)
    forces = torch.empty_like(out)
    forces[perm] = out
    return forces


def _forces(case, bodies, theta):
    if case.get("solver") == "naive":
        return _direct(bodies, bodies, case["epsilon"])
    return _tree_forces(bodies, theta, case["leaf"], case["epsilon"], 1 if case.get("solver") == "monopole" else 2)


def _steps(case, bodies, velocities, theta, steps):
    # FP64 state; each step's decisions and sources are the positions rounded to FP32
    pos, vel, dt = bodies.double(), velocities.double(), float(np.float32(case["dt"]))
    for _ in range(int(steps)):
        vel[:, :3] += _forces(case, pos.float(), theta) * dt
        pos[:, :3] += vel[:, :3] * dt
    return pos, vel


def exact(case, seed):
    kind = case["kind"]
    case = dict(case, epsilon=float(np.float32(case["epsilon"]))) if "epsilon" in case else case
    if kind == "forces":
        bodies, _ = _bodies(case, seed)
        acc = torch.zeros(len(bodies), 4, dtype=torch.float64, device=bodies.device)
        acc[:, :3] = _forces(case, bodies, case["theta"])
        return acc
    if kind in ("scenario", "step"):
        return _steps(case, *_bodies(case, seed), case["theta"], case["steps"])
    if kind == "sort":
        codes = _codes(_plummer(_gen(seed), case["n"])[0][:, :3])
        values, ids = torch.sort(codes, stable=True)
        return values, ids.to(torch.int32)
    if kind == "direct64":
        bodies, _ = _bodies(case, seed)
        targets = bodies[:: max(1, case["n"] // case["targets"])][: case["targets"]]
        return _direct(bodies, targets, case["epsilon"])
    if kind == "energy":
        bodies, velocities = (x.double() for x in _bodies(case, seed))
        kinetic = 0.5 * (bodies[:, 3] * (velocities[:, :3] ** 2).sum(1)).sum()
        potential = -0.5 * (bodies[:, 3] * _direct(bodies, bodies, case["epsilon"], potential=True)).sum()
        return float(kinetic), float(potential)
    if kind in ("batch", "serve") and case["count"] * case["n_max"] < 1 << 20:
        sizes, thetas, steps = _instances(case)
        done = [_steps(case, b, v, float(t), s) for (b, v), t, s in zip(
            _spheres(case, seed, sizes), thetas, [case["steps"] + 1] * len(sizes) if kind == "batch" else steps)]
        if kind == "serve":
            return done
        return torch.cat([p for p, _ in done]), torch.cat([v for _, v in done])
    return None  # the dual tree's field expansions, and batches that would take too long
