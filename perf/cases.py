"""Performance cases of naga_b200, each one call sequence a user's program makes.

kind "scene"       one acoustic scene (naga.Scene): the initial pulse, a run of
                   time steps, then the probe traces and the solution (density
                   and velocity of every node; on the small scenes also the
                   populations). The framework's main path.
kind "batch"       many ragged scenes stepped together (naga.Batch).
kind "create"      a request of the serving loop: build the scene from its
                   point cloud, run its first steps, read it, release it.
kind "knn"         exact nearest neighbours of many clouds (naga.knn_clouds).
kind "divergence"  the standalone divergence operator: build the stencil of a
                   point cloud, apply it to a vector field.
kind "interp"      radial point interpolation: neighbours, weights, field.
kind "inverse"     batched inverse of the RBF moment matrices, FP64 or FP32
                   factors with FP64 refinement.

exact() restates each in 64-bit torch: brute-force neighbours, torch.linalg for
the small systems and sparse matrix products for the step.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import naga_b200 as naga

PROBES = {2: [[0.3, 0.5], [0.7, 0.5], [0.5, 0.3], [0.5, 0.7]],
          3: [[x, y, z] for z in (0.35, 0.65) for y in (0.35, 0.65) for x in (0.35, 0.65)]}
K_OF = {2: 16, 3: 32}      # stencil size of the 2-D and 3-D scenes
SHAPE_OF = {2: 1, 3: 0}    # r^3 in 2-D, the multiquadric in 3-D
Q_OF = {2: 9, 3: 27}


def listed() -> list[dict]:
    return [
        # the smallest 2-D scene of the batched workload, run alone: ten
        # kernels a step over a few thousand nodes, bound by launch latency.
        # A run ends within three sides of travel at half a spacing a step:
        # past that the layer has absorbed the pulse and the solution is the
        # rounding of what is left
        dict(name="scene2d_2k", kind="scene", dim=2, n_side=45, steps=135, state=True),
        # the plain 2-D scene: 20,164 nodes, 500 steps
        dict(name="scene2d_20k", kind="scene", dim=2, n_side=142, steps=500, state=True),
        # the batched 2-D workload: ragged scenes of 2k to 100k nodes
        dict(name="batch2d_32", kind="batch", dim=2, scenes=32, lo=2000, hi=100000, sizes=100, steps=100),
        # the smallest 3-D request of the serving loop
        dict(name="scene3d_10k", kind="scene", dim=3, n_side=22, steps=66, state=True),
        # the plain 3-D scene: 250,047 nodes
        dict(name="scene3d_250k", kind="scene", dim=3, n_side=63, steps=200, state=False),
        # the largest 3-D request of the serving loop
        dict(name="scene3d_1m", kind="scene", dim=3, n_side=100, steps=60, state=False),
        # a served 3-D request from its point cloud to its first results
        dict(name="create3d_100k", kind="create", dim=3, n_side=47, steps=10),
        # the set-up microbenchmark: 64 clouds of 5k to 200k points, k = 32
        dict(name="knn_64_clouds", kind="knn", dim=3, clouds=64, lo=5000, hi=200000, sizes=2, k=32),
        # the divergence operator of the plain 3-D cloud, and one field
        dict(name="divergence3d_250k", kind="divergence", dim=3, n_side=63, k=32),
        # interpolation of a velocity field to scattered receivers
        dict(name="interp3d_50k", kind="interp", dim=3, n_side=63, queries=50000, k=32, fields=3),
        # 36 x 36 moment matrices of random stencils, r^3, FP64
        dict(name="inverse_f64_36", kind="inverse", n=36, batch=200000, refined=False),
        # the moment matrices of jittered-grid stencils, refined FP32
        dict(name="inverse_f32r_36", kind="inverse", n=36, batch=20000, refined=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["scene2", "scene2", "scene3", "scene3", "batch", "create", "knn", "divergence", "interp",
                       "inverse"])
    if kind == "scene2":
        n = _log_int(rng, 45, 316)
        return dict(kind="scene", dim=2, n_side=n, steps=rng.randint(60, min(500, 3 * n)), state=n < 150)
    if kind == "scene3":
        n = _log_int(rng, 16, 100)
        return dict(kind="scene", dim=3, n_side=n, steps=max(20, min(200, 3 * n, 50_000_000 // n ** 3)),
                    state=n < 30)
    if kind == "batch":
        return dict(kind="batch", dim=2, scenes=rng.randint(3, 32), lo=2000, hi=100000, sizes=rng.randint(0, 9999),
                    steps=rng.randint(20, 100))
    if kind == "create":
        return dict(kind="create", dim=3, n_side=_log_int(rng, 16, 47), steps=rng.randint(3, 10))
    if kind == "knn":
        dim = rng.choice([2, 3])
        return dict(kind="knn", dim=dim, clouds=rng.randint(1, 64), lo=5000, hi=_log_int(rng, 8000, 200000),
                    sizes=rng.randint(0, 9999), k=rng.choice([K_OF[dim], K_OF[dim], 24, 40]))
    if kind == "divergence":
        dim = rng.choice([2, 3])
        n = _log_int(rng, 45, 316) if dim == 2 else _log_int(rng, 16, 63)
        return dict(kind="divergence", dim=dim, n_side=n, k=rng.choice([K_OF[dim], K_OF[dim], 24]))
    if kind == "interp":
        dim = rng.choice([2, 3])
        n = _log_int(rng, 45, 316) if dim == 2 else _log_int(rng, 16, 63)
        return dict(kind="interp", dim=dim, n_side=n, queries=_log_int(rng, 500, 50000),
                    k=rng.choice([K_OF[dim], K_OF[dim], 24]), fields=rng.choice([1, dim]))
    refined = rng.choice([False, True])
    n = rng.choice([19, 20, 24, 35, 36, 36, 45])
    return dict(kind="inverse", n=n, batch=_log_int(rng, 1000, 20000 if refined else 150000), refined=refined)


# ------------------------------------------------------------------ inputs
def _layers(dim, n_side):
    return min(10, n_side // 4) if dim == 2 else max(2, n_side // 8)


def _grid(case, seed):
    return naga.generate_grid(case["dim"], case["n_side"], _layers(case["dim"], case["n_side"]), seed)


def _pulse(points, dim, rng):
    return naga.gaussian_pulse(points, list(rng.uniform(0.35, 0.65, dim)), 1e-3, float(rng.uniform(0.04, 0.08)))


def _scene_args(dim):
    return dict(k=K_OF[dim], shape=SHAPE_OF[dim], probes=np.array(PROBES[dim], np.float32), probe_capacity=1024)


def _ragged(case):
    """The sizes of a ragged set, log-uniform, fixed by the case."""
    r = np.random.default_rng(case["sizes"])
    m = case["scenes"] if case["kind"] == "batch" else case["clouds"]
    return np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), m)).astype(np.int64)


def _batch_sides(case):
    return [max(45, int(round(math.sqrt(n)))) for n in _ragged(case)]


def _moment_matrices(case, seed):
    """Augmented moment matrices [[Phi, P], [P^T, 0]] of k + 1 + d rows over
    random 3-D stencils (2-D for n = 19): the k points nearest the origin of
    a random cloud scaled to the unit box, r^3 (FP64 case), or of a jittered
    grid, multiquadric (refined case)."""
    n, m = case["n"], case["batch"]
    d = 2 if n == 19 else 3
    k = n - d - 1
    gen = torch.Generator(device="cuda").manual_seed(seed)
    A = torch.zeros((m, n, n), dtype=torch.float64, device="cuda")
    for a in range(0, m, 50000):
        b = min(m, a + 50000)
        if case["refined"]:
            ax = torch.arange(-3, 4, device="cuda", dtype=torch.float64)
            base = torch.cartesian_prod(*([ax] * d))
            jit = torch.rand((b - a, base.shape[0], d), generator=gen, device="cuda", dtype=torch.float64)
            pts = base + (jit - 0.5) * 0.5
        else:
            pts = torch.rand((b - a, 2 * k, d), generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
        near = pts.square().sum(2).topk(k, largest=False).indices
        X = torch.gather(pts, 1, near[:, :, None].expand(-1, -1, d))
        X = X - X[:, :1]
        if not case["refined"]:
            X = X / X.abs().amax(dim=(1, 2), keepdim=True)
        r2 = (X[:, :, None] - X[:, None]).square().sum(3)
        A[a:b, :k, :k] = (r2 + 0.01).sqrt() if case["refined"] else r2 * r2.sqrt()
        A[a:b, :k, k] = 1.0
        A[a:b, k, :k] = 1.0
        A[a:b, :k, k + 1:] = X
        A[a:b, k + 1:, :k] = X.transpose(1, 2)
    return A


def _interp_inputs(case, seed):
    g = _grid(case, seed)
    r = np.random.default_rng(seed)
    dim = case["dim"]
    src = torch.from_numpy(g["points"]).cuda()
    qry = torch.from_numpy(r.uniform(0.05, 0.95, (case["queries"], dim)).astype(np.float32)).cuda()
    return src, qry, _field(src, case["fields"], r), float(g["h"])


def _field(pts, comps, r):
    """Smooth fields of a point cloud: sums of plane waves, FP32 [n][comps]."""
    dim = pts.shape[1]
    wave = torch.from_numpy(r.uniform(1.0, 8.0, (comps, 4, dim))).cuda()
    ph = torch.from_numpy(r.uniform(0.0, 6.28, (comps, 4))).cuda()
    return torch.sin(torch.einsum("nd,cwd->ncw", pts.double(), wave) + ph).sum(2).float().contiguous()


def _knn_points(case, seed):
    off = np.concatenate([[0], np.cumsum(_ragged(case))]).astype(np.int64)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((int(off[-1]), case["dim"]), generator=gen, device="cuda"), off


def prepare(case: dict, seed: int):
    kind, r = case["kind"], np.random.default_rng(seed)
    if kind == "scene":
        g = _grid(case, seed)
        s = naga.Scene(g, **_scene_args(case["dim"]))
        return dict(case=case, scene=s, drho=_pulse(g["points"], case["dim"], r))
    if kind == "batch":
        b, drho = naga.Batch(case["dim"]), []
        for t, n in enumerate(_batch_sides(case)):
            g = _grid(dict(dim=case["dim"], n_side=n), seed * 1000 + t)
            b.add(naga.Scene(g, **_scene_args(case["dim"])))
            drho.append(_pulse(g["points"], case["dim"], r))
        b.prepare()
        return dict(case=case, batch=b, drho=drho)
    if kind == "create":
        g = _grid(case, seed)
        return dict(case=case, grid=g, drho=_pulse(g["points"], case["dim"], r))
    if kind == "knn":
        pts, off = _knn_points(case, seed)
        return dict(case=case, pts=pts, off=off)
    if kind == "divergence":
        pts = torch.from_numpy(_grid(case, seed)["points"]).cuda()
        return dict(case=case, pts=pts, field=_field(pts, case["dim"], r))
    if kind == "interp":
        src, qry, field, h = _interp_inputs(case, seed)
        return dict(case=case, src=src, qry=qry, field=field, h=h)
    return dict(case=case, A=_moment_matrices(case, seed))


# --------------------------------------------------------------------- run
def _solution(scene, steps):
    density, velocity = scene.macros()
    return dict(probes=scene.probes(0, steps), density=density, velocity=velocity)


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "scene":
        s = state["scene"]
        s.set_initial_condition(state["drho"])
        s.step(case["steps"])
        out = _solution(s, case["steps"])
        if case["state"]:
            out["populations"] = s.state()[0]
        return out
    if kind == "batch":
        b = state["batch"]
        for s, drho in zip(b.scenes, state["drho"]):
            s.set_initial_condition(drho)
        b.step(case["steps"])
        each = [_solution(s, case["steps"]) for s in b.scenes]
        return {n: np.concatenate([e[n] for e in each]) for n in each[0]}
    if kind == "create":
        s = naga.Scene(state["grid"], **_scene_args(case["dim"]))
        s.set_initial_condition(state["drho"])
        s.step(case["steps"])
        out = _solution(s, case["steps"])
        s.close()
        return out
    if kind == "knn":
        idx, d2 = naga.knn_clouds(state["pts"], state["off"], case["k"])
        return dict(idx=idx, d2=d2)
    if kind == "divergence":
        idx, W, delta = naga.divergence_build_f32(state["pts"], case["k"], SHAPE_OF[case["dim"]])
        return dict(idx=idx, W=W, delta=delta, div=naga.divergence_apply(W, idx, state["field"]))
    if kind == "interp":
        idx, _ = naga.knn(state["src"], state["qry"], case["k"])
        w = naga.rbf_weights_f32(state["src"], idx, state["qry"], 1, state["h"], SHAPE_OF[case["dim"]])
        return dict(idx=idx, weights=w, values=naga.rbf_interpolate(w, idx, state["field"]))
    inverse = naga.batched_inverse_f32r if case["refined"] else naga.batched_inverse_f64
    inv, info = inverse(state["A"])
    return dict(inverse=inv, info=info)


# -------------------------------------------------------------------- work
def _step_work(dim, nodes):
    """One step of `nodes` nodes: the populations, the PML integrals and the
    macros read and written once; the stencil (weights, filter weight, index)
    read once. Five weighted sums over the stencil and the collision."""
    k, q = K_OF[dim], Q_OF[dim]
    return nodes * (4 * q * 4 + 32 + k * 4 * (dim + 2)), nodes * (5 * 2 * k * q + 40 * q)


def _stencil_flops(dim, k):
    """One RPIM system: assembly, LU of the augmented matrix, solves."""
    n = k + dim + 1
    return 2 * n ** 3 / 3 + 2 * dim * n * n + 6 * k * k


def work(case: dict) -> dict:
    kind, dim = case["kind"], case.get("dim", 3)
    if kind in ("scene", "create"):
        nodes = case["n_side"] ** dim
        b, f = _step_work(dim, nodes)
        b, f = b * case["steps"], f * case["steps"]
        if kind == "create":
            b += nodes * (4 * dim + K_OF[dim] * 4 * (dim + 2))
            f += nodes * _stencil_flops(dim, K_OF[dim])
        return dict(bytes=b, flops=f)
    if kind == "batch":
        b, f = _step_work(dim, sum(n ** dim for n in _batch_sides(case)))
        return dict(bytes=b * case["steps"], flops=f * case["steps"])
    if kind == "knn":
        n = int(_ragged(case).sum())
        return dict(bytes=n * (4 * dim + 8 * case["k"]), flops=n * 3 * dim * 4 * case["k"])
    if kind == "divergence":
        n, k = case["n_side"] ** dim, case["k"]
        return dict(bytes=n * (8 * dim + 4 * k * (dim + 1) + 8),
                    flops=n * (_stencil_flops(dim, k) + (16 if dim == 2 else 64) * k * (3 * dim + 4)))
    if kind == "interp":
        n, q, k = case["n_side"] ** dim, case["queries"], case["k"]
        return dict(bytes=n * 4 * (dim + case["fields"]) + q * (4 * dim + 8 * k + 4 * case["fields"]),
                    flops=q * (_stencil_flops(dim, k) + 2 * k * case["fields"]))
    n, m = case["n"], case["batch"]
    return dict(bytes=m * (16 * n * n + 4), flops=2 * m * n ** 3)


def tolerance(case: dict):
    # about four times the largest error against exact() over the ranges:
    # FP32 populations over a run of steps 2.4e-6 (velocity), a dozen steps
    # 1.7e-7; FP32 distances, weights and sums 2.5e-8 to 5.1e-7; the inverses
    # of r^3 systems in FP64 5e-12 to 1.5e-10 (a rare close pair of points
    # dominates), of the multiquadric systems refined to the FP64 residual
    # 3e-15
    if case["kind"] == "inverse":
        return {"rel": 2e-14, "max": 2e-13} if case["refined"] else {"rel": 1e-9, "max": 4e-9}
    return {"scene": {"rel": 1e-5}, "batch": {"rel": 1e-5}, "create": {"rel": 1e-6}, "knn": {"rel": 1e-7},
            "divergence": {"rel": 2e-6}, "interp": {"rel": 1e-6}}[case["kind"]]


# ------------------------------------------------- exact: 64-bit restatement
def _exact_knn(src, qry, k):
    """The k sources smallest under (squared distance, index), the distance
    rounded as FP32 with the highest dimension added last."""
    n = src.shape[0]
    rows = max(1, min(4096, 200_000_000 // n))
    out = []
    for a in range(0, qry.shape[0], rows):
        q = qry[a:a + rows]
        d2 = None
        for d in range(src.shape[1]):
            t = (q[:, d, None] - src[None, :, d]).square_()
            d2 = t if d2 is None else t.add_(d2)
        m = min(n, k + 8)
        v, i = d2.topk(m, dim=1, largest=False)
        key = (v.view(torch.int32).long() << 32) | i
        out.append(key.sort(dim=1).values[:, :k] & 0xFFFFFFFF)
    return torch.cat(out)


def _phi(r2, shape):
    return (r2 + 0.01).sqrt() if shape == 0 else r2 * r2.sqrt()


def _moment(xs, shape):
    m, k, d = xs.shape
    G = torch.zeros((m, k + d + 1, k + d + 1), dtype=torch.float64, device=xs.device)
    G[:, :k, :k] = _phi((xs[:, :, None] - xs[:, None]).square().sum(3), shape)
    G[:, :k, k] = G[:, k, :k] = 1.0
    G[:, :k, k + 1:] = xs
    G[:, k + 1:, :k] = xs.transpose(1, 2)
    return G


def _right_side(xs, x, shape):
    """[phi(|x - x_s|); 1; x] of points x [m][p][d]: [m][p][k + d + 1]."""
    phi = _phi((xs[:, None] - x[:, :, None]).square().sum(3), shape)
    return torch.cat([phi, torch.ones_like(x[:, :, :1]), x], dim=2)


def _exact_rpim(src, idx, qry, h, shape):
    out = []
    for a in range(0, qry.shape[0], 16384):
        q = qry[a:a + 16384].double()
        xs = (src[idx[a:a + 16384]].double() - q[:, None]) / h
        rhs = _right_side(xs, torch.zeros_like(q)[:, None], shape).transpose(1, 2)
        out.append(torch.linalg.solve(_moment(xs, shape), rhs)[:, :idx.shape[1], 0])
    return torch.cat(out)


@functools.lru_cache(None)
def _quadrature(dim):
    """Unit offsets u_q and a_d(u_q) w_q of the nonlocal divergence at
    interaction radius 1: Gauss-Legendre radii (six-digit values), the
    antisymmetric B-spline kernel."""
    gw = [0.652145, 0.652145, 0.347855, 0.347855]
    gx = [0.339981, -0.339981, 0.861136, -0.861136]
    us, ks = [], []
    for p in range(4 if dim == 3 else 1):
        for t in range(4):
            for w, x in zip(gw, gx):
                r, th, ph = (x + 1.0) / 2.0, t * math.pi / 2, p * math.pi / 4 + math.pi / 8
                s = [round(math.cos(th)), round(math.sin(th))]
                u = [r * s[0], r * s[1]] if dim == 2 else [r * math.sin(ph) * s[0], r * math.sin(ph) * s[1],
                                                          r * math.cos(ph)]
                c = 240.0 / 7.0 if dim == 2 else 48.0
                m = c * r * (2.0 - 3.0 * r) if 2.0 * r < 1 else c * (1.0 - r) ** 2
                wq = w / 2.0 * (math.pi / 2)
                wq *= r if dim == 2 else math.pi / 4 * r * math.hypot(u[0], u[1])
                us.append(u)
                ks.append([m * v / r / math.pi * wq for v in u])
    return np.array(us), np.array(ks)


def _exact_stencil(pts, k, shape):
    """Neighbours, divergence weights [n][k][d] and interaction radii."""
    n, dim = pts.shape
    idx = _exact_knn(pts, pts, k)
    P = pts.double()
    nn = (P - P[idx[:, 1]]).square().sum(1).sqrt()
    spacing = torch.cat([c.mean().expand(c.shape[0]) for c in nn.split(16384)])
    u, K = (torch.from_numpy(t).cuda() for t in _quadrature(dim))
    delta, W = 0.05 * nn, []
    for a in range(0, n, 8192):
        s = slice(a, min(n, a + 8192))
        xs = (P[idx[s]] - P[s][:, None]) / spacing[s][:, None, None]
        xq = (delta[s] / spacing[s])[:, None, None] * u
        Kq = K / delta[s][:, None, None]
        b = _right_side(xs, xq, shape).transpose(1, 2) @ Kq
        w = torch.linalg.solve(_moment(xs, shape), b)[:, :k]
        w[:, 0] += Kq.sum(1)
        W.append(w)
    return idx, torch.cat(W), delta


def _lattice(dim):
    """Directions, weights and opposites in the framework's order."""
    if dim == 2:
        c = [(0, 0), (-1, 1), (-1, 0), (-1, -1), (0, -1), (1, -1), (1, 0), (1, 1), (0, 1)]
        w = {0: 4 / 9, 1: 1 / 9, 2: 1 / 36}
    else:
        c = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
        for z, y in (("x", "y"), ("x", "z"), ("y", "z")):
            i, j = "xyz".index(z), "xyz".index(y)
            order = [(1, 1), (-1, 1), (1, -1), (-1, -1)]
            for a, b in order:
                v = [0, 0, 0]
                v[i], v[j] = a, b
                c.append(tuple(v))
        c += [(x, y, z) for z in (1, -1) for y in (1, -1) for x in (1, -1)]
        w = {0: 8 / 27, 1: 2 / 27, 2: 1 / 54, 3: 1 / 216}
    weights = [w[sum(abs(v) for v in t)] for t in c]
    opposite = [c.index(tuple(-v for v in t)) for t in c]
    return (torch.tensor(c, dtype=torch.float64, device="cuda"), torch.tensor(weights, dtype=torch.float64, device="cuda"),
            opposite)


def _moments27(c):
    """The orthogonal moment basis of D3Q27: [27][27], column j = moment j."""
    x, y, z = c.T
    x2, y2, z2 = x * x, y * y, z * z
    s2, s4 = x2 + y2 + z2, x2 * y2 + x2 * z2 + y2 * z2
    cols = [x * 0 + 1, x, y, z, x * y, x * z, y * z, x2 - y2, x2 + y2 - 2 * z2, s2 - 2,
            x * (3 * (y2 + z2) - 4), y * (3 * (x2 + z2) - 4), z * (3 * (x2 + y2) - 4),
            x * (y2 - z2), y * (x2 - z2), z * (x2 - y2), x * y * z, 3 * s4 - 4 * s2 + 4,
            3 * (x2 * y2 + x2 * z2 - 2 * y2 * z2) - 2 * (2 * x2 - y2 - z2), 3 * (x2 * y2 - x2 * z2) - 2 * (y2 - z2),
            y * z * (3 * x2 - 2), x * z * (3 * y2 - 2), x * y * (3 * z2 - 2),
            x * (9 * y2 * z2 - 6 * (y2 + z2) + 4), y * (9 * x2 * z2 - 6 * (x2 + z2) + 4),
            z * (9 * x2 * y2 - 6 * (x2 + y2) + 4), 27 * x2 * y2 * z2 - 18 * s4 + 12 * s2 - 8]
    return torch.stack(cols, 1)


class _Collision3:
    """Relaxation of every moment above the momentum towards the equilibrium
    with factorised central moments (1, u, 1/3 + u^2 per axis)."""

    def __init__(self, c, w, nu, dt):
        self.c, self.w, self.B = c, w, _moments27(c)
        rates = ([0.0] * 4 + [1 / (3 * nu + 0.5)] * 6 + [1.5] * 3 + [1.83] * 3 + [1.4, 1.61] + [1.98] * 5 + [1.74] * 4)
        self.scale = torch.tensor(rates, dtype=torch.float64, device="cuda") / self.B.square().sum(0)

    def __call__(self, g, drho, u):
        eq = 1.0 + drho[:, None]
        for d in range(3):
            second = 1 / 3 + u[:, d, None] ** 2
            cd = self.c[:, d]
            eq = eq * torch.where(cd == 0, 1 - second, 0.5 * (second + cd * u[:, d, None]))
        return -(((g + self.w - eq) @ self.B) * self.scale) @ self.B.T


class _Collision2:
    """The cascaded D2Q9 collision, moments 3 .. 8."""

    def __init__(self, c, w, nu, dt):
        self.w, self.dt, self.om = w, dt, 1 / (3 * nu + 0.5 * dt)
        x, y = c.T
        x2, y2 = x * x, y * y
        self.K = torch.stack([3 * (x2 + y2) - 4, x2 - y2, -x * y, -y * (3 * x2 - 2), -x * (3 * y2 - 2),
                              9 * x2 * y2 - 6 * (x2 + y2) + 4], 1)

    def __call__(self, g, drho, u):
        R, NW, W, SW, S, SE, E, NE, N = (g + self.w).unbind(1)
        rho, (a, b) = 1 + drho, u.unbind(1)
        i = 1 / self.dt
        k3 = i * (rho * (a * a + b * b) - E - N - S - W - 2 * (SE + SW + NE + NW - rho / 3)) / 12
        k4 = self.om * (N + S - E - W + rho * (a * a - b * b)) / 4
        k5 = self.om * (NE + SW - NW - SE + rho * a * b) / 4
        k6 = (-i * ((SE + SW - NE - NW - 2 * a * a * b * rho + b * (rho - N - S - R)) / 4 + a / 2 * (NE - NW - SE + SW))
              - b / 2 * (-3 * k3 - k4) - 2 * a * k5)
        k7 = (-i * ((SW + NW - SE - NE - 2 * a * b * b * rho + a * (rho - W - E - R)) / 4 + b / 2 * (NE + SW - SE - NW))
              - a / 2 * (-3 * k3 + k4) - 2 * b * k5)
        t = (rho / 9 - NE - NW - SE - SW + 2 * (a * (NE - NW + SE - SW) + b * (NE + NW - SE - SW))
             + 4 * a * b * (NW - NE + SE - SW) - a * a * (N + NE + NW + S + SE + SW)
             + b * b * (3 * a * a * rho - E - NE - NW - SE - SW - W))
        k8 = (i * t / 4 - 2 * k3 - 2 * a * k7 - 2 * b * k6 + 4 * a * b * k5
              - (1.5 * k3 - k4 / 2) * (a * a + b * b))
        return self.dt * torch.stack([k3, k4, k5, k6, k7, k8], 1) @ self.K.T


def _csr(rows, idx, w, n):
    """The [rows][n] sparse matrix with w [m][k] at (row of w, idx)."""
    m, k = idx.shape
    ptr = torch.arange(rows + 1, device="cuda").clamp(max=m) * k
    return torch.sparse_csr_tensor(ptr, idx.reshape(-1), w.reshape(-1), (rows, n), dtype=torch.float64)


def _exact_scene(grid, drho, dim, steps, state):
    k, shape, h = K_OF[dim], SHAPE_OF[dim], grid["h"]
    pts = torch.from_numpy(grid["points"]).cuda()
    n, nb, nl, nbd = pts.shape[0], grid["n_bulk"], grid["n_layer"], grid["n_boundary"]
    nbl = nb + nl
    sigma = torch.from_numpy(grid["sigma"]).cuda().double()[:, None]
    normals = torch.from_numpy(grid["normals"]).cuda().double()
    c, w, opposite = _lattice(dim)
    idx, W, _ = _exact_stencil(pts, k, shape)
    D = [_csr(n, idx, W[:, :, d].contiguous(), n) for d in range(dim)]
    r2 = (pts[idx].double() - pts[:, None].double()).square().sum(2)
    fw = torch.exp(-0.5 * r2 / (h / 2.5) ** 2)[:nbl]
    filt = _csr(nbl, idx[:nbl], fw / fw.sum(1, keepdim=True), n)
    bidx = _exact_knn(pts[:nbl], pts[nbl:], k)
    wall = _csr(nbd, bidx, _exact_rpim(pts, bidx, pts[nbl:], h, shape), n)
    probes = torch.tensor(PROBES[dim], dtype=torch.float32, device="cuda")
    pidx = _exact_knn(pts, probes, k)
    pw = _exact_rpim(pts, pidx, probes, h, shape)
    del W, r2, fw, idx
    cs = 1 / math.sqrt(3.0)
    dt = 0.5 * h / cs
    collide = (_Collision2 if dim == 2 else _Collision3)(c, w, 1e-5 / cs, dt)
    facing = [c[a] @ normals.T > 0 for a in range(len(opposite))]

    def divergence(v):
        out = (D[0] @ v) * c[:, 0]
        for d in range(1, dim):
            out += (D[d] @ v) * c[:, d]
        return out

    g = torch.from_numpy(drho).cuda().double()[:, None] * w
    old, q1_old = torch.zeros_like(g), torch.zeros_like(g)
    shift, trace = nb, []
    layer, solid = slice(nb, nbl), slice(nbl, nbl + nbd)
    for _ in range(steps):
        dr = g.sum(1)
        u = (g @ c) / (1 + dr)[:, None]
        trace.append((pw * dr[pidx]).sum(1))
        uc = u @ c.T
        new = w * (dr[:, None] + (1 + dr)[:, None] * (3 * uc + 4.5 * uc * uc - u.square().sum(1)[:, None]))
        q1 = (new + old) * (dt / 2)
        q2 = (q1 + q1_old) * (dt / 2)
        s = g.clone()
        s[layer] -= sigma * (3 * new[layer] + 3 * sigma * q1[layer] + sigma ** 2 * q2[layer])
        f = torch.zeros_like(g)
        f[layer] = (-2 * sigma * (q1[nb - shift:nbl - shift] - q1[layer].mean(0))
                    + sigma ** 2 * (q2[nb - shift:nbl - shift] - q2[layer].mean(0)))
        s += divergence(f)
        s[solid] = wall @ s
        s += collide(g, dr, u)
        old, q1_old = new, q1
        g = s
        g[:nbl] += 0.75 * (filt @ s - s[:nbl])
        b = g[solid].clone()
        for a, o in enumerate(opposite):
            g[solid, a] = torch.where(facing[a], b[:, o], b[:, a])
        v = g
        for fac in (dt / 4, dt / 3, dt / 2, dt):
            rate = divergence(v)
            rate[nbl:] = 0
            v = g - fac * rate
        g = v
        g[solid] = wall @ g
    velocity = u / cs
    velocity[solid] = 0
    out = dict(probes=torch.stack(trace), density=1 + dr, velocity=velocity)
    if state:
        out["populations"] = g
    return out


def exact(case: dict, seed: int):
    kind, r = case["kind"], np.random.default_rng(seed)
    if kind in ("scene", "create"):
        nodes = case["n_side"] ** case["dim"]
        # past this the restatement takes over about 20 s
        if nodes * case["steps"] * Q_OF[case["dim"]] * K_OF[case["dim"]] > 5e10 or nodes > 400_000:
            return None
        g = _grid(case, seed)
        return _exact_scene(g, _pulse(g["points"], case["dim"], r), case["dim"], case["steps"], case.get("state"))
    if kind == "batch":
        sides = _batch_sides(case)
        if len(sides) * case["steps"] > 3200:
            return None
        each = []
        for t, n in enumerate(sides):
            g = _grid(dict(dim=case["dim"], n_side=n), seed * 1000 + t)
            each.append(_exact_scene(g, _pulse(g["points"], case["dim"], r), case["dim"], case["steps"], False))
        return {n: torch.cat([e[n] for e in each]) for n in each[0]}
    if kind == "knn":
        if float((_ragged(case).astype(float) ** 2).sum()) > 1.5e11:
            return None
        pts, off = _knn_points(case, seed)
        idx, d2 = [], []
        for a, b in zip(off[:-1], off[1:]):
            p = pts[a:b]
            idx.append(_exact_knn(p, p, case["k"]))
            P = p.double()
            d2.append((P[idx[-1]] - P[:, None]).square().sum(2))
        return dict(idx=torch.cat(idx).int(), d2=torch.cat(d2))
    if kind == "divergence":
        pts = torch.from_numpy(_grid(case, seed)["points"]).cuda()
        field = _field(pts, case["dim"], r).double()
        idx, W, delta = _exact_stencil(pts, case["k"], SHAPE_OF[case["dim"]])
        return dict(idx=idx.int(), W=W, delta=delta, div=(W * field[idx]).sum((1, 2)))
    if kind == "interp":
        src, qry, field, h = _interp_inputs(case, seed)
        idx = _exact_knn(src, qry, case["k"])
        w = _exact_rpim(src, idx, qry, float(np.float32(h)), SHAPE_OF[case["dim"]])
        values = torch.einsum("qk,qkc->qc", w, field.double()[idx])
        return dict(idx=idx.int(), weights=w, values=values)
    A = _moment_matrices(case, seed)
    inv = torch.cat([torch.linalg.inv(a) for a in A.split(20000)])
    return dict(inverse=inv, info=torch.zeros(A.shape[0], dtype=torch.int32, device="cuda"))
