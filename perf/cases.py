"""Performance cases: the deforms that programs ask of this library, through its
Python binding (which wraps the C entry points one to one).

A case is one call as a user's program makes it, host arrays in and out:

  drag      one frame of interactive handle dragging: the rest pose and the
            handles' new targets are set and the mesh is deformed. As in the
            reference, setting constraints makes the deform dirty: cotan
            weights, Laplacian and Cholesky factor are formed again. The
            constrained set stays the same, so the symbolic analysis is kept.
  repick    the same with the analysis redone on every call, as a program
            does that picks other handles each time.
  repose    new targets for a resident factor, then the vertex normals of the
            deformed mesh, as a viewer's frame needs them.
  poses     many handle poses of one mesh in one call.
  batch     several meshes of uneven sizes in one set of launches.
  inflight  several meshes' dirty deforms in flight at once, a context each.

Meshes: "sphere" (icosphere of level a, radius noise), "bar" (surface of an
a x b x c grid of cells, spacing 1/b, length a/b) and "sheet" (an open
a x b height field with shuffled vertex numbers, as scans have). Precision
"fp64" is the reference's PrecisionType double, "mixed" the FP32 form with
FP64-residual refinement, for programs whose meshes hold single-precision
points (PrecisionType float; OpenMesh's default): they take the positions into
such a mesh.
"""
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = str(Path(__file__).resolve().parent.parent / "mesh-deform_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import arap_gpu  # noqa: E402


def _case(name, call, mesh, a, b=0, c=0, precision="mixed", iterations=10, count=1):
    d = {"call": call, "mesh": mesh, "a": a, "b": b, "c": c, "precision": precision, "iterations": iterations,
         "count": count}
    return dict(d, name=name) if name else d


def listed():
    return [
        # the reference's sphere example: 642 vertices, deform(5) per frame, double
        _case("drag_sphere_l3_fp64", "drag", "sphere", 3, precision="fp64", iterations=5),
        # about the reference's bar example (386 vertices, deform(20) per frame): 380
        _case("drag_bar_30x3x3_fp64", "drag", "bar", 30, 3, 3, precision="fp64", iterations=20),
        # a small character part: 2,562 vertices in double
        _case("drag_sphere_l4_fp64", "drag", "sphere", 4, precision="fp64", iterations=10),
        # an open scanned patch of odd size (7,979 vertices), interactive
        _case("drag_sheet_101x79_mixed", "drag", "sheet", 101, 79, iterations=15),
        # the twisted bar (67,202 vertices): the benchmark's mesh and iterations
        _case("drag_bar_400x40x40_mixed", "drag", "bar", 400, 40, 40, iterations=30),
        _case("drag_bar_400x40x40_fp64", "drag", "bar", 400, 40, 40, precision="fp64", iterations=30),
        # the same with other handles on every call
        _case("repick_bar_400x40x40_mixed", "repick", "bar", 400, 40, 40, iterations=30),
        # the largest interactive mesh: 163,842 vertices, 50 iterations
        _case("drag_sphere_l7_mixed", "drag", "sphere", 7, iterations=50),
        # a viewer's frame on a resident factor: 40,962 vertices
        _case("repose_sphere_l6_mixed", "repose", "sphere", 6, iterations=10),
        # the pose sweep: 256 poses of 10,242 vertices
        _case("poses_256_sphere_l5", "poses", "sphere", 5, iterations=20, count=256),
        # 16 meshes of uneven sizes at once
        _case("batch_16_bars", "batch", "bar", 60, 8, 8, iterations=30, count=16),
        # 8 independent requests in flight (16,802 vertices each)
        _case("inflight_8_bars_200x20x20", "inflight", "bar", 200, 20, 20, iterations=30, count=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_mesh(rng, vmax):
    kind = rng.choice(["sphere", "bar", "bar", "sheet", "sheet"])
    if kind == "sphere":
        top = max(k for k in range(3, 8) if 10 * 4 ** k + 2 <= vmax)
        return kind, rng.randint(3, top), 0, 0
    v = _log_int(rng, 400, vmax)
    if kind == "bar":
        ratio = rng.uniform(4.0, 12.0)  # length over width
        b = max(2, int(math.sqrt(v / (4.0 * ratio))))
        return kind, max(8, int(ratio * b)), b, max(2, int(b * rng.uniform(0.7, 1.0)))
    ratio = rng.uniform(0.5, 2.0)
    a = max(12, int(math.sqrt(v * ratio)))
    return kind, a, max(12, int(v / a)), 0


def draw(rng):
    call = rng.choice(["drag", "drag", "drag", "repick", "repose", "repose", "poses", "poses", "batch", "inflight"])
    precision = rng.choice(["fp64", "mixed"])
    iterations = rng.randint(5, 30)
    if call in ("drag", "repick", "repose"):
        return _case(None, call, *_draw_mesh(rng, 64000), precision=precision, iterations=iterations)
    if call == "poses":
        m = _draw_mesh(rng, 10300)
        return _case(None, call, *m, iterations=min(iterations, 20), count=_log_int(rng, 3, 256))
    if call == "batch":
        m = _draw_mesh(rng, 1500)
        return _case(None, call, *m, precision=precision, iterations=iterations, count=rng.randint(2, 16))
    m = _draw_mesh(rng, 12000)
    return _case(None, call, *m, precision=precision, iterations=iterations, count=rng.randint(2, 8))


# ---------------------------------------------------------------------------
# meshes


def _outward(p, f, centre):
    n = np.cross(p[f[:, 1]] - p[f[:, 0]], p[f[:, 2]] - p[f[:, 0]])
    flip = (n * (p[f].mean(1) - centre)).sum(1) < 0
    f = f.copy()
    f[flip] = f[flip][:, [0, 2, 1]]
    return f


@functools.lru_cache(maxsize=None)
def _sphere(level):
    t = (1.0 + math.sqrt(5.0)) / 2.0
    v = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                  (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)], np.float64)
    f = np.array([(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
                  (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11),
                  (6, 2, 10), (8, 6, 7), (9, 8, 1)], np.int64)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    for _ in range(level):
        e = np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]])
        e.sort(axis=1)
        key, inv = np.unique(e[:, 0] * len(v) + e[:, 1], return_inverse=True)
        inv = inv.reshape(-1)
        mid = v[key // len(v)] + v[key % len(v)]
        a, b, c = (len(v) + inv[k * len(f):(k + 1) * len(f)] for k in range(3))
        v = np.concatenate([v, mid / np.linalg.norm(mid, axis=1, keepdims=True)])
        f = np.concatenate([np.stack(q, 1) for q in ((f[:, 0], a, c), (f[:, 1], b, a), (f[:, 2], c, b), (a, b, c))])
    return v, f.astype(np.int32)


@functools.lru_cache(maxsize=None)
def _bar(nx, ny, nz):
    g = np.stack(np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), np.arange(nz + 1), indexing="ij"), -1)
    n = np.array([nx, ny, nz])
    on = ((g == 0) | (g == n)).any(-1)
    ids = np.full(on.shape, -1, np.int64)
    ids[on] = np.arange(int(on.sum()))
    quads = []
    for ax in range(3):
        for end in (0, n[ax]):
            side = np.take(ids, end, axis=ax)
            quads.append(np.stack([side[:-1, :-1], side[1:, :-1], side[1:, 1:], side[:-1, 1:]], -1).reshape(-1, 4))
    q = np.concatenate(quads)
    f = np.concatenate([q[:, [0, 1, 2]], q[:, [0, 2, 3]]])
    p = g[on] / float(ny)
    return p, _outward(p, f, n / (2.0 * ny)).astype(np.int32)


@functools.lru_cache(maxsize=None)
def _sheet(nx, ny):
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij"), -1).reshape(-1, 2)
    ids = np.random.RandomState(nx * 1009 + ny).permutation(nx * ny).reshape(nx, ny)
    q = np.stack([ids[:-1, :-1], ids[1:, :-1], ids[1:, 1:], ids[:-1, 1:]], -1).reshape(-1, 4)
    f = np.concatenate([q[:, [0, 1, 2]], q[:, [0, 2, 3]]])
    p = np.zeros((nx * ny, 3))
    xy = g / float(max(nx, ny) - 1)
    p[ids.reshape(-1), :2] = xy
    p[ids.reshape(-1), 2] = 0.08 * np.sin(7.0 * xy[:, 0]) * np.cos(5.0 * xy[:, 1])
    return p, f.astype(np.int32)


def _turn(rng, most):
    axis = rng.normal(size=3)
    x, y, z = axis / np.linalg.norm(axis)
    t = rng.uniform(0.3, 1.0) * most
    k = np.array([[0, -z, y], [z, 0, -x], [-y, x, 0]])
    return np.eye(3) + math.sin(t) * k + (1.0 - math.cos(t)) * k @ k


def _problem(mesh, a, b, c, seed, poses=1):
    """Rest positions, faces, constrained indices and poses x n x 3 targets: an
    anchored region stays, a handle region is turned and shifted per pose."""
    rng = np.random.default_rng(seed)
    if mesh == "sphere":
        p, f = _sphere(a)
        p = p * (1.0 + rng.normal(0.0, 0.004, (len(p), 1)))
        anchor, handle, span = p[:, 2] < -0.8, p[:, 2] > 0.8, 1.0
    elif mesh == "bar":
        p, f = _bar(a, b, c)
        x = np.rint(p[:, 0] * b)
        p = p + rng.normal(0.0, 0.02 / b, p.shape)
        ring = max(1, round(0.2 * b))
        anchor, handle, span = x < ring, x > a - ring, 1.0
    else:
        p, f = _sheet(a, b)
        h = 1.0 / (max(a, b) - 1)
        x, y = np.rint(p[:, 0] / h), np.rint(p[:, 1] / h)
        p = p + rng.normal(0.0, 0.05 * h, p.shape)
        ring = max(1, min(a, b) // 16)
        anchor = (x < ring) | (x > a - 1 - ring)
        handle = (abs(x - a // 2) <= max(1, a // 12)) & (abs(y - b // 2) <= max(1, b // 12))
        span = 0.4
    idx = np.nonzero(anchor | handle)[0].astype(np.int32)
    h = handle[idx]
    t = np.repeat(p[None, idx], poses, 0)
    mid = p[handle].mean(0)
    for k in range(poses):
        t[k, h] = (p[idx[h]] - mid) @ _turn(rng, math.pi / 3).T + mid + span * rng.uniform(-0.4, 0.4, 3)
    return p, f, idx, t


def _problems(case, seed):
    """One (rest, faces, indices, targets) per mesh of the case."""
    m, n = (case["mesh"], case["a"], case["b"], case["c"]), case["count"]
    if case["call"] == "poses":
        return [_problem(*m, seed, n)]
    if case["call"] == "batch":  # uneven sizes: each mesh up to four times as fine as the smallest
        out = []
        for k in range(n):
            s = 1.0 + (k % 4)
            mk = m if m[0] == "sphere" else (m[0], int(m[1] * s), int(m[2] * s), int(m[3] * s))
            if m[0] == "sphere":
                mk = (m[0], max(2, m[1] - k % 3), 0, 0)
            out.append(_problem(*mk, seed * 1000 + k))
        return out
    return [_problem(*m, seed * 1000 + k) for k in range(n if case["call"] == "inflight" else 1)]


# ---------------------------------------------------------------------------
# the calls


def prepare(case, seed):
    probs = _problems(case, seed)
    s = {"call": case["call"], "iterations": case["iterations"], "rest": [p[0] for p in probs],
         "idx": [p[2] for p in probs], "targets": [p[3][0] for p in probs], "poses": probs[0][3]}
    if case["precision"] == "mixed":  # the program's own vertex arrays, in single precision
        shapes = [(len(s["poses"]),) + p[0].shape if s["call"] == "poses" else p[0].shape for p in probs]
        s["mesh"] = [torch.empty(q, dtype=torch.float32) for q in shapes]
        s["normals"] = torch.empty(shapes[0], dtype=torch.float32)
    if s["call"] == "batch":
        mb = arap_gpu.MeshBatch([(len(p), f) for p, f, _, _ in probs])
        mb.ctx.set_precision(case["precision"])
        mb.set_rest_positions(s["rest"])
        mb.set_constraints(s["idx"], s["targets"])
        s["batch"] = mb
        return s
    s["ctx"] = []
    for p, f, idx, t in probs:
        ctx = arap_gpu.ArapContext(len(p), f)
        ctx.set_precision(case["precision"])
        if s["call"] == "repick":
            ctx.set_symbolic_cache(False)
        if s["call"] == "inflight":
            ctx.set_solve_ctas(64)
        ctx.set_rest_positions(p)
        ctx.set_constraints(idx, t[0])
        if s["call"] in ("repose", "poses"):
            ctx.deform(0, want_output=False)  # the factor stays resident
        s["ctx"].append(ctx)
    if s["call"] == "inflight":  # results arrive in pinned memory while other requests run
        s["out"] = [torch.empty(p.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
                    for p in s["rest"]]
    return s


def _store(s, out):
    """The positions in the program's own vertex arrays."""
    if "mesh" not in s:
        return out
    for mesh, x in zip(s["mesh"], out):
        mesh.copy_(torch.from_numpy(x))
    return s["mesh"]


def run(s):
    call, it = s["call"], s["iterations"]
    if call in ("drag", "repick"):
        ctx = s["ctx"][0]
        ctx.set_rest_positions(s["rest"][0])
        ctx.set_constraints(s["idx"][0], s["targets"][0])
        return _store(s, [ctx.deform(it)])
    if call == "repose":
        ctx = s["ctx"][0]
        ctx.set_targets(s["targets"][0])
        out, normals = _store(s, [ctx.deform(it)])[0], ctx.vertex_normals()
        if "mesh" in s:
            normals = s["normals"].copy_(torch.from_numpy(normals))
        return [out, normals]
    if call == "poses":
        return _store(s, [s["ctx"][0].deform_poses(s["poses"], it)])
    if call == "batch":
        mb = s["batch"]
        mb.set_rest_positions(s["rest"])
        mb.set_constraints(s["idx"], s["targets"])
        return _store(s, mb.deform(it))
    for ctx, rest, idx, t, out in zip(s["ctx"], s["rest"], s["idx"], s["targets"], s["out"]):
        ctx.set_rest_positions(rest)
        ctx.set_constraints(idx, t)
        ctx.deform_async(it, out)
    for ctx in s["ctx"]:
        ctx.wait()
    return _store(s, s["out"])


def work(case):
    """Bytes: rest poses, faces and targets read once, positions (and normals)
    written once, and the factor's entries written once where it is formed
    (read once where it is resident). Flops: per iteration and vertex about 7
    neighbours x (18 covariance + 30 right-hand side) and 200 for the rotation,
    the two triangular solves with 3 columns (4 nnz(L) x 3), and the
    factorisation; nnz(L) and its flops as planar nested dissection gives them
    (7.75 n log2 n and 9.9 n^1.5, George 1973)."""
    nbytes = flops = 0.0
    for p, f, idx, t in _problems(dict(case, count=min(case["count"], 4) if case["call"] != "batch" else case["count"]), 1):
        v, m = len(p), len(p) - len(idx)
        poses = case["count"] if case["call"] == "poses" else 1
        nnz = 7.75 * m * math.log2(max(m, 2)) / 4.0  # a dissection's constant in practice: a quarter of the bound
        size = 8 if case["precision"] == "fp64" else 4
        nbytes += 24.0 * v + 4.0 * f.size + poses * (24.0 * len(idx) + 3.0 * size * v) + size * nnz
        flops += poses * case["iterations"] * (v * (7 * 48 + 200.0) + 12.0 * nnz)
        if case["call"] == "repose":
            nbytes += 3.0 * size * v
        elif case["call"] != "poses":
            flops += 9.9 * m ** 1.5
    if case["call"] == "inflight":
        k = case["count"] / min(case["count"], 4)
        nbytes, flops = nbytes * k, flops * k
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch alone: ARAP by its definition, the global
# step by a dense Cholesky factor or, for many unknowns, conjugate gradients


def _weights(p, f):
    """Clamped cotan weights: (i, j, w) of every directed edge, per face."""
    v = [p[f[:, k]] for k in range(3)]
    sq = [((v[(k + 1) % 3] - v[k]) ** 2).sum(-1).clamp_min(1e-8) for k in range(3)]
    ln = [s.sqrt() for s in sq]
    sp = 0.5 * (ln[0] + ln[1] + ln[2])
    heron = (sp * (sp - ln[0]) * (sp - ln[1]) * (sp - ln[2])).clamp_min(0.0)
    area = heron.sqrt().clamp_min(1e-8)
    i, j, w = [], [], []
    for k in range(3):
        cot = ((sq[0] + sq[1] + sq[2] - 2.0 * sq[k]) / (4.0 * area)).clamp_min(1e-10)
        a, b = f[:, k], f[:, (k + 1) % 3]
        i += [a, b]
        j += [b, a]
        w += [0.5 * cot, 0.5 * cot]
    return torch.cat(i), torch.cat(j), torch.cat(w)


def _rotations(S):
    """R maximising tr(R S) for S of shape (n, 3, 3): one-sided Jacobi SVD."""
    S = S / S.flatten(1).norm(dim=1).clamp_min(1e-300)[:, None, None]
    b = [S[:, :, k] for k in range(3)]
    one = torch.eye(3, dtype=S.dtype, device=S.device)
    v = [one[k].expand(len(S), 3) for k in range(3)]
    for _ in range(12):
        for x, y in ((0, 1), (0, 2), (1, 2)):
            al, be, ga = ((b[x] * b[x]).sum(1), (b[y] * b[y]).sum(1), (b[x] * b[y]).sum(1))
            small = ga.abs() <= 1e-17 * (al * be).sqrt()
            z = (be - al) / (2.0 * torch.where(small, torch.ones_like(ga), ga))
            t = torch.where(z < 0, -1.0, 1.0) / (z.abs() + torch.hypot(torch.ones_like(z), z))
            t = torch.where(small, torch.zeros_like(t), t)
            cs = 1.0 / torch.hypot(torch.ones_like(t), t)
            sn = (cs * t)[:, None]
            cs = cs[:, None]
            b[x], b[y] = cs * b[x] - sn * b[y], sn * b[x] + cs * b[y]
            v[x], v[y] = cs * v[x] - sn * v[y], sn * v[x] + cs * v[y]
    order = torch.stack([q.norm(dim=1) for q in b], 1).argsort(1, descending=True)[:, :2]
    B, W = torch.stack(b, 1), torch.stack(v, 1)
    pick = lambda M, k: M.gather(1, order[:, k, None, None].expand(-1, 1, 3))[:, 0]  # noqa: E731
    u1 = pick(B, 0)
    u1 = u1 / u1.norm(dim=1, keepdim=True).clamp_min(1e-300)
    u2 = pick(B, 1)
    u2 = u2 - (u1 * u2).sum(1, keepdim=True) * u1
    u2 = u2 / u2.norm(dim=1, keepdim=True).clamp_min(1e-300)
    v1, v2 = pick(W, 0), pick(W, 1)
    u3, v3 = torch.linalg.cross(u1, u2), torch.linalg.cross(v1, v2)
    return v1[:, :, None] * u1[:, None, :] + v2[:, :, None] * u2[:, None, :] + v3[:, :, None] * u3[:, None, :]


class _Dense:
    def __init__(self, n, i, j, w, d):
        A = torch.zeros(n, n, dtype=torch.float64, device=d.device)
        A.index_put_((i, j), -w, accumulate=True)
        A.diagonal().add_(d)
        self.c = torch.linalg.cholesky(A)

    def solve(self, b, x):
        return torch.cholesky_solve(b, self.c)


class _Cg:
    def __init__(self, n, i, j, w, d):
        k = torch.arange(n, device=d.device)
        A = torch.sparse_coo_tensor(torch.stack([torch.cat([i, k]), torch.cat([j, k])]), torch.cat([-w, d]), (n, n))
        self.A, self.m = A.coalesce().to_sparse_csr(), (1.0 / d)[:, None]

    def solve(self, b, x):
        r = b - self.A @ x
        z = self.m * r
        p, rz, top = z, (r * z).sum(0), (b * self.m * b).sum(0)
        for k in range(20000):
            if k % 64 == 0 and bool((rz <= 1e-28 * top).all()):
                break
            q = self.A @ p
            al = rz / (p * q).sum(0).clamp_min(1e-300)
            x = x + al * p
            r = r - al * q
            z = self.m * r
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        return x


def _normals(p, f):
    unit = lambda q: q / q.norm(dim=1, keepdim=True).clamp_min(1e-300)  # noqa: E731
    n = unit(torch.linalg.cross(p[f[:, 1]] - p[f[:, 0]], p[f[:, 2]] - p[f[:, 0]]))
    out = torch.zeros_like(p)
    for k in range(3):
        out.index_add_(0, f[:, k], n)
    return unit(out)


def _arap(rest, f, idx, targets, iterations):
    """Positions (poses, V, 3) after the iterations from the rest pose."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rest, f = torch.tensor(rest, device=dev), torch.tensor(f, device=dev).long()
    idx, targets = torch.tensor(idx, device=dev).long(), torch.tensor(targets, device=dev)
    V, P = len(rest), len(targets)
    i, j, w = _weights(rest, f)
    e = rest[i] - rest[j]
    diag = torch.zeros(V, dtype=torch.float64, device=dev).index_add_(0, i, w)
    free = torch.ones(V, dtype=torch.bool, device=dev)
    free[idx] = False
    at = torch.cumsum(free, 0) - 1
    n = int(free.sum())
    ff, fc = free[i] & free[j], free[i] & ~free[j]
    solver = (_Dense if n <= 12000 else _Cg)(n, at[i[ff]], at[j[ff]], w[ff], diag[free])
    x = rest[:, None].repeat(1, P, 1)
    x[idx] = targets.transpose(0, 1)
    bfix = torch.zeros(V, P, 3, dtype=torch.float64, device=dev)
    bfix.index_add_(0, i[fc], w[fc, None, None] * x[j[fc]])
    we = w[:, None] * e
    for _ in range(iterations):
        R = torch.empty(V, P, 3, 3, dtype=torch.float64, device=dev)
        step = max(1, 2000000 // V)
        for k in range(0, P, step):
            d = x[i, k:k + step] - x[j, k:k + step]
            S = torch.zeros(V, d.shape[1], 3, 3, dtype=torch.float64, device=dev)
            S.index_add_(0, i, we[:, None, :, None] * d[:, :, None, :])
            R[:, k:k + step] = _rotations(S.reshape(-1, 3, 3)).reshape(S.shape)
        b = bfix.clone()
        for k in range(0, P, step):
            Re = 0.5 * torch.einsum("epab,eb->epa", R[i, k:k + step] + R[j, k:k + step], we)
            b[:, k:k + step].index_add_(0, i, Re)
        x[free] = solver.solve(b[free].reshape(n, -1), x[free].reshape(n, -1)).reshape(n, P, 3)
    return x.transpose(0, 1), f


def exact(case, seed):
    out = []
    for p, f, idx, t in _problems(case, seed):
        x, ft = _arap(p, f, idx, t, case["iterations"])
        out.append((x if case["call"] == "poses" else x[0]).cpu().numpy())
        if case["call"] == "repose":
            out.append(_normals(x[0], ft).cpu().numpy())
    return out
