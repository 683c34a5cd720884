"""Launch shapes that only large or densely coupled meshes reach: per-vertex
blocks of 128 and 256 threads, and the tiled top products of an FP64 plan."""
import numpy as np
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu


def make(gpu, V, p, faces, cidx, targets, precision):
    ctx = gpu.ArapContext(V, faces)
    ctx.set_precision(precision, 1)
    ctx.set_rest_positions(p)
    ctx.set_constraints(cidx, targets)
    return ctx


@pytest.mark.parametrize("name,threads", [("bar", 128), ("sphere", 256)])
def test_large_vertex_blocks(gpu, name, threads):
    """105,002 and 163,842 vertices: automatic blocks of 128 and 256 give the bits
    of blocks of 64 and of two launches for the RHS and the first residual."""
    w = W.cfg_twisted_bar(h=0.02, iterations=2) if name == "bar" else W.cfg_noisy_sphere(level=7, iterations=2)
    # the rule: the most threads that leave a block to each of 608 schedulers
    assert threads * 608 <= w.V and (threads == 256 or w.V < 2 * threads * 608)
    with make(gpu, w.V, w.positions, w.faces, w.cidx, w.ctargets, "mixed") as ctx:
        a = ctx.deform(w.iterations)
        for k in ("local", "rhs", "residual"):
            ctx.set_vertex_launch(k, 1, 64)
        ctx.invalidate()
        np.testing.assert_array_equal(ctx.deform(w.iterations), a)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-6)])
def test_tiled_top_of_random_triangles(gpu, precision, tol):
    """2,600 vertices in random triangles: the last group has 1,720 columns, in
    FP64 too. One iteration of the phases against the sweeps, which solve the
    same right-hand side: the form's tolerance."""
    rng = np.random.default_rng(0)
    n = 2600
    faces = np.array([rng.choice(n, 3, replace=False) for _ in range(3 * n)], np.int32)
    p = rng.normal(size=(n, 3))
    cidx = np.arange(5, dtype=np.int32)
    out = []
    for sweeps in (False, True):
        with make(gpu, n, p, faces, cidx, p[:5] + 0.3, precision) as ctx:
            if sweeps:
                ctx.set_dense_top(-1)
            out.append(ctx.deform(1))
    assert W.bbox_rel_error(out[0], out[1], p) <= tol
