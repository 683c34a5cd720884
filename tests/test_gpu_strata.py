"""The dense-phase solves (the default of a single request) against the
supernodal sweeps and the oracle: sizes at the edges of the plan (one group,
several phases, a last group large enough for the tiled top products), any CTA
cap bit for bit, and both kinds of solve arrays used in turn on one context.

Tolerances: both paths solve the same factored system; their sums differ in
order, so FP64 positions agree to a few thousand roundings (1e-11 of the
bounding box, as between the sweeps' own variants) and mixed ones to the mixed
form's 1e-6."""
import numpy as np
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    "sphere1": lambda: W.cfg_icosphere_l4(level=1, iterations=4),
    "sphere3": lambda: W.cfg_icosphere_l4(level=3, iterations=5),
    "sphere4": lambda: W.cfg_icosphere_l4(level=4, iterations=5),
    "noisy5": lambda: W.cfg_noisy_sphere(level=5, iterations=4),
    "bar.1": lambda: W.cfg_twisted_bar(h=0.1, iterations=4),
    "bar.05": lambda: W.cfg_twisted_bar(h=0.05, iterations=4),
}


def make(gpu, w, precision):
    ctx = gpu.ArapContext(w.V, w.faces)
    ctx.set_precision(precision, 1)
    ctx.set_rest_positions(w.positions)
    ctx.set_constraints(w.cidx, w.ctargets)
    return ctx


@pytest.mark.parametrize("precision,tol,otol", [("fp64", 1e-11, 1e-10), ("mixed", 1e-6, 1e-6)])
@pytest.mark.parametrize("name", CASES)
def test_phases_match_sweeps_and_oracle(gpu, name, precision, tol, otol):
    from oracle import oracle as O

    w = CASES[name]()
    ok, ref = O.run_deform(w.positions, w.faces, w.cidx, w.ctargets, w.iterations)
    assert ok
    with make(gpu, w, precision) as ctx:
        ctx.set_dense_top(-1)  # asks for the sweeps
        sweeps = ctx.deform(w.iterations)
    outs = []
    for cap in (0, 3, 64):
        with make(gpu, w, precision) as ctx:
            ctx.set_solve_ctas(cap)
            a = ctx.deform(w.iterations)
            ctx.invalidate()
            np.testing.assert_array_equal(ctx.deform(w.iterations), a)
            outs.append(a)
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])
    assert W.bbox_rel_error(outs[0], sweeps, w.positions) <= tol
    assert W.bbox_rel_error(outs[0], ref, w.positions) <= otol


def test_poses_and_deforms_in_turn(gpu):
    """A pose batch and a deform have plans of their own, whose arrays are each
    formed from the resident factor when its call comes; both give what a
    context that ran nothing else gives."""
    w = W.cfg_pose_batch(level=4, n_poses=5, iterations=4)
    with make(gpu, w, "mixed") as ctx:
        lone = ctx.deform(w.iterations)
        ctx.set_targets(w.ctargets + 0.05)
        lone2 = ctx.deform(w.iterations)
    with make(gpu, w, "mixed") as ctx:
        poses = ctx.deform_poses(w.poses, w.iterations)
    with make(gpu, w, "mixed") as ctx:
        ctx.set_targets(w.ctargets)
        np.testing.assert_array_equal(ctx.deform(w.iterations), lone)
        np.testing.assert_array_equal(ctx.deform_poses(w.poses, w.iterations), poses)
        ctx.set_targets(w.ctargets + 0.05)
        np.testing.assert_array_equal(ctx.deform(w.iterations), lone2)
        ctx.invalidate()
        np.testing.assert_array_equal(ctx.deform_poses(w.poses, w.iterations), poses)
        ctx.set_targets(w.ctargets + 0.05)
        np.testing.assert_array_equal(ctx.deform(w.iterations), lone2)


@pytest.mark.parametrize("n_poses", [1, 7, 33])
def test_pose_phases_overlap(gpu, n_poses):
    """Phases whose launches overlap give the bits of launches that do not (a
    CTA cap turns the overlap off)."""
    w = W.cfg_pose_batch(level=4, n_poses=n_poses, iterations=4)
    outs = []
    for cap in (0, 64):
        with make(gpu, w, "mixed") as ctx:
            ctx.set_solve_ctas(cap)
            outs.append(ctx.deform_poses(w.poses, w.iterations))
    np.testing.assert_array_equal(outs[1], outs[0])


def test_several_large_roots(gpu):
    """Disjoint meshes: the last phase holds one group per mesh."""
    from oracle import oracle as O

    ws = [W.cfg_twisted_bar(h=0.1, iterations=3), W.cfg_noisy_sphere(level=4, iterations=3)]
    with gpu.MeshBatch([(w.V, w.faces) for w in ws]) as mb:
        mb.ctx.set_precision("fp64")
        mb.set_rest_positions([w.positions for w in ws])
        mb.set_constraints([w.cidx for w in ws], [w.ctargets for w in ws])
        out = mb.deform(3)
    for w, x in zip(ws, out):
        ok, ref = O.run_deform(w.positions, w.faces, w.cidx, w.ctargets, 3)
        assert ok and W.bbox_rel_error(x, ref, w.positions) <= 1e-10


@pytest.mark.parametrize("level", [0, 3, 5, 6])
def test_vertex_blocks_by_size(gpu, level):
    """Per-vertex kernels' blocks chosen by the mesh's size (12, 642, 10,242 and
    40,962 vertices: blocks of 32 and 128), with the RHS and the first residual
    in one launch, give the bits of blocks of 256 and of two launches."""
    w = W.cfg_noisy_sphere(level=level, iterations=3) if level else W.cfg_icosphere_l4(level=0, iterations=3)
    with make(gpu, w, "mixed") as ctx:
        a = ctx.deform(w.iterations)
    with make(gpu, w, "mixed") as ctx:
        for k in ("local", "rhs", "residual"):
            ctx.set_vertex_launch(k, 1, 256)
        np.testing.assert_array_equal(ctx.deform(w.iterations), a)

@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-6)])
@pytest.mark.parametrize("pull", [0.02, 0.3, 1.0])
def test_rotation_seeds(gpu, precision, tol, pull):
    """Local steps from the rotations before: a small move (every fit ends in
    the Newton steps), a large one and one that stretches the one-rings at the
    handles to near rank one (refinement, Jacobi fits), against the oracle's
    SVD; one deform of n iterations gives the bits of n deforms of one."""
    from oracle import oracle as O

    w = W.cfg_icosphere_l4(level=3, iterations=6)
    targets = w.ctargets + pull * np.array([0.3, 1.0, -0.2]) * (np.arange(len(w.cidx)) % 2)[:, None]
    ok, ref = O.run_deform(w.positions, w.faces, w.cidx, targets, w.iterations)
    assert ok
    outs = []
    for parts in ([6], [1, 1, 1, 3]):
        with make(gpu, w, precision) as ctx:
            ctx.set_constraints(w.cidx, targets)
            for n in parts:
                out = ctx.deform(n)
            outs.append(out)
    np.testing.assert_array_equal(outs[1], outs[0])
    assert W.bbox_rel_error(outs[0], ref, w.positions) <= tol
    with make(gpu, w, "mixed") as ctx:
        poses = np.stack([targets, w.ctargets])
        got = ctx.deform_poses(poses, w.iterations)
    assert W.bbox_rel_error(got[0], ref, w.positions) <= 1e-6


@pytest.mark.parametrize("level", [0, 5, 6])
def test_fp64_lanes_by_size(gpu, level):
    """FP64 local steps with four lanes per vertex (12 and 10,242 vertices) and
    with one (40,962), against the oracle."""
    from oracle import oracle as O

    w = W.cfg_noisy_sphere(level=level, iterations=3) if level else W.cfg_icosphere_l4(level=0, iterations=3)
    ok, ref = O.run_deform(w.positions, w.faces, w.cidx, w.ctargets, w.iterations)
    assert ok
    with make(gpu, w, "fp64") as ctx:
        assert W.bbox_rel_error(ctx.deform(w.iterations), ref, w.positions) <= 1e-10
