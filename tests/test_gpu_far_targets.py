"""Covariances that FP32 does not carry.

Handles dragged 1e2 to 1e6 mesh sizes away: in the first iterations the
covariances of the one-rings beside them are that close to rank one, and their
rotations still have to be the oracle's. They turn rest edges, so an error
shows at the rest mesh's scale, and the forms keep their bounds of its bounding
box (mixed 1e-6; FP64 1e-10 times the distance over 1e2, the positions' own
rounding)."""
import numpy as np
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pull", [1e2, 1e4, 1e5, 1e6])
def test_rotations_near_rank_one(gpu, pull):
    from oracle import oracle as O

    w = W.cfg_icosphere_l4(level=3, iterations=6)
    targets = w.ctargets + pull * np.array([0.3, 1.0, -0.2]) * (np.arange(len(w.cidx)) % 2)[:, None]
    ok, ref = O.run_deform(w.positions, w.faces, w.cidx, targets, w.iterations)
    assert ok
    for precision, tol in (("fp64", 1e-10 * pull / 1e2), ("mixed", 1e-6)):
        with gpu.ArapContext(w.V, w.faces) as ctx:
            ctx.set_precision(precision, 1)
            ctx.set_rest_positions(w.positions)
            ctx.set_constraints(w.cidx, targets)
            assert W.bbox_rel_error(ctx.deform(w.iterations), ref, w.positions) <= tol
    with gpu.ArapContext(w.V, w.faces) as ctx:
        ctx.set_precision("mixed", 1)
        ctx.set_rest_positions(w.positions)
        ctx.set_constraints(w.cidx, targets)
        got = ctx.deform_poses(np.stack([w.ctargets, targets]), w.iterations)
    assert W.bbox_rel_error(got[1], ref, w.positions) <= 1e-6


@pytest.mark.parametrize("exponent", [-40, -70, -90])
def test_tiny_meshes(gpu, exponent):
    """Coordinates whose FP32 covariances underflow: a pose batch turns the
    one-rings as the FP64 covariances say."""
    from oracle import oracle as O

    w = W.cfg_icosphere_l4(level=3, iterations=4)
    p, t = w.positions * 2.0 ** exponent, w.ctargets * 2.0 ** exponent
    ok, ref = O.run_deform(p, w.faces, w.cidx, t, w.iterations)
    assert ok
    with gpu.ArapContext(w.V, w.faces) as ctx:
        ctx.set_precision("mixed", 1)
        ctx.set_rest_positions(p)
        ctx.set_constraints(w.cidx, t)
        single = ctx.deform(w.iterations)
        poses = ctx.deform_poses(np.stack([t, p[w.cidx]]), w.iterations)
    assert W.bbox_rel_error(poses[0], ref, p) <= 1e-6
    assert W.bbox_rel_error(single, ref, p) <= 1e-6


def test_huge_coordinates(gpu):
    """Coordinates beyond FP32's range, whose differences are inside it."""
    from oracle import oracle as O

    w = W.cfg_icosphere_l4(level=3, iterations=4)
    p, t = w.positions * 2.0 ** 120 + 2.0 ** 130, w.ctargets * 2.0 ** 120 + 2.0 ** 130
    ok, ref = O.run_deform(p, w.faces, w.cidx, t, w.iterations)
    assert ok
    with gpu.ArapContext(w.V, w.faces) as ctx:
        ctx.set_precision("mixed", 1)
        ctx.set_rest_positions(p)
        ctx.set_constraints(w.cidx, t)
        got = ctx.deform_poses(t[None], w.iterations)[0]
    assert W.bbox_rel_error(got, ref, p) <= 1e-6
