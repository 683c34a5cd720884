"""arap_plan_bytes names what the next call will hold, and asking changes
nothing: neither the bits nor the launches of the calls that follow."""
import ctypes as C

import numpy as np
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu


def plan_bytes(ctx, n_poses):
    v = C.c_int64()
    ctx._check(ctx.lib.arap_plan_bytes(ctx.h, n_poses, C.byref(v)))
    return v.value


def make(gpu, w, precision):
    ctx = gpu.ArapContext(w.V, w.faces)
    ctx.set_precision(precision, 1)
    ctx.set_rest_positions(w.positions)
    ctx.set_constraints(w.cidx, w.ctargets)
    return ctx


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_asking_keeps_the_resident_plan(gpu, precision):
    w = W.cfg_icosphere_l4(level=4, iterations=3)
    runs = []
    for ask in (False, True):
        with make(gpu, w, precision) as ctx:
            ctx.deform(w.iterations)
            ctx.set_targets(w.ctargets + 0.05)
            if ask:
                plan_bytes(ctx, 4)
                plan_bytes(ctx, 0)
            out = ctx.deform(w.iterations)
            runs.append((ctx.launch_count(), ctx.device_bytes(), out))
    assert runs[1][:2] == runs[0][:2]
    np.testing.assert_array_equal(runs[1][2], runs[0][2])


@pytest.mark.parametrize("precision,n_poses,after_deform", [("fp64", 0, False), ("mixed", 0, False), ("mixed", 5, False),
                                                            ("mixed", 33, True)])
@pytest.mark.parametrize("level", [3, 5])
def test_planned_is_what_is_held(gpu, precision, n_poses, after_deform, level):
    w = W.cfg_pose_batch(level=level, n_poses=max(n_poses, 1), iterations=2)
    with make(gpu, w, precision) as ctx:
        if after_deform:
            ctx.deform(1)
        planned = plan_bytes(ctx, n_poses)
        if n_poses:
            ctx.deform_poses(w.poses, w.iterations)
        else:
            ctx.deform(w.iterations)
        assert ctx.device_bytes() == planned
