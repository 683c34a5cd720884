"""The byte model of the dense phases: a pose batch reads the groups' matrices
once per tile of 32 poses, and a set-up writes the matrices its solves read."""
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu


def make(gpu, w, precision):
    ctx = gpu.ArapContext(w.V, w.faces)
    ctx.set_precision(precision, 1)
    ctx.set_rest_positions(w.positions)
    ctx.set_constraints(w.cidx, w.ctargets)
    return ctx


def test_pose_matrices_per_tile(gpu):
    w = W.cfg_pose_batch(level=4, n_poses=65, iterations=1)
    B = {}
    with make(gpu, w, "mixed") as ctx:
        for n in (31, 32, 33, 64, 65):
            ctx.deform_poses(w.poses[:n], 1)
            B[n], flops = ctx.kernel_model()["solve_fwd"]
            entries = flops / 6 / n
    pose = B[32] - B[31]
    assert pose > 0
    assert B[33] - B[32] == pytest.approx(pose + 4 * entries, rel=1e-12)
    assert B[64] - B[33] == pytest.approx(31 * pose, rel=1e-12)
    assert B[65] - B[64] == pytest.approx(pose + 4 * entries, rel=1e-12)


@pytest.mark.parametrize("precision,size", [("fp64", 8), ("mixed", 4)])
def test_set_up_writes_what_the_solves_read(gpu, precision, size):
    w = W.cfg_icosphere_l4(level=4, iterations=1)
    models = []
    for sweeps in (False, True):
        with make(gpu, w, precision) as ctx:
            if sweeps:
                ctx.set_dense_top(-1)  # the sweeps, without a dense top
            ctx.deform(1)
            models.append(ctx.kernel_model())
    phases, sweeps = models
    entries = [m["solve_fwd"][1] / 6 for m in models]
    assert phases["factor"][0] - sweeps["factor"][0] == pytest.approx(size * (entries[0] - entries[1]), rel=1e-12)
