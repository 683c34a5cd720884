"""A target that is not a number, infinite or beyond FP32 in one pose of a
batch: that pose's free vertices come out non-finite, and the other poses keep
their bits."""
import numpy as np
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e300])
def test_non_finite_target_of_one_pose(gpu, value):
    w = W.cfg_icosphere_l4(level=3, iterations=3)
    poses = np.stack([w.ctargets, w.ctargets + 0.05, w.ctargets - 0.1])
    bad = poses.copy()
    bad[1, 3, 1] = value
    free = np.setdiff1d(np.arange(w.V), w.cidx)
    with gpu.ArapContext(w.V, w.faces) as ctx:
        ctx.set_precision("mixed", 1)
        ctx.set_rest_positions(w.positions)
        ctx.set_constraints(w.cidx, w.ctargets)
        clean = ctx.deform_poses(poses, w.iterations)
        got = ctx.deform_poses(bad, w.iterations)
    np.testing.assert_array_equal(got[0], clean[0])
    np.testing.assert_array_equal(got[2], clean[2])
    assert not np.isfinite(got[1][free]).all(axis=1).any()
