"""A ribbon all of whose triangles are collinear: its cotan weights are the
squared edges over the clamped area, alike for every edge and above 1.8e19 from
edges of 2^20 on, where the product of two of them leaves FP32's range. The
system is as well conditioned as that of unit weights, and the FP32 factor
solves it as the FP64 one does."""
import numpy as np
import pytest

import arap_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 40])
@pytest.mark.parametrize("exponent", [0, 20, 24, 27])
@pytest.mark.parametrize("bits", [64, 32])
def test_collinear_ribbon(gpu, n, exponent, bits):
    from oracle import oracle as O

    edge = 2.0 ** exponent
    p = np.zeros((2 * n, 3))
    p[:n, 0] = np.arange(n) * edge
    p[n:, 0] = (np.arange(n) + 0.5) * edge
    faces = np.array([t for i in range(n - 1) for t in ((i, i + 1, n + i), (n + i, i + 1, n + i + 1))], np.int32)
    cidx = np.array([0, n, n - 1, 2 * n - 1], np.int32)
    targets = p[cidx] + np.array([[0, 0, 0]] * 3 + [[0, edge, 0]])
    ok, ref = O.run_deform(p, faces, cidx, targets, 3)
    assert ok
    with gpu.ArapContext(len(p), faces) as ctx:
        ctx.set_precision("mixed", 1)
        ctx.set_factor_precision(bits)
        ctx.set_rest_positions(p)
        ctx.set_constraints(cidx, targets)
        assert W.bbox_rel_error(ctx.deform(3), ref, p) <= 1e-6
