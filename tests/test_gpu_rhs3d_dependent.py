"""The 3D gather launched beside the flux kernel it depends on (profiling off) and after it
(profiling on, events between the two): the same sums, so the same bits, for states that
change from call to call; clouds of less than a group, a ragged last group and several waves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [4, 11, 40])
@pytest.mark.parametrize("halo", [128, 256])
def test_gather_waits_for_flux(gpu_lib, side, halo):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, _h = W.jittered_grid3(side, seed=6)
    ctx = L.Context(0)
    ctx.set_option(L.OPT_HALO_ROWS, halo)
    ctx.set_points(pts, (1.0, 1.0, 1.0))
    ctx.knn(20)
    ctx.weights(L.OP_GRAD, 3, 1, 1)
    ctx.set_equations(L.EQ_EULER3D, [1.4])
    u0 = W.euler3d_wave(pts)
    ctx.set_option(L.OPT_FP64_ARITH, L.ARITH_DW)
    beside, after = [], []
    for on, out in ((False, beside), (True, after)):
        ctx.profile(on)
        for k in range(12):
            du = np.empty_like(u0)
            ctx.rhs(du, u0 * (1.0 + 0.01 * k), 0.0)
            out.append(du)
        ctx.profile(False)
    for k, (a, b) in enumerate(zip(beside, after)):
        assert np.array_equal(a, b), k
    ctx.close()
