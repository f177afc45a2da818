"""Set-up outputs around the sizes of the staged host copies (plain below 1 MB, one pinned
block, several with a ragged last one) and the degenerate searches: neighbours and distances
equal the oracle's bit for bit, and the weights asked for equal those of a second call that
keeps them in the engine only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,k", [(8, 1), (9, 2), (60, 35), (100, 35), (181, 35), (131, 61)])
def test_knn_and_weight_outputs(oracle, gpu_lib, side, k):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(side, seed=3)
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    idx, dist, dmin, davg = ctx.knn(k, want_dist=True)
    oidx, odist, odmin, odavg = oracle.knn(pts, k, period=per)
    assert np.array_equal(idx, oidx) and np.array_equal(dist, odist)
    if k > 1:
        assert (dmin, davg) == (odmin, odavg)
    if k >= 35:
        w, _ = ctx.weights(L.OP_GRAD, 3, 3, 1, want_w=True)
        ctx.set_equations(L.EQ_EULER2D, [1.4])
        u = W.isentropic_vortex(pts, 0.0)
        du = [np.empty_like(u), np.empty_like(u)]
        ctx.rhs(du[0], u.copy(), 0.0)
        ctx.weights(L.OP_GRAD, 3, 3, 1)
        ctx.rhs(du[1], u.copy(), 0.0)
        assert np.array_equal(du[0], du[1])
        rows = np.arange(0, side * side, 97)
        ref = oracle.weights_rows(pts, np.arange(side * side + 1) * k, oidx.ravel(), rows, period=per)
        at = (rows[:, None] * k + np.arange(k)).ravel()
        assert np.array_equal(w[at], ref[at])
    ctx.close()
