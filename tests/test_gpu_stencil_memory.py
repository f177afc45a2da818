"""The stencils that a neighbour search leaves on the device for the weights are given back when the
operators are placed for the first evaluation, with a new cloud and with operators from outside;
weights formed after that (from the host's stencils) are the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE, K = 300, 30


def _free():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def _cloud(L):
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(SIDE, seed=4)
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    return ctx, pts, per


@pytest.mark.parametrize("how", ["new cloud", "csc"])
def test_given_back(gpu_lib, how):
    from meshfree_gb300 import _lib as L
    ctx, pts, per = _cloud(L)
    n = pts.shape[0]
    idx = ctx.knn(K)[0]
    held = _free()
    if how == "new cloud":
        ctx.set_points(pts, per)
    else:
        colptr = np.arange(1, n + 2, dtype=np.int64)
        ctx.load_csc(L.OP_GRAD, 0, colptr, np.arange(1, n + 1, dtype=np.int64), np.ones(n))
    assert _free() - held >= idx.size * 4
    ctx.close()


def test_weights_after_the_first_evaluation(gpu_lib):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    ctx, pts, per = _cloud(L)
    ctx.knn(K)
    w0, _ = ctx.weights(L.OP_GRAD, 3, 2, 1, want_w=True)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    ctx.set_sources([], [])
    u = W.isentropic_vortex(pts, 0.0)
    ctx.rhs(np.empty_like(u), u.copy(), 0.0)
    w1, _ = ctx.weights(L.OP_GRAD, 3, 2, 1, want_w=True)
    ctx.close()
    assert np.array_equal(np.asarray(w0), np.asarray(w1))


def test_a_refused_search_leaves_the_stencils(gpu_lib):
    from meshfree_gb300 import _lib as L
    ctx, pts, per = _cloud(L)
    ctx.knn(K)
    w0, _ = ctx.weights(L.OP_GRAD, 3, 2, 1, want_w=True)
    with pytest.raises(L.MFTError):
        ctx.knn(2000)
    w1, _ = ctx.weights(L.OP_GRAD, 3, 2, 1, want_w=True)
    ctx.close()
    assert np.array_equal(np.asarray(w0), np.asarray(w1))
