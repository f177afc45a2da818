"""The double-word adjoint gather where row groups have no neighbour list (scattered node numbers
kept as the layout order: no group staged, or some) and read the cotangent's pairs from global
memory: the bits of the direct gather and of the one with every group staged (Morton order;
entries in structure order, so that every row forms the same sum in the same order), with and
without boundary conditions and Flyer hyperviscosity.  Where every group is staged the pairs'
memory is not held."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffled", [1.0, 0.4])
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("flyer", [False, True])
def test_unstaged_groups(gpu_lib, shuffled, walls, flyer):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, tags, _h = W.advection_cloud(32, seed=4)
    n = pts.shape[0]
    m = int(shuffled * n)
    perm = np.arange(n)
    perm[n - m:] = n - m + np.random.default_rng(3).permutation(m)
    pts = np.ascontiguousarray(pts[perm])
    place = np.argsort(perm)
    ctx = L.Context(0)
    ctx.set_option(L.OPT_LAYOUT_ORDER, 0)
    ctx.set_option(L.OPT_ENTRY_ORDER, 0)
    ctx.set_points(pts)
    ctx.knn(20)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.weights(L.OP_HV, 5, 3, 4)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    if walls:
        idx = np.concatenate([place[np.asarray(t[0])] for t in tags.values()]).astype(np.int32)
        nrm = np.concatenate([np.asarray(t[1]) for t in tags.values()])
        ctx.set_bcs([L.BC_SLIP_WALL], [0, len(idx)], idx, nrm)
    else:
        ctx.set_bcs([], [0], np.zeros(0, np.int32), None)
    ctx.set_sources(*(([L.SRC_HV_FLYER], [[1e-9, 0, 0, 0]]) if flyer else ([], [])))
    ctx.set_option(L.OPT_FP64_ARITH, L.ARITH_DW)
    u = W.isentropic_vortex(pts, 0.0)
    lam = np.random.default_rng(2).standard_normal(u.shape)
    got = ctx.rhs_adjoint(lam, u)
    assert ctx.get_option(L.OPT_HALO_STAGED_REV) < ctx.get_option(L.OPT_HALO_GROUPS)
    ctx.set_option(L.OPT_DW_VARIANT, 2)
    assert np.array_equal(ctx.rhs_adjoint(lam, u), got)
    ctx.set_option(L.OPT_DW_VARIANT, -1)
    ctx.set_option(L.OPT_LAYOUT_ORDER, 1)
    assert np.array_equal(ctx.rhs_adjoint(lam, u), got)
    assert ctx.get_option(L.OPT_HALO_STAGED_REV) == ctx.get_option(L.OPT_HALO_GROUPS)
    ctx.close()


def test_pairs_not_held_when_staged(gpu_lib):
    """Every group staged: an adjoint product holds no pairs (4 MB of them per 131,072 nodes);
    the direct gather's are given back by the next staged one."""
    import torch
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(512, seed=4)
    n = pts.shape[0]
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    ctx.knn(20)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    ctx.set_sources([], [])
    ctx.set_option(L.OPT_FP64_ARITH, L.ARITH_DW)
    u = W.isentropic_vortex(pts, 0.0)
    lam = np.ones_like(u)
    free = []
    for variant in (-1, 2, -1):
        ctx.set_option(L.OPT_DW_VARIANT, variant)
        ctx.rhs_adjoint(lam, u)
        free.append(torch.cuda.mem_get_info(0)[0])
    ctx.close()
    assert free[0] - free[1] >= 32 * n and free[2] - free[1] >= 32 * n
