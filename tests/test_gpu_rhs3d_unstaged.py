"""The 3D gather where row groups have no neighbour list and read the flux records from global
memory, which the flux kernel before it must have completed: scattered node numbers kept as the
layout order (no group staged, or half of them).  The same bits with the launches back to back and
with events between them (profiling), for states that change from call to call; and the bits of
the staged gather on the same cloud in Morton order (entries in structure order, so that every row
forms the same sum in the same order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [11, 40])
@pytest.mark.parametrize("shuffled", [1.0, 0.5])
def test_unstaged_groups_wait_for_flux(gpu_lib, side, shuffled):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, _h = W.jittered_grid3(side, seed=6)
    n = pts.shape[0]
    m = int(shuffled * n)
    perm = np.arange(n)
    perm[n - m:] = n - m + np.random.default_rng(3).permutation(m)
    pts = np.ascontiguousarray(pts[perm])
    ctx = L.Context(0)
    ctx.set_option(L.OPT_LAYOUT_ORDER, 0)
    ctx.set_option(L.OPT_ENTRY_ORDER, 0)
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
    assert ctx.get_option(L.OPT_HALO_STAGED_FWD) < ctx.get_option(L.OPT_HALO_GROUPS)
    for k, (a, b) in enumerate(zip(beside, after)):
        assert np.array_equal(a, b), k
    ctx.set_option(L.OPT_LAYOUT_ORDER, 1)
    staged = np.empty_like(u0)
    ctx.rhs(staged, u0.copy(), 0.0)
    assert ctx.get_option(L.OPT_HALO_STAGED_FWD) == ctx.get_option(L.OPT_HALO_GROUPS)
    assert np.array_equal(staged, beside[0])
    ctx.close()
