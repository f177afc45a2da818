"""The IGR solve of the double-word engine form keeps FP64 arithmetic: its part of the momentum
rows (du with it less du without it) against the FP64 form's, which runs the unstaged kernels.
The two solves differ in the order of the dot products' parts alone; solves in FP64 lie up to
2.2e-12 of the part's maximum from one in quad precision (100 combinations of size, stencil, state
and alpha), so two of them within 4.4e-12: 1e-11 is asked.  (Solves in double-word sums are 1e-11
to 1.4e-10 off here.)  Staged clouds of one group and of several, ragged last groups, rows of several
lengths modulo the register group of five; scattered node numbers, where no group is staged
and the unstaged kernels run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,k,shuffled", [(11, 20, False), (33, 35, False), (33, 21, False), (64, 24, False),
                                             (64, 22, False), (96, 28, False), (64, 24, True)])
def test_igr_part_is_fp64(gpu_lib, side, k, shuffled):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, h = W.vortex_cloud(side, seed=2)
    n = pts.shape[0]
    if shuffled:
        pts = np.ascontiguousarray(pts[np.random.default_rng(3).permutation(n)])
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    ctx.set_option(L.OPT_LAYOUT_ORDER, 0 if shuffled else 1)
    ctx.knn(k)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    a = 2 * np.pi * pts / 10.0
    rho = 1.0 + 0.1 * np.sin(a[:, 0]) * np.cos(2 * a[:, 1] + 0.3)
    v1 = 0.5 + 0.15 * np.sin(a[:, 1] + 1.0) * np.cos(a[:, 0])
    v2 = -0.3 + 0.1 * np.cos(2 * a[:, 0] + 2.0) * np.sin(a[:, 1])
    p = 1.0 + 0.1 * np.sin(a[:, 0]) * np.sin(a[:, 1] + 0.7)
    u = np.ascontiguousarray(np.stack([rho, rho * v1, rho * v2, p / 0.4 + 0.5 * rho * (v1 * v1 + v2 * v2)]))
    part = {}
    for arith in (L.ARITH_DW, L.ARITH_DFMA):
        ctx.set_option(L.OPT_FP64_ARITH, arith)
        du = []
        for source in (True, False):
            ctx.set_sources(*(([L.SRC_IGR], [[20.0 * h * h, 20.0, 0, 0]]) if source else ([], [])))
            du.append(np.empty_like(u))
            ctx.rhs(du[-1], u.copy(), 0.0)
        part[arith] = du[0][1:3] - du[1][1:3]
        if arith == L.ARITH_DW:
            staged = ctx.get_option(L.OPT_HALO_STAGED_FWD)
            assert (staged < ctx.get_option(L.OPT_HALO_GROUPS)) == shuffled
    ctx.close()
    ref = part[L.ARITH_DFMA]
    assert np.abs(part[L.ARITH_DW] - ref).max() <= 1e-11 * np.abs(ref).max()
