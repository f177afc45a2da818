"""The IGR solve in double-word arithmetic over the staged layout against the FP64 kernels
(MFT_ARITH_DFMA) on the same inputs: all row groups staged, none (a shuffled node order kept as
the layout order) and a mix; row lengths of every remainder modulo the register group of three
entries; one group and several.  Within 1e-9 of the largest |du|, the bound of the solve
against the oracle; the iteration counts agree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,shuffled,k", [(11, 0.0, 20), (33, 0.0, 21), (64, 0.0, 35), (64, 1.0, 22),
                                             (64, 0.5, 20)])
def test_igr_forms_agree(gpu_lib, side, shuffled, k):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, h = W.vortex_cloud(side, seed=2)
    n = pts.shape[0]
    perm = np.arange(n)
    m = int(shuffled * n)
    if m:
        perm[n - m:] = n - m + np.random.default_rng(3).permutation(m)
        pts = np.ascontiguousarray(pts[perm])
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    ctx.set_option(L.OPT_LAYOUT_ORDER, 0 if m else 1)
    ctx.knn(k)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    ctx.set_sources([L.SRC_IGR], [[h * h, 20.0, 0.0, 0.0]])
    u = W.isentropic_vortex(pts, 0.0)
    out, its = [], []
    for arith in (L.ARITH_DW, L.ARITH_DFMA):
        ctx.set_option(L.OPT_FP64_ARITH, arith)
        du = np.empty_like(u)
        ctx.rhs(du, u.copy(), 0.0)
        if arith == L.ARITH_DW and m:
            assert ctx.get_option(L.OPT_HALO_STAGED_FWD) < ctx.get_option(L.OPT_HALO_GROUPS)
        its.append(ctx.get_option(L.OPT_IGR_ITERS))
        out.append(du)
    ctx.close()
    assert its[0] == its[1]
    assert np.abs(out[0] - out[1]).max() <= 1e-9 * np.abs(out[1]).max()
