"""Row lengths around the groups of the software-pipelined staged gathers (three entries in
2D, four in 3D; rows of several lengths in one warp): every staged variant and the direct one
give the same bits, and rhs! with residual viscosity and hyperviscosity agrees with the FP64
fused-multiply-add form to the double-word sums' error (n = 20 products: below 1e-11 of the
largest |du|, as the worst-case bound 4.4e-12 of the condition scale at k = 35 allows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmin", [10, 15, 18])
def test_row_lengths_bit_identical(gpu_lib, kmin):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(33, seed=8)
    n = pts.shape[0]
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    idx, _, dmin, davg = ctx.knn(kmin + 6)
    ks = kmin + np.arange(n) % 7  # seven lengths inside every warp
    rp = np.concatenate([[0], np.cumsum(ks)]).astype(np.int64)
    cols = np.concatenate([idx[i, :k] for i, k in enumerate(ks)]).astype(np.int32)
    ctx.set_stencils(rp, cols)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.weights(L.OP_LAP, 3, 2, 2)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    u0 = W.isentropic_vortex(pts, 0.0)
    for sources, params in (([], []), ([L.SRC_RV], [[1, 1, davg, 0]]),
                            ([L.SRC_RV, L.SRC_HV_TOMINEC], [[1, 1, davg, 0], [dmin ** 4.5, 0, 0, 0]])):
        ctx.set_sources(sources, params)
        ctx.set_rv_state(0.1 * u0, 2)
        got = {}
        for v in (0, 6, 7, 9, 11):
            ctx.set_option(L.OPT_FP64_ARITH, L.ARITH_DW)
            ctx.set_option(L.OPT_DW_VARIANT, v)
            got[v] = np.empty_like(u0)
            ctx.rhs(got[v], u0.copy(), 0.0)
            assert np.array_equal(got[v], got[0]), v
        ctx.set_option(L.OPT_FP64_ARITH, L.ARITH_DFMA)
        ref = np.empty_like(u0)
        ctx.rhs(ref, u0.copy(), 0.0)
        assert np.abs(got[0] - ref).max() <= 1e-11 * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("k", [12, 13, 14, 15])
def test_row_lengths_3d(gpu_lib, k):
    """3D rows of every remainder modulo four against the FP64 fused-multiply-add form."""
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, _h = W.jittered_grid3(11, seed=6)
    ctx = L.Context(0)
    ctx.set_points(pts, (1.0, 1.0, 1.0))
    ctx.knn(k)
    ctx.weights(L.OP_GRAD, 3, 1, 1)
    ctx.set_equations(L.EQ_EULER3D, [1.4])
    u0 = W.euler3d_wave(pts)
    out = []
    for arith in (L.ARITH_DW, L.ARITH_DFMA):
        ctx.set_option(L.OPT_FP64_ARITH, arith)
        du = np.empty_like(u0)
        ctx.rhs(du, u0.copy(), 0.0)
        out.append(du)
    assert np.abs(out[0] - out[1]).max() <= 1e-11 * np.abs(out[1]).max()
    ctx.close()


@pytest.mark.parametrize("kmin", [10, 15])
def test_fp32_row_lengths_bit_identical(gpu_lib, kmin):
    """The FP32 gathers' mappings (direct, bulk copies, staged in register groups of three) on
    rows of seven lengths, with every source combination: the same bits."""
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(33, seed=8)
    n = pts.shape[0]
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    idx, _, dmin, davg = ctx.knn(kmin + 6)
    ks = kmin + np.arange(n) % 7
    rp = np.concatenate([[0], np.cumsum(ks)]).astype(np.int64)
    ctx.set_stencils(rp, np.concatenate([idx[i, :k] for i, k in enumerate(ks)]).astype(np.int32))
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.weights(L.OP_LAP, 3, 2, 2)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    ctx.set_precision(L.PREC_FP32)
    u0 = W.isentropic_vortex(pts, 0.0)
    rv, hv = [1, 1, davg, 0], [dmin ** 4.5, 0, 0, 0]
    for sources, params in (([], []), ([L.SRC_RV], [rv]), ([L.SRC_HV_TOMINEC], [hv]),
                            ([L.SRC_RV, L.SRC_HV_TOMINEC], [rv, hv])):
        ctx.set_sources(sources, params)
        ctx.set_rv_state(0.1 * u0, 2)
        ref = None
        for mode in (L.GATHER_THREAD, L.GATHER_HALO, L.GATHER_STAGED):
            ctx.set_option(L.OPT_GATHER, mode)
            du = np.empty_like(u0)
            ctx.rhs(du, u0.copy(), 0.0)
            ref = du if ref is None else ref
            assert np.array_equal(du, ref), mode
    ctx.close()
