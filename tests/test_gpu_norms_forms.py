"""The residual viscosity's means and norms where their forms meet, and with states that are not
finite.  The FP32 form on either side of its change from one cluster to grid reductions (24,576
nodes; just above it some blocks of the grid have one node or none in their last round): within
1e-5 of the FP64 form's viscosity (a dozen FP32 operations of 6e-8 each on norms that both forms
take in FP64).  An infinity or a NaN in one component of one node, in the cluster and in the grid
reductions with their skipping maximum pass (NaN orders above infinity in the maximum): the
viscosity of the other nodes against numpy, 1e-12, the upwind one where the residual one is not
finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(pts, per, k=20):
    from meshfree_gb300 import _lib as L
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    _, _, _, h = ctx.knn(k)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    return ctx, h


def _visc(ctx, L, u, ad, par):
    ctx.set_sources([L.SRC_RV], [par])
    ctx.set_rv_state(ad, 3)
    ctx.rhs(np.empty_like(u), u.copy(), 0.0)
    return ctx.viscosity()


@pytest.mark.parametrize("nx,ny", [(128, 192), (163, 151), (211, 199)])  # 24,576, 24,613, 41,989
@pytest.mark.parametrize("mode", [0, 1])
def test_fp32_form(gpu_lib, nx, ny, mode):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    h = 10.0 / max(nx, ny)
    pts, _ = W.jittered_grid(nx, ny, hi=(nx * h, ny * h), seed=3)
    ctx, davg = _ctx(pts, (nx * h, ny * h))
    rng = np.random.default_rng(nx)
    u = W.isentropic_vortex(pts, 0.0) * (1.0 + 0.01 * rng.standard_normal((4, nx * ny)))
    ad = 100.0 * rng.standard_normal(u.shape)  # large beside du: the residual is ad's
    eps = {}
    for prec in (L.PREC_FP64, L.PREC_FP32):
        ctx.set_precision(prec)
        eps[prec] = _visc(ctx, L, u, ad, [1e-3, 1e9, davg, mode])
    ctx.close()
    ref = eps[L.PREC_FP64]
    assert (np.abs(eps[L.PREC_FP32] - ref) / ref.max()).max() < 1e-5


@pytest.mark.parametrize("side", [33, 257, 300])  # the cluster; the grid reductions
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("component", [0, 3])
def test_not_finite_states(gpu_lib, side, mode, value, component):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(side, seed=4)
    n = side * side
    ctx, h = _ctx(pts, per)
    rng = np.random.default_rng(side)
    u = W.isentropic_vortex(pts, 0.0) * (1.0 + 0.01 * rng.standard_normal((4, n)))
    u[component, n // 2] = value
    ad = rng.standard_normal(u.shape)
    du = np.empty_like(u)
    ctx.set_sources([], [])
    with pytest.raises(L.MFTError, match="NaN or infinite"):  # the outputs are written all the same
        ctx.rhs(du, u.copy(), 0.0)
    with pytest.raises(L.MFTError, match="NaN or infinite"):
        _visc(ctx, L, u, ad, [1.0, 1.0, h, mode])
    eps = ctx.viscosity()
    ctx.close()
    with np.errstate(all="ignore"):
        mean = u.sum(axis=1) / (n * (4 if mode == 0 else 1))
        y = np.abs(u - mean[:, None])
        norm = y[:, np.lexsort(y[::-1])[-1]] if mode == 0 else y.max(axis=1)  # NaN last, NaN kept
        rv = 0.5 * h * h * (np.abs(ad - du) / norm[:, None]).max(axis=0)
    fin = np.arange(n) != n // 2
    rho, v = u[0, fin], u[1:3, fin] / u[0, fin]
    p = 0.4 * (u[3, fin] - 0.5 * rho * (v * v).sum(axis=0))
    uw = 0.5 * h * (np.sqrt((v * v).sum(axis=0)) + np.sqrt(1.4 * p / rho))
    ref = np.where(np.isfinite(rv[fin]), np.minimum(rv[fin], uw), uw)
    assert (np.abs(eps[fin] - ref) / ref).max() < 1e-12
