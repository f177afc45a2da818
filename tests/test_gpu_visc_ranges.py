"""The viscosity's FP32 shortcut where FP32 runs out of range: an upwind coefficient whose square
is subnormal in FP32 (large energy, tiny c_uw), and a residual viscosity that is subnormal itself
(huge density).  Nearly still flow, so that the shortcut's bound is the upwind viscosity; residual
viscosities on both sides of it, a few per cent apart.  min(eps_rv, eps_uw) against numpy, 1e-12
relative (a dozen FP64 operations, as in the test of the norms)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho,energy,uwc", [(1.0, 1e16, 4.735e-23), (1e30, 1.37e-30, 2e-15),
                                            (1.0, 2.5, 0.5)])
def test_min_of_viscosities(gpu_lib, rho, energy, uwc):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(33, seed=4)
    n = pts.shape[0]
    rng = np.random.default_rng(5)
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    ctx.knn(20)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    ctx.set_option(L.OPT_FP64_ARITH, L.ARITH_DW)  # with and without sources: the same du bits
    sound = np.sqrt(1.4 * 0.4 * energy / rho)
    u = np.empty((4, n))
    u[0] = rho * (1.0 + 0.01 * rng.uniform(-1, 1, n))
    u[1:3] = 1e-3 * sound * u[0] * rng.uniform(-1, 1, (2, n))
    u[3] = energy * (1.0 + 0.01 * rng.uniform(-1, 1, n))
    ctx.set_sources([], [])
    du = np.empty_like(u)
    ctx.rhs(du, u.copy(), 0.0)
    y = np.abs(u - u.sum(axis=1, keepdims=True) / n)
    norm = y.max(axis=1)
    v = u[1:3] / u[0]
    p = 0.4 * (u[3] - 0.5 * (u[1] * v[0] + u[2] * v[1]))
    uw = uwc * (np.sqrt((v * v).sum(axis=0)) + np.sqrt(1.4 * p / u[0]))
    c_rv = 2.0 * uw.mean()
    ad = du.copy()  # the residual in the density alone
    ad[0] += rng.uniform(0.8, 1.25, n) * norm[0]
    ctx.set_sources([L.SRC_RV], [[c_rv, 2.0 * uwc, 1.0, 1]])
    ctx.set_rv_state(ad, 3)
    out = np.empty_like(u)
    ctx.rhs(out, u.copy(), 0.0)
    rv = 0.5 * c_rv * (np.abs(ad - du) / norm[:, None]).max(axis=0)
    ref = np.minimum(rv, uw)
    err = np.abs(ctx.viscosity() - ref) / ref
    ctx.close()
    assert (rv < uw).sum() > n // 4 and (rv > uw).sum() > n // 4
    assert err.max() < 1e-12
