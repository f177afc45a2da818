"""The residual viscosity's means and norms at the edges of their two forms (one cluster of
blocks up to 65,536 nodes, two grid reductions above; fewer nodes than threads; ties of the
first component, which the lexicographic maximum breaks by the later ones; NaN-free states
with every node equal in one component): the viscosity of one rhs! against numpy, 1e-12
relative (a dozen FP64 operations on norms whose sums carry at most n u = 1.5e-11 of the mean,
here below 1e-13 by the pairwise-like block sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [12, 33, 256, 257])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("ties", [False, True])
def test_viscosity_norms(gpu_lib, side, mode, ties):
    from meshfree_gb300 import _lib as L
    from meshfree_gb300 import workloads as W
    pts, per, _h = W.vortex_cloud(side, seed=4)
    ctx = L.Context(0)
    ctx.set_points(pts, per)
    _, _, _, h = ctx.knn(20)
    ctx.weights(L.OP_GRAD, 3, 2, 1)
    ctx.set_equations(L.EQ_EULER2D, [1.4])
    u = W.isentropic_vortex(pts, 0.0)
    rng = np.random.default_rng(side)
    u *= 1.0 + 0.01 * rng.standard_normal(u.shape)
    if ties:  # three densities only, on both sides of the mean
        u[0] = np.array([0.75, 1.0, 1.25])[rng.integers(0, 3, u.shape[1])]
    ctx.set_sources([], [])
    du = np.empty_like(u)
    ctx.rhs(du, u.copy(), 0.0)
    ad = rng.standard_normal(u.shape)
    ctx.set_sources([L.SRC_RV], [[1.0, 1e9, h, mode]])
    ctx.set_rv_state(ad, 3)
    out = np.empty_like(u)
    ctx.rhs(out, u.copy(), 0.0)
    mean = u.sum(axis=1) / (u.shape[1] * (4 if mode == 0 else 1))
    y = np.abs(u - mean[:, None])
    norm = y[:, np.lexsort(y[::-1])[-1]] if mode == 0 else y.max(axis=1)
    ref = 0.5 * h * h * (np.abs(ad - du) / norm[:, None]).max(axis=0)
    err = np.abs(ctx.viscosity() - ref) / ref
    ctx.close()
    assert err.max() < 1e-12
