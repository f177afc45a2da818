"""The weight kernel at the edges of its size classes (one, two or three warps per system;
rows of the backward solve within one, two or more warps; one to three right-hand sides):
the weights equal the oracle's bit for bit, alone and mixed in one batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# n = k + monomials around 16/17, 32/33, 48/49, 64/65, 80/81 and a large one
SIZES = {1: (3, [7, 8, 13, 14, 29, 30]), 2: (10, [11, 22, 23, 38, 39, 54, 55, 70, 71, 95]),
         3: (10, [14, 22, 23, 38, 39, 54, 55, 70, 71, 90])}
DEG = {1: 2, 2: 3, 3: 2}


def _group(dim, seed, order):
    rng = np.random.default_rng(seed)
    n = 240
    pts = np.ascontiguousarray(rng.uniform(-1, 1, (n, dim)))
    ks = np.resize(SIZES[dim][1], n)
    d2 = ((pts[:, None] - pts[None]) ** 2).sum(-1)
    idx = np.argsort(d2, axis=1, kind="stable")
    rp = np.concatenate([[0], np.cumsum(ks)]).astype(np.int64)
    cols = np.concatenate([idx[i, :k] for i, k in enumerate(ks)]).astype(np.int32)
    return pts, rp, cols, 3, DEG[dim], order


@pytest.mark.parametrize("dims,order", [((1,), 1), ((2,), 1), ((2,), 2), ((3,), 1), ((3,), 2),
                                        ((2, 3), 1)])
def test_size_classes_match_oracle(oracle, gpu_lib, dims, order):
    from meshfree_gb300 import _lib as L
    groups = [_group(d, 50 + d, order) for d in dims]
    ctx = L.Context(0)
    got, _ = ctx.weights_batch(groups)
    ctx.close()
    for (pts, rp, cols, p, deg, o), w in zip(groups, got):
        ref = oracle.weights(pts, rp, cols, rbf_pow=p, polydeg=deg, deriv_order=o)
        assert np.array_equal(w.view(np.int64), np.ascontiguousarray(ref).view(np.int64))
