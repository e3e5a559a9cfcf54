"""Small FP64 products: tiles of 4 x 4 and 8 x 8 outputs at the edges of their k blocks (64) and
of the offset window (512), the last step written straight into the result's leg order, and a
map applied in place."""
import numpy as np
import pytest

from grafttn import _lib
from grafttn.contractions import EffectiveMap

pytestmark = pytest.mark.gpu


def crandn(rng, shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


# (a, b) x (n,) outputs: 5 x 7 x 3 in 4 x 4 tiles, 40 x 4 x 150 and more in 8 x 8 tiles.  K above 64
# so that the product is not a narrow one; K at most 1200 keeps it in one slice for many outputs.
@pytest.mark.parametrize("a,b,n", [(5, 7, 3), (1, 1, 1), (40, 4, 150), (33, 5, 129)])
@pytest.mark.parametrize("K", [65, 127, 128, 129, 300])
@pytest.mark.parametrize("out", [(-1, -2, -3), (-3, -1, -2), (-2, -3, -1), (-2, -1, -3)])
def test_small_products_in_any_leg_order(ctx, a, b, n, K, out):
    rng = np.random.default_rng(a + b + n + K)
    A, B = crandn(rng, (a, K, b)), crandn(rng, (K, n))
    y = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[out[0], 1, out[1]], [1, out[2]]], None, None,
                                  _lib.PRECISIONS["fp64"]))
    perm = np.argsort([-l for l in out])
    ref = np.transpose(np.einsum("akb,kn->abn", A, B), perm)
    mag = np.transpose(np.einsum("akb,kn->abn", np.abs(A), np.abs(B)), perm)
    # 2K fused multiply-adds a part, in any order of summation
    assert y.shape == ref.shape and np.all(np.abs(y - ref) <= 2 * (2 * K + 20) * 2.0 ** -53 * np.sqrt(2) * mag)


@pytest.mark.parametrize("K", [511, 512, 513, 1100])
def test_offset_window(ctx, K):
    rng = np.random.default_rng(K)
    A, B = crandn(rng, (K, 3)), crandn(rng, (K, 2))
    y = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[1, -1], [1, -2]], None, None,
                                  _lib.PRECISIONS["fp64"]))
    bound = 2 * (2 * K + 20) * 2.0 ** -53 * np.sqrt(2) * (np.abs(A).T @ np.abs(B))
    assert np.all(np.abs(y - A.T @ B) <= bound)


@pytest.mark.parametrize("labels", [[[1, -2], [-1, 1]], [[-2, 1], [1, -1]]])
def test_one_step_map_in_place(ctx, labels):
    rng = np.random.default_rng(3)
    x, S = crandn(rng, (70, 70)), crandn(rng, (70, 70))
    m = EffectiveMap(ctx, x.shape, labels, [0, 1], [ctx.upload(S)], "fp64")
    d = ctx.upload(x)
    ref = ctx.download(m(d))
    m.apply_into(d, d)
    assert np.array_equal(ctx.download(d), ref)
    assert np.allclose(ref, S @ x if labels[0][0] == 1 else (x @ S).T, rtol=0, atol=1e-11)
    m.close()


# the staged elements (16 a thread) at K around their number, N around the outputs of a pass
@pytest.mark.parametrize("M", [1, 33, 300, 40001])
@pytest.mark.parametrize("K", [1, 14, 15, 16, 17, 31, 64])
@pytest.mark.parametrize("N", [1, 9, 17, 33])
def test_narrow_products_skip_zeros(ctx, M, K, N):
    rng = np.random.default_rng(M + K + N)
    A, B = crandn(rng, (K, M)), crandn(rng, (K, N))
    B = np.where(rng.random((K, N)) < 0.3, np.where(rng.random((K, N)) < 0.5, B.real, B), 0)
    y = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[1, -1], [1, -2]], None, None,
                                  _lib.PRECISIONS["fp64"]))
    assert np.all(np.abs(y - A.T @ B) <= 2 * (2 * K + 2) * 2.0 ** -53 * np.sqrt(2) * (np.abs(A).T @ np.abs(B)))
    A[K // 2, M - 1] = np.inf  # times a complex zero: NaN, in this row only
    y = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[1, -1], [1, -2]], None, None,
                                  _lib.PRECISIONS["fp64"]))
    bad = np.zeros((M, N), dtype=bool)
    bad[M - 1] = True
    assert np.array_equal(~np.isfinite(y), bad)
