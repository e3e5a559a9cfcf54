"""FP64 products of more than 64 terms, component by component: |y - exact| within the a-priori
bound of an FP64 sum, 2K 2^-53 sum_k |a_k| |b_k| a part, for operands graded within a row, with
zeros, noise, subnormal rows and rows out of the digit planes' range."""
import numpy as np
import pytest

from grafttn import _lib

pytestmark = pytest.mark.gpu


def crandn(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2)


def check(ctx, A, B, K):
    got = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[-1, 1], [1, -2]], None, None,
                                    _lib.PRECISIONS["fp64"]))
    # the bound for the kernel and once more for numpy's own sum, sqrt 2 for both parts
    tol = 2 * (2 * K + 4) * 2.0 ** -53 * np.sqrt(2) * (np.abs(A) @ np.abs(B)) + 5e-324 * K
    bad = ~(np.abs(got - A @ B) <= tol)
    assert not bad.any(), (int(bad.sum()), np.argwhere(bad)[:4].tolist())


SIZES = [(300, 700, 200), (129, 333, 161), (1100, 130, 700), (64, 66, 2000)]


@pytest.mark.parametrize("M,K,N", SIZES)
def test_graded_within_rows(ctx, M, K, N):
    rng = np.random.default_rng(M + K)
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N))
    check(ctx, A, B, K)
    A1, B1 = A.copy(), B.copy()
    A1[5, :] = 0
    A1[5, 0], A1[5, 1] = 1.0, 1e-18            # a row (1, 1e-18, 0 ..)
    B1[:, 7] = 0
    B1[1, 7] = 1.0                             # meets a column (0, 1, 0 ..)
    check(ctx, A1, B1, K)
    for lo in (-4, -12, -30):                  # Schmidt weights along the sum, and random sizes
        w = np.logspace(0, lo, K)
        check(ctx, A * w[None, :], B, K)
        check(ctx, A * w[None, :], B * w[:, None], K)
        check(ctx, A * w[None, :], B * w[::-1, None], K)
        check(ctx, A * 10.0 ** rng.uniform(lo, 0, (M, K)), B * 10.0 ** rng.uniform(lo, 0, (K, N)), K)


@pytest.mark.parametrize("noise", [0.0, 1e-16])
def test_identity_channel_meets_a_decaying_state(ctx, noise):
    rng = np.random.default_rng(11)
    M, K = 400, 250
    A = crandn(rng, (M, K)) * np.logspace(0, -12, K)[None, :]
    B = np.concatenate([np.eye(K) + noise * crandn(rng, (K, K)), crandn(rng, (K, K)) / 16], axis=1)
    check(ctx, A, B, K)


@pytest.mark.parametrize("M,K,N", SIZES[:2])
def test_sparse_operands(ctx, M, K, N):
    rng = np.random.default_rng(K)
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N))
    A[rng.random((M, K)) < 0.97] = 0
    B[rng.random((K, N)) < 0.97] = 0
    check(ctx, A, B, K)
    A *= 10.0 ** rng.uniform(-20, 0, (M, K))
    check(ctx, A, B, K)


@pytest.mark.parametrize("M,K,N", [(7700, 70, 645), (64 * 152 * 2 + 5, 130, 200)])
def test_many_tiles(ctx, M, K, N):
    """More tiles than CTAs of the check: dense rows are counted, graded, sparse and infinite ones met."""
    rng = np.random.default_rng(M)
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N))
    check(ctx, A, B, K)
    w = np.logspace(0, -18, K)
    for m in (0, 127, 128, 3333, M - 1):
        A[m] *= w if m % 2 else w[::-1]
    A[4000:4100][rng.random((100, K)) < 0.95] = 0
    A[2000] = 0
    B[:, 3] *= w
    B[:, N - 1] = 0
    B[K - 1, N - 1] = 1.0
    check(ctx, A, B, K)
    A[5000, K // 2] = np.inf
    got = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[-1, 1], [1, -2]], None, None,
                                    _lib.PRECISIONS["fp64"]))
    assert np.array_equal(np.isfinite(got).all(axis=1), np.arange(M) != 5000)


def test_a_map_with_decaying_input(ctx):
    """A compiled map (offset tables), its input and environments graded, in two leg orders."""
    from grafttn.contractions import EffectiveMap
    rng = np.random.default_rng(2)
    D, w = 100, 5
    L = crandn(rng, (D, w, D)) * np.logspace(0, -9, D)[None, None, :]
    R = crandn(rng, (D, w, D))
    L[:, 0], R[:, 0] = np.eye(D) + 1e-16 * crandn(rng, (D, D)), np.eye(D)
    x = crandn(rng, (D, 2, D)) * np.logspace(0, -10, D)[:, None, None] * np.logspace(0, -6, D)[None, None, :]
    for order in ([0, 1, 2], [0, 2, 1]):
        m = EffectiveMap(ctx, x.shape, [[1, -2, 2], [1, 3, -1], [2, 3, -3]], order, [ctx.upload(L), ctx.upload(R)],
                         "fp64")
        got = ctx.download(m(ctx.upload(x)))
        m.close()
        ref = np.einsum("asb,awc,bwd->csd", x, L, R, optimize=["einsum_path", (0, 1), (0, 1)])
        mag = np.einsum("asb,awc,bwd->csd", abs(x), abs(L), abs(R), optimize=["einsum_path", (0, 1), (0, 1)])
        # two steps of at most w D terms, each with the bound of its own sum; numpy's as well
        tol = 2 * 2 * (2 * w * D + 4) * 2.0 ** -53 * np.sqrt(2) * mag
        assert np.all(np.abs(got - ref) <= tol)


@pytest.mark.parametrize("M,K,N", [(300, 128, 300), (1000, 77, 154), (129, 1030, 1100)])
def test_noisy_identity_meets_flat_and_graded_rows(ctx, M, K, N):
    """Columns with one large entry among rounding noise of several sizes: the eighth digits decide."""
    rng = np.random.default_rng(K)
    A = crandn(rng, (M, K))
    A[1::3] *= np.logspace(0, -8, K)
    A[2::7] *= 10.0 ** rng.uniform(-20, 0, (len(A[2::7]), K))
    B = np.zeros((K, N), dtype=complex)
    B[np.arange(N) % K, np.arange(N)] = np.exp(1j * rng.uniform(0, 6, N)) * 10.0 ** rng.uniform(-3, 3, N)
    for noise in (1e-15, 1e-16, 1e-17, 1e-19):
        check(ctx, A, B + noise * np.abs(B).max(0) * crandn(rng, (K, N)), K)
        check(ctx, A, B + noise * np.abs(B).max(0) * 10.0 ** rng.uniform(-6, 0, (K, N)), K)


@pytest.mark.parametrize("tiny", [1e-10, 1e-18, 1e-30, 1e-100])
def test_the_only_terms_that_meet_are_tiny(ctx, tiny):
    """Rows and columns whose large entries meet zeros: the product of two tiny ones is all there is."""
    rng = np.random.default_rng(3)
    M, K, N = 300, 700, 200
    A, B = np.zeros((M, K), dtype=complex), np.zeros((K, N), dtype=complex)
    A[:, :300], B[400:, :] = crandn(rng, (M, 300)), crandn(rng, (300, N))
    check(ctx, A, B, K)  # nothing meets
    A[:, 350], B[350, :] = tiny * crandn(rng, M), tiny * crandn(rng, N)
    check(ctx, A, B, K)
    A[::2, 399], B[399, ::3] = tiny, -tiny
    check(ctx, A, B, K)
