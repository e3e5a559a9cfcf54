"""Truncated SVDs of finite matrices whose columns differ by more than the FP64 range of a square,
and of matrices with exact zero singular values among the kept ones: finite, orthonormal factors."""
import numpy as np
import pytest

from oracle import ttn_oracle as O

pytestmark = pytest.mark.gpu


def factors(ctx, a, **kw):
    U, S, Vh, _ = ctx.svd_trunc(ctx.upload(a), **kw)
    return ctx.download(U), S, ctx.download(Vh)


def check(ctx, a, **kw):
    U, S, Vh = factors(ctx, a, **kw)
    r, eps = len(S), 2.0 ** -52 * max(a.shape)
    assert np.isfinite(U).all() and np.isfinite(Vh).all() and np.isfinite(S).all()
    s = np.linalg.svd(a, compute_uv=False)
    assert np.all(np.abs(S - s[:r]) <= eps * s[0])
    assert np.linalg.norm(U.conj().T @ U - np.eye(r)) <= 30 * eps
    assert np.linalg.norm(Vh @ Vh.conj().T - np.eye(r)) <= 30 * eps
    assert np.linalg.norm(a - (U * S) @ Vh, 2) <= (s[r] if r < len(s) else 0.0) + 30 * eps * s[0]


@pytest.mark.parametrize("scale", [1e-140, 1e-150, 1e-154, 1e-156, 1e-160, 1e-170, 1e-250, 5e-324])
@pytest.mark.parametrize("m,n", [(100, 90), (90, 100), (900, 80), (80, 900)])
def test_one_tiny_column(ctx, m, n, scale):
    rng = np.random.default_rng(m)
    a = O.randn_c(rng, (m, n))
    for pos in (-1, 0, 17):
        b = a.copy()
        if m >= n:
            b[:, pos] *= scale
        else:
            b[pos] *= scale
        check(ctx, b, maxdim=40)
        check(ctx, b)


def test_columns_of_every_size(ctx):
    rng = np.random.default_rng(3)
    a = O.randn_c(rng, (120, 100))
    check(ctx, a * np.logspace(0, -300, 100)[None, :])
    check(ctx, a * np.logspace(-300, 0, 100)[None, :], maxdim=30)
    check(ctx, a * np.logspace(0, -300, 120)[:, None])


def zero_padded(rng, m, n, zero_rows, zero_cols):
    a = O.randn_c(rng, (m, n))
    a[rng.permutation(m)[:zero_rows]] = 0
    a[:, rng.permutation(n)[:zero_cols]] = 0
    return a


@pytest.mark.parametrize("m,n", [(100, 90), (90, 100), (67, 67), (900, 80), (80, 900)])
def test_kept_values_of_zero(ctx, m, n):
    rng = np.random.default_rng(n)
    for zr, zc in [(0, 1), (1, 0), (13, 20), (min(m, n) - 1, 3)]:
        check(ctx, zero_padded(rng, m, n, zr, zc))
        check(ctx, zero_padded(rng, m, n, zr, zc), maxdim=min(m, n) - 1)
    for z in (1, 17, min(m, n) - 1):  # padding at the end: values of exactly zero
        a = O.randn_c(rng, (m, n))
        if m >= n:
            a[:, n - z:] = 0
        else:
            a[m - z:] = 0
        check(ctx, a)
        check(ctx, a, maxdim=min(m, n) - 1)
    one = np.zeros((m, n), dtype=np.complex128)
    one[3, 5] = 2j
    check(ctx, one)
    check(ctx, np.zeros_like(one) + np.diag(np.r_[1.0, np.zeros(max(m, n) - 1)])[:m, :n], maxdim=2)


def test_zeros_cost_no_second_factorisation(ctx):
    """A padded matrix takes about the time of a full one: the rotations' result is used (a second
    factorisation, by bidiagonalisation, takes three times as long as they do)."""
    import time
    rng = np.random.default_rng(1)
    mats = [ctx.upload(a) for a in (O.randn_c(rng, (192, 192)),
                                  np.pad(O.randn_c(rng, (192, 180)), ((0, 0), (0, 12))))]
    best = [1e9, 1e9]
    for _ in range(4):
        for i, a in enumerate(mats):
            t = time.perf_counter()
            ctx.svd_trunc(a)
            best[i] = min(best[i], time.perf_counter() - t)
    assert best[1] <= 2.0 * best[0], best
