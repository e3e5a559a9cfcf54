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
