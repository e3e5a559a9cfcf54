"""The whole-chip Jacobi SVD (and its QR front end) against numpy: odd column counts, wide and
tall, graded, rank-deficient, zero and badly scaled matrices."""
import numpy as np
import pytest

from oracle import ttn_oracle as O

pytestmark = pytest.mark.gpu


def check(ctx, a, **kw):
    U, S, Vh, disc = ctx.svd_trunc(ctx.upload(a), **kw)
    U, Vh = ctx.download(U), ctx.download(Vh)
    s = np.linalg.svd(a, compute_uv=False)
    r, eps = len(S), 2.0 ** -52 * max(a.shape)
    assert np.all(np.diff(S) <= 0) and np.all(np.abs(S - s[:r]) <= eps * s[0])
    assert np.linalg.norm(U.conj().T @ U - np.eye(r)) <= 30 * eps
    assert np.linalg.norm(Vh @ Vh.conj().T - np.eye(r)) <= 30 * eps
    rest = np.linalg.norm(s[r:])
    assert abs(disc - rest) <= eps * s[0] * np.sqrt(len(s))
    assert np.linalg.norm(a - (U * S) @ Vh, 2) <= (s[r] if r < len(s) else 0.0) + 30 * eps * s[0]
    return S


@pytest.mark.parametrize("m,n", [(65, 65), (66, 67), (192, 192), (191, 200), (240, 131), (383, 383), (100, 700),
                                 (1500, 70), (70, 1500), (20, 1000), (5000, 33), (90, 180)])
def test_jacobi_svd_matches_numpy(ctx, m, n):
    rng = np.random.default_rng(m + n)
    a = O.randn_c(rng, (m, n))
    assert len(check(ctx, a)) == min(m, n)
    graded = a * np.logspace(0, -11, n)[None, :] * np.logspace(0, -3, m)[:, None]
    check(ctx, graded)
    check(ctx, graded, maxdim=min(m, n) // 3)
    check(ctx, a * 1e-200, maxdim=min(m, n) // 2)


@pytest.mark.parametrize("m,n", [(128, 150), (300, 90), (400, 66)])
def test_jacobi_svd_of_deficient_matrices(ctx, m, n):
    rng = np.random.default_rng(m)
    low = O.randn_c(rng, (m, 7)) @ O.randn_c(rng, (7, n))
    assert len(check(ctx, low, rtol=1e-12)) == 7
    U, S, Vh, _ = ctx.svd_trunc(ctx.upload(np.zeros((m, n), dtype=np.complex128)))
    assert len(S) == min(m, n) and np.all(S == 0.0)
    ident = np.zeros((m, n), dtype=np.complex128)
    np.fill_diagonal(ident, 1.0)
    assert np.allclose(check(ctx, ident), 1.0, atol=1e-14)
