"""The Krylov projections, updates and steps at the group and block edges: gtn_dot and the
allocation-free projections against numpy, solves with and without a step queued ahead, and an
expansion that ends early."""
import ctypes as C

import numpy as np
import pytest

from grafttn.contractions import EffectiveMap
from oracle import ttn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 1024, 1025, 70000])
@pytest.mark.parametrize("J", [1, 2, 3, 5, 8, 9, 23, 64])
def test_projections_of_every_group_size(ctx, n, J):
    import torch
    rng = np.random.default_rng(n + J)
    V, w = O.randn_c(rng, (J, n)), O.randn_c(rng, (n,))
    dV, dw, out = ctx.upload(V), ctx.upload(w), ctx.empty((J,))
    st = ctx.lib.gtn_multidot_noalloc(C.c_void_p(torch.cuda.current_stream().cuda_stream), n, J,
                                      C.c_void_p(dV.data_ptr()), n, C.c_void_p(dw.data_ptr()),
                                      C.c_void_p(out.data_ptr()))
    assert st == 0
    got = ctx.download(out)
    assert np.all(np.abs(got - V.conj() @ w) <= (n + 4) * 2.0 ** -52 * (np.abs(V) @ np.abs(w)))
    assert abs(ctx.dot(dV[0], dw) - np.vdot(V[0], w)) <= (n + 4) * 2.0 ** -52 * (np.abs(V[0]) @ np.abs(w))


def dense_map(ctx, H, prec="fp64"):
    return EffectiveMap(ctx, (H.shape[0],), [[1], [-1, 1]], [0, 1], [ctx.upload(H)], prec)


@pytest.mark.parametrize("n", [3, 40, 300])
def test_exponential_of_a_map_with_an_invariant_start(ctx, n):
    """A start vector in a two-dimensional invariant subspace ends the expansion at once, with the
    next step already queued."""
    rng = np.random.default_rng(n)
    A = O.randn_c(rng, (n, n))
    H = (A + A.conj().T) / 2
    w, U = np.linalg.eigh(H)
    for v in (U[:, 0], (U[:, 0] + 2j * U[:, -1]) / np.sqrt(5), O.randn_c(rng, (n,))):
        m = dense_map(ctx, H)
        y, _ = m.exponentiate(-0.3j, ctx.upload(v), krylovdim=min(30, n), tol=1e-12)
        ref = U @ (np.exp(-0.3j * w) * (U.conj().T @ v))
        assert np.linalg.norm(ctx.download(y) - ref) <= 1e-10 * np.linalg.norm(ref)
        E, x, info = m.lanczos_min(ctx.upload(v + 1e-3 * O.randn_c(rng, (n,))), krylovdim=min(20, n), tol=1e-10)
        assert info["converged"] and abs(E - w[0]) <= 1e-9 * max(1.0, abs(w[0]))
        m.close()
