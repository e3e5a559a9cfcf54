"""Rows of FP64 products that the digit planes cannot hold (subnormal, infinite), and what such a
row leaves behind in a captured application."""
import numpy as np
import pytest
import torch

from grafttn import _lib
from grafttn.contractions import EffectiveMap
from grafttn.device import Context

pytestmark = pytest.mark.gpu


def crandn(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2)


def contract(ctx, A, B, prec):
    return ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[-1, 1], [1, -2]], None, None,
                                     _lib.PRECISIONS[prec]))


def test_a_replay_forgets_an_infinite_row():
    """A captured FP64 application, replayed on good input, on input with an infinity, and on the
    good input again: the last result has the bits of the first."""
    rng = np.random.default_rng(8)
    D, w = 96, 5
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = Context(0)
        labels, order = [[1, 2], [1, 3, -1], [2, 3, -2]], [0, 1, 2]
        statics = [crandn(rng, (D, w, D)), crandn(rng, (D, w, D))]
        m = EffectiveMap(ctx, (D, D), labels, order, [ctx.upload(s) for s in statics], "fp64")
        good, bad = ctx.upload(crandn(rng, (D, D))), ctx.upload(crandn(rng, (D, D)))
        bad[7, 9] = complex(np.inf, 0.0)
        x, y = ctx.copy(good), ctx.empty(m.y_shape)
        m.apply_into(x, y)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            m.apply_into(x, y)

        def replay(v):
            x.copy_(v)
            graph.replay()
            stream.synchronize()
            return ctx.download(y)
        first = replay(good)
        assert not np.isfinite(replay(bad)).all()
        assert np.array_equal(replay(good), first)
        m.close()
        ctx.close()


@pytest.mark.parametrize("prec", ["fp64", "fp64e"])
def test_subnormal_rows_are_multiplied(ctx, prec):
    rng = np.random.default_rng(5)
    M, K, N = 300, 700, 200
    A, B = crandn(rng, (M, K)), crandn(rng, (K, N)) * 1e100
    A[3] *= 1e-310
    got, ref = contract(ctx, A, B, prec), A @ B
    assert np.abs(ref[3]).min() > 1e-213
    assert np.all(np.abs(got - ref) <= 4 * K * 2.0 ** -52 * (np.abs(A) @ np.abs(B)))
    got = contract(ctx, np.ascontiguousarray(B.T), np.ascontiguousarray(A.T), prec)
    assert np.all(np.abs(got - ref.T) <= 4 * K * 2.0 ** -52 * (np.abs(A) @ np.abs(B)).T)


@pytest.mark.parametrize("K", [524281, 600001, 2097120])
def test_very_long_sums(ctx, K):
    """Products of more than 2^19 terms, the summed index slow and fast in memory."""
    rng = np.random.default_rng(1)
    A, B = crandn(rng, (K, 40)), crandn(rng, (K, 33))
    ref = A.T @ B
    tol = 4 * K * 2.0 ** -52 * (np.abs(A).T @ np.abs(B))
    for la, a in (([1, -1], A), ([-1, 1], A.T)):
        got = ctx.download(ctx.contract([ctx.upload(a), ctx.upload(B)], [la, [1, -2]], None, None,
                                        _lib.PRECISIONS["fp64"]))
        assert np.all(np.abs(got - ref) <= tol)


def test_very_long_sums_of_a_map(ctx):
    """The same with offset tables, beyond 2^20 terms."""
    K = 1048600
    rng = np.random.default_rng(2)
    A, B = crandn(rng, (K, 40)), crandn(rng, (K, 33))
    m = EffectiveMap(ctx, A.shape, [[1, -1], [1, -2]], [0, 1], [ctx.upload(B)], "fp64")
    got = ctx.download(m(ctx.upload(A)))
    m.close()
    assert np.all(np.abs(got - A.T @ B) <= 4 * K * 2.0 ** -52 * (np.abs(A).T @ np.abs(B)))
