"""Captured FP64 applications of two maps of one context, replayed on two streams at the same time:
each has buffers of its own (tiles of these products are shared by several CTAs, whose partial sums
go through memory), so every replay has the bits of an application by itself."""
import ctypes as C

import numpy as np
import pytest
import torch

from grafttn._lib import check
from grafttn.contractions import EffectiveMap
from grafttn.device import Context

pytestmark = pytest.mark.gpu


def crandn(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / np.sqrt(2)


@pytest.mark.parametrize("prec", ["fp64", "fp64e"])
def test_two_graphs_on_two_streams(prec):
    rng = np.random.default_rng(4)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with torch.cuda.stream(streams[0]):
        ctx = Context(0)
        labels, order = [[1, 2], [1, 3, -1], [2, 3, -2]], [0, 1, 2]
        maps, xs, ys, alone = [], [], [], []
        for D in (130, 161):
            statics = [crandn(rng, (D, 5, D)), crandn(rng, (D, 5, D))]
            maps.append(EffectiveMap(ctx, (D, D), labels, order, [ctx.upload(s) for s in statics], prec))
            xs.append(ctx.upload(crandn(rng, (D, D))))
            ys.append(ctx.empty(maps[-1].y_shape))
            maps[-1].apply_into(xs[-1], ys[-1])
            ctx.sync()
            alone.append(ctx.download(ys[-1]))
    graphs = []
    for m, x, y, s in zip(maps, xs, ys, streams):
        check(ctx.lib.gtn_ctx_set_stream(ctx.h, C.c_void_p(s.cuda_stream)), ctx.h)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            m.apply_into(x, y)
        graphs.append(g)
    for _ in range(30):
        for y in ys:
            y.zero_()
        torch.cuda.synchronize()
        for _ in range(5):
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
        for y, ref in zip(ys, alone):
            assert np.array_equal(ctx.download(y), ref)
    for m in maps:
        m.close()
    ctx.close()
