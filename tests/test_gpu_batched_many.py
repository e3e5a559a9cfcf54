"""More maps in a batch than one grouped launch takes (64 tensor-core problems, 128 table-driven
gathers): the last map of a launch, the first of the next and every other match the single
application, with rows and columns at the edges of the gather tiles (64 x 32, 128 x 16)."""
import numpy as np
import pytest

from grafttn.contractions import EffectiveMap, apply_batched
from oracle import ttn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16x6", "fp16x3"])
def test_131_maps(ctx, prec):
    rng = np.random.default_rng(7)
    labels, order = O.h1_spec(O.mps_topology(3), 1, 3, 4)
    maps, xs = [], []
    for i in range(131):
        a, b = 20 + i % 14, 31 + i % 5
        statics = [O.randn_c(rng, (5, 2, 2, 5)), O.randn_c(rng, (a, 5, a)), O.randn_c(rng, (b, 5, b))]
        maps.append(EffectiveMap(ctx, (a, 2, b), labels, order, [ctx.upload(s) for s in statics], prec))
        xs.append(ctx.upload(O.randn_c(rng, (a, 2, b))))
    for m, x, y in zip(maps, xs, apply_batched(maps, xs)):
        y, ref = ctx.download(y), ctx.download(m(x))
        assert np.linalg.norm(y - ref) <= 1e-6 * np.linalg.norm(ref)  # as for the uneven batches
    for m in maps:
        m.close()
