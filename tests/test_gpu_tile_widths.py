"""The persistent tcgen05 kernel cuts a problem's 2N real columns into tiles of equal width
(multiples of 16).  Every element is the sum of the same products in the same order as in
the kernel with one CTA per tile of fixed width, so the outputs are the same bits."""
import numpy as np
import pytest

from grafttn import _lib

pytestmark = pytest.mark.gpu


# (N, fixed, persistent): 2N just above one and two tiles (one column pair in a last tile of
# fixed width), widths that are odd multiples of 16 (uneven halves for the two warps of a
# lane quarter: 144, 80, 112), one that equals the full tile, and 2N below 16 in the last pair
@pytest.mark.parametrize("N,fixed,persistent", [
    (65, "ps128", "persist128"), (129, "ps256", "persist128"), (129, "ps256", "persist256"),
    (140, "ps256", "persist256"), (76, "ps256", "persist256"), (168, "ps256", "persist128"),
    (256, "ps256", "persist256"), (333, "ps256", "persist256"), (55, "ps128", "persist128")])
@pytest.mark.parametrize("prec", ["fp16x3", "bf16x6"])
def test_equal_tile_widths_same_bits(ctx, N, fixed, persistent, prec):
    M, K = 301, 70
    rng = np.random.default_rng(N)
    A = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    B = rng.standard_normal((K, N)) + 1j * rng.standard_normal((K, N))
    old = _lib.tc_tuning(None)
    try:
        out = []
        for v in (fixed, persistent):
            _lib.tc_tuning(v)
            out.append(ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[-1, 1], [1, -2]], None, None,
                                                 _lib.PRECISIONS[prec])))
    finally:
        _lib.tc_tuning(old, clear=True)
    assert np.array_equal(out[0], out[1])
