"""FP64 steps with K <= 64 on either side of the rule that takes them off the small-K kernel
(more than 512 entries of the static, or little work) run in place instead."""
import numpy as np
import pytest

from grafttn import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [30, 2000, 30000])
@pytest.mark.parametrize("K", [15, 16, 17, 64])
@pytest.mark.parametrize("N", [32, 33, 48])
@pytest.mark.parametrize("prec", ["fp64", "fp64e"])
def test_either_side(ctx, M, K, N, prec):
    rng = np.random.default_rng(M + K + N)
    A = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    B = rng.standard_normal((K, N)) + 1j * rng.standard_normal((K, N))
    y = ctx.download(ctx.contract([ctx.upload(A), ctx.upload(B)], [[-1, 1], [1, -2]], None, None,
                                  _lib.PRECISIONS[prec]))
    # 2K fused multiply-adds a part, or seven signed base-256 digits of either row: 2^-50 at least
    bound = (2 * (2 * K + 2) * 2.0 ** -53 + 2.0 ** -48) * np.sqrt(2)
    scale = np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=0)[None, :] * K
    assert np.all(np.abs(y - A @ B) <= bound * scale)
