"""FP64 contractions with no room for their digit planes run on the FP64 pipe."""
import numpy as np
import pytest
import torch

from grafttn import _lib
from grafttn.device import Context

pytestmark = pytest.mark.gpu


def test_one_shot_contraction_beside_a_full_device():
    M, K, N = 1 << 18, 512, 64
    torch.cuda.empty_cache()
    ctx = Context(0)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)

    def randn(shape):
        return torch.view_as_complex(torch.randn(shape + (2,), generator=g, device="cuda", dtype=torch.float64))
    A, B, out = randn((M, K)), randn((K, N)), ctx.empty((M, N))
    del out  # torch keeps the block for the result
    torch.cuda.synchronize()
    # two running tensors and a K-major copy of 16 bytes an element, as an FP64 contraction with a staged
    # operand takes, fit; the digit planes, 28 bytes an element, do not
    need = 2 * 16 * M * K + 16 * M * K + (1 << 29)
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(max(0, free - need), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):  # the second call finds the context's arena refused
            y = ctx.contract([A, B], [[-1, 1], [1, -2]], None, None, _lib.PRECISIONS["fp64"])
            ctx.sync()
            rows = [0, 1, 127, 128, M // 3, M - 1]
            a, b, got = ctx.download(A[rows]), ctx.download(B), ctx.download(y[rows])
            del y
            tol = 2 * (2 * K + 4) * 2.0 ** -53 * np.sqrt(2) * (np.abs(a) @ np.abs(b))
            assert np.all(np.abs(got - a @ b) <= tol)
    finally:
        del fill, A, B
        ctx.close()
        torch.cuda.empty_cache()
