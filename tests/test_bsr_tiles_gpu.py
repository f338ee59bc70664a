"""BSR thread-per-output kernel: tiles of rows and columns per thread, bit-exact in f32, the oracle's bits in bf16 (of which blocks
of 8 and 16 run on warp-level MMAs)."""
import numpy as np
import pytest
import torch

import oracle
from sparsewave_b200 import workloads as W
from tests.helpers import assert_bf16_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 8, 9, 16, 20, 33])
@pytest.mark.parametrize("n", [1, 2, 6, 7, 64])
def test_row_tiles(ctx, bs, n):
    rows, cols = (40, 23) if n < 64 else (400, 23)  # few threads: narrow columns; many: the widest
    for dtype in (torch.float32, torch.bfloat16):
        if bs == 16 and n % 8 == 0 and dtype == torch.bfloat16:
            continue  # aligned operands of the tensor-core kernels have tests of their own
        a = W.random_bsr(rows, cols, bs, 0.2, seed=bs * 100 + n, dtype=dtype)
        B = W.dense_normal((cols * bs, n), seed=n, dtype=dtype)
        h = (a.block_row_ptr.numpy(), a.block_col_idx.numpy())
        for off in (0, 1):  # values and B that start one element past an aligned address
            bv = torch.empty(a.block_values.numel() + off, dtype=dtype, device="cuda")[off:].copy_(a.block_values)
            Bd = torch.empty(B.numel() + off, dtype=dtype, device="cuda")[off:].view(B.shape).copy_(B)
            C = ctx.bsr_spmm("", a.block_row_ptr.cuda(), a.block_col_idx.cuda(), bv, Bd, bs)
            if dtype == torch.float32:
                assert np.array_equal(C.cpu().numpy(), oracle.bsr_spmm_f32(*h, a.block_values.numpy(), B.numpy(), bs))
            else:
                assert_bf16_close(C, *h, a.block_values.view(torch.uint16).numpy(), B.view(torch.uint16).numpy(), bs)
