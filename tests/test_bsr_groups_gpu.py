"""f32 BSR SpMM by groups of lanes: every number of columns per lane, bit for bit the sequential sums."""
import numpy as np
import pytest
import torch

import oracle
from sparsewave_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [4, 8])
@pytest.mark.parametrize("brows,n", [(1, 8), (1, 20000), (620, 33), (600, 64), (2500, 9), (2300, 43), (1700, 54), (4200, 124), (5700, 16),
                                     (16300, 32), (19000, 32), (3650, 124), (3700, 124)])
def test_groups(ctx, bs, brows, n):
    """Empty block rows, parts of chunks, whole chunks and more; columns that fill a tile, leave lanes idle, make several tiles."""
    counts = torch.tensor([0, 1, 3, 4, 5, 8, 9, 0, 17, 2])[(torch.arange(brows) * 7 + brows) % 10]
    brp = torch.zeros(brows + 1, dtype=torch.int32)
    brp[1:] = torch.cumsum(counts, 0)
    cols = 40
    gen = torch.Generator().manual_seed(brows + n)
    bci = torch.randint(cols, (int(brp[-1]),), generator=gen, dtype=torch.int32)
    values = W.dense_normal((int(brp[-1]) * bs, bs), seed=bs).view(-1).float()
    B = W.dense_normal((cols * bs, n), seed=n).float()
    values[::7] = 0.0
    values[3::11] *= -1e-38  # products below the smallest normal number
    B[::5] = -0.0
    expected = oracle.bsr_spmm_f32(brp.numpy(), bci.numpy(), values.numpy(), B.numpy(), bs).view(np.int32)
    for off in (0, 1):  # values and B that start one element past an aligned address
        v = torch.empty(values.numel() + off, device="cuda")[off:].copy_(values)
        Bd = torch.empty(B.numel() + off, device="cuda")[off:].view(B.shape).copy_(B)
        C = ctx.bsr_spmm("", brp.cuda(), bci.cuda(), v, Bd, bs).cpu().numpy().view(np.int32)
        assert np.array_equal(C, expected)
