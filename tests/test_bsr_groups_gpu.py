"""f32 BSR SpMM by groups of lanes: every number of columns per lane, bit for bit the sequential sums."""
import numpy as np
import pytest
import torch

import oracle
from sparsewave_b200 import workloads as W
from tests.helpers import launched

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


@pytest.mark.parametrize("bs,n", [(4, 128), (8, 64)])
def test_b_of_four_gib_and_more(ctx, bs, n):
    """Whole numbers, so that every sum is exact: block columns on both sides of 4 GiB, aligned values and B."""
    cols, brows = (1 << 30) // (bs * n) + 100, 2400
    gen = torch.Generator("cuda").manual_seed(bs)
    B = torch.empty((cols * bs, n), device="cuda").random_(-8, 9, generator=gen)
    brp = torch.arange(0, 3 * brows + 1, 3, dtype=torch.int32, device="cuda")
    bci = torch.randint(cols, (brows, 3), generator=gen, dtype=torch.int32, device="cuda")
    bci[:, 2] = cols - 1 - torch.arange(brows, device="cuda", dtype=torch.int32) % 90
    values = torch.randint(-8, 9, (brows, 3, bs, bs), generator=gen, device="cuda").float()
    C, names = launched(lambda: ctx.bsr_spmm("", brp, bci.reshape(-1), values.reshape(-1), B, bs))
    if names is not None:
        assert len(names) == 1 and names[0].startswith(f"bsr_spmm_row_group_kernel<{bs}, ") and names[0].endswith("true, unsigned long>")
    slabs = B.view(cols, bs, n)[bci.long()]
    want = torch.einsum("bprk,bpkn->brn", values.double(), slabs.double()).float()
    assert torch.equal(C.view(brows, bs, n), want)
