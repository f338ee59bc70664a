"""BSR SpMM with warp-level MMAs: column counts around the widths of a warp's tile and of a load, views that start off an
aligned address, few block rows (shared out among warps) and many, odd block counts, empty block rows."""
import pytest
import torch

from sparsewave_b200 import workloads as W
from tests.helpers import assert_bf16_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [8, 16, 32])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 16, 17, 18, 31, 32, 36, 64, 66, 72, 95, 132])
@pytest.mark.parametrize("rows,density", [(1, 1.0), (40, 0.12), (3, 0.97), (600, 0.1)])
def test_shapes(ctx, bs, n, rows, density):
    a = W.random_bsr(rows, 70, bs, density, seed=bs + n + rows)
    B = W.dense_normal((70 * bs, n), seed=n)
    h = (a.block_row_ptr.numpy(), a.block_col_idx.numpy(), a.block_values.view(torch.uint16).numpy(),
         B.view(torch.uint16).numpy())
    for values_off, B_off in ((0, 0), (1, 0), (4, 2)):  # elements past an aligned address
        bv = torch.empty(a.block_values.numel() + values_off, dtype=torch.bfloat16, device="cuda")[values_off:].copy_(a.block_values)
        Bd = torch.empty(B.numel() + B_off, dtype=torch.bfloat16, device="cuda")[B_off:].view(B.shape).copy_(B)
        C = torch.full((rows * bs + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")  # the last row is not the call's
        ctx.bsr_spmm("", a.block_row_ptr.cuda(), a.block_col_idx.cuda(), bv, Bd, bs, C[:rows * bs])
        assert bool((C[rows * bs:] == 7.0).all())
        assert_bf16_close(C[:rows * bs], *h, bs)


@pytest.mark.parametrize("n", [9, 16, 40, 75])
@pytest.mark.parametrize("copies", [1, 14, 31, 66, 140])
def test_segments_of_32_x_32_blocks(ctx, n, copies):
    """Block rows around the lengths at which segments grow and block columns no longer fit a warp, by teams of eight warps down to
    one per block row: the oracle's results, and the same bits however often the block rows are repeated."""
    counts = torch.tensor([0, 1, 2, 15, 16, 17, 31, 32, 33, 64, 65])
    gen = torch.Generator().manual_seed(n)
    nnzb, cols = int(counts.sum()), 40
    brp = torch.zeros(len(counts) + 1, dtype=torch.int32)
    brp[1:] = torch.cumsum(counts, 0)
    bci = torch.randint(cols, (nnzb,), generator=gen, dtype=torch.int32)
    values = torch.randn((nnzb, 32, 32), generator=gen).bfloat16()
    B = torch.randn((cols * 32, n), generator=gen).bfloat16()
    many = torch.cat([torch.zeros(1, dtype=torch.int32), torch.cumsum(counts.repeat(copies), 0).int()])
    C = ctx.bsr_spmm("", many.cuda(), bci.repeat(copies).cuda(), values.repeat(copies, 1, 1).view(-1).cuda(), B.cuda(), 32)
    C = C.view(copies, len(counts) * 32, n)
    assert_bf16_close(C[0], brp.numpy(), bci.numpy(), values.view(-1).view(torch.uint16).numpy(), B.view(torch.uint16).numpy(), 32)
    assert torch.equal(C.view(torch.int16), C[:1].view(torch.int16).expand_as(C))
    few = ctx.bsr_spmm("", brp.cuda(), bci.cuda(), values.view(-1).cuda(), B.cuda(), 32)
    assert torch.equal(few.view(torch.int16), C[0].view(torch.int16))
