"""BSR SpMM on the tensor cores for blocks of 8 x 8 (two per step), 16 x 16 and 32 x 32, in whichever of the two kernels the sizes
lead to (few block rows: warp-level MMAs; the tcgen05 kernel by name: test_bsr_tcgen05_gpu.py)."""
import pytest
import torch

from sparsewave_b200 import workloads as W
from tests.helpers import assert_bf16_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [8, 16, 32])
@pytest.mark.parametrize("n", [8, 64, 72, 96, 128, 136, 256, 264, 520])
@pytest.mark.parametrize("rows,density", [(1, 1.0), (40, 0.12), (3, 0.9), (700, 0.2)])
def test_shapes(ctx, bs, n, rows, density):
    """Empty block rows, odd and even block counts, fewer and more steps than stages, one and two halves of a tile, few and
    many CTAs per SM."""
    if rows == 700 and (n > 136 or bs == 32):
        pytest.skip("covered by the smaller sizes")
    a = W.random_bsr(rows, 37, bs, density, seed=bs + n + rows)
    B = W.dense_normal((37 * bs, n), seed=n)
    C = ctx.bsr_spmm("", a.block_row_ptr.cuda(), a.block_col_idx.cuda(), a.block_values.cuda(), B.cuda(), bs)
    assert ctx.device_status() == 0
    assert_bf16_close(C, a.block_row_ptr.numpy(), a.block_col_idx.numpy(), a.block_values.view(torch.uint16).numpy(),
                      B.view(torch.uint16).numpy(), bs)


@pytest.mark.parametrize("bs", [8, 16, 32])
def test_values_of_other_block_rows_do_not_leak(ctx, bs):
    brp = torch.tensor([0, 1, 4, 7, 9], dtype=torch.int32)  # odd counts before, at and after the poisoned row
    bci = torch.tensor([2, 0, 1, 2, 0, 1, 2, 0, 3], dtype=torch.int32)
    values = torch.ones(9 * bs * bs, dtype=torch.bfloat16)
    values[4 * bs * bs:7 * bs * bs] = float("nan")
    B = torch.ones((4 * bs, 128), dtype=torch.bfloat16)
    B[3 * bs:] = float("inf")
    C = ctx.bsr_spmm("", brp.cuda(), bci.cuda(), values.cuda(), B.cuda(), bs).float().cpu()
    assert torch.equal(C[:bs], torch.full((bs, 128), float(bs))) and torch.equal(C[bs:2 * bs], torch.full((bs, 128), 3.0 * bs))
    assert bool(C[2 * bs:3 * bs].isnan().all()) and bool(C[3 * bs:].isinf().all())


@pytest.mark.parametrize("bs,rows,n", [(16, 3, 128), (16, 1900, 128), (16, 1000, 320), (16, 700, 232), (16, 1300, 512),
                                       (32, 450, 64), (32, 1500, 72), (32, 300, 200), (8, 2100, 256), (8, 4400, 440), (32, 1600, 192), (32, 2100, 256)])
def test_several_units_per_cta(ctx, bs, rows, n):
    """Persistent CTAs: one to nine units each, with empty block rows, whole and partial groups, and both tile widths."""
    counts = torch.tensor([0, 1, 2, 3, 4, 5, 9, 0, 16, 35])[torch.arange(rows) % 10]
    brp = torch.zeros(rows + 1, dtype=torch.int32)
    brp[1:] = torch.cumsum(counts, 0)
    cols = 37
    bci = torch.cat([torch.randperm(cols, generator=torch.Generator().manual_seed(i))[:c].sort()[0] for i, c in enumerate(counts)])
    values = W.dense_normal((int(brp[-1]) * bs, bs), seed=bs).view(-1)
    B = W.dense_normal((cols * bs, n), seed=n)
    C = ctx.bsr_spmm("", brp.cuda(), bci.int().cuda(), values.cuda(), B.cuda(), bs)
    assert ctx.device_status() == 0
    assert_bf16_close(C, brp.numpy(), bci.int().numpy(), values.view(torch.uint16).numpy(), B.view(torch.uint16).numpy(), bs)
