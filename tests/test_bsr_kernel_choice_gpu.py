"""bf16 BSR SpMM of sizes with short, long and ragged last tiles of columns on both tensor-core kernels, against the oracle (the line
between the two, by kernel name: test_bsr_tcgen05_gpu.py)."""
import pytest
import torch

from sparsewave_b200 import workloads as W
from tests.helpers import assert_bf16_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs,brows,per,n", [(16, 599, 9, 80), (16, 600, 8, 96), (16, 610, 7, 112), (16, 600, 9, 104), (16, 1000, 30, 72),
                                            (16, 300, 9, 160), (16, 300, 9, 168), (16, 1334, 9, 264), (16, 200, 8, 296), (16, 3000, 16, 136),
                                            (8, 1500, 6, 128), (8, 750, 5, 192), (8, 1499, 6, 128),
                                            (8, 450, 24, 128), (8, 500, 5, 320), (16, 150, 16, 128), (16, 75, 17, 256), (16, 175, 5, 512),
                                            (32, 84, 9, 264), (32, 400, 16, 72), (32, 400, 5, 72)])
def test_both_sides(ctx, bs, brows, per, n):
    cols = 40
    gen = torch.Generator().manual_seed(brows + n)
    counts = torch.randint(0, 2 * per + 1, (brows,), generator=gen)
    counts[0] += max(0, per * brows - int(counts.sum()))
    brp = torch.zeros(brows + 1, dtype=torch.int32)
    brp[1:] = torch.cumsum(counts, 0)
    bci = torch.randint(cols, (int(brp[-1]),), generator=gen, dtype=torch.int32)
    values = W.dense_normal((int(brp[-1]) * bs, bs), seed=bs).view(-1)
    B = W.dense_normal((cols * bs, n), seed=n)
    C = ctx.bsr_spmm("", brp.cuda(), bci.cuda(), values.cuda(), B.cuda(), bs)
    assert ctx.device_status() == 0
    assert_bf16_close(C, brp.numpy(), bci.numpy(), values.view(torch.uint16).numpy(), B.view(torch.uint16).numpy(), bs)
