"""bf16 BSR SpMM: a block row's results are the same bits however many block rows and columns the call has, on which of the
tensor-core kernels it runs, and where its operands start."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(bs, brows, cols, n, seed):
    """Blocks that nearly cancel in pairs, so that the results are the roundings of the sums."""
    gen = torch.Generator().manual_seed(seed)
    counts = torch.tensor([0, 1, 2, 5, 16, 33, 51, 78])[torch.randint(8, (brows,), generator=gen)]
    brp = torch.zeros(brows + 1, dtype=torch.int32)
    brp[1:] = torch.cumsum(counts, 0)
    nnzb = int(brp[-1])
    bci = torch.randint(cols, (nnzb,), generator=gen, dtype=torch.int32)
    values = torch.randn((nnzb, bs, bs), generator=gen) * torch.exp(torch.randn((nnzb, bs, bs), generator=gen))
    pair = 2 * torch.arange(nnzb // 2)
    values[pair + 1], bci[pair + 1] = -values[pair], bci[pair]
    B = torch.randn((cols * bs, n), generator=gen)
    return brp.cuda(), bci.cuda(), values.bfloat16().reshape(-1).cuda(), B.bfloat16().cuda()


def _bits(ctx, brp, bci, values, B, bs):
    C = ctx.bsr_spmm("", brp, bci, values, B, bs)
    assert ctx.device_status() == 0
    return C.view(torch.int16)


@pytest.mark.parametrize("bs", [8, 16, 32])
@pytest.mark.parametrize("n", [3, 8, 16, 32, 56, 64, 128, 200, 256])
def test_rows_of_a_larger_matrix(ctx, bs, n):
    brows = 3000
    brp, bci, values, B = _case(bs, brows, 60, n, bs + n)
    whole = _bits(ctx, brp, bci, values, B, bs)
    assert bool((whole != 0).any())
    for lo, hi in ((0, 1), (7, 47), (1500, 1900), (0, 1500)):
        p0, p1 = int(brp[lo]), int(brp[hi])
        part = _bits(ctx, (brp[lo:hi + 1] - p0).contiguous(), bci[p0:p1].contiguous(),
                     values[p0 * bs * bs:p1 * bs * bs].clone(), B, bs)
        assert torch.equal(part, whole[lo * bs:hi * bs])


@pytest.mark.parametrize("bs", [8, 16, 32])
@pytest.mark.parametrize("brows", [40, 2500])
def test_columns_of_a_wider_matrix(ctx, bs, brows):
    brp, bci, values, B = _case(bs, brows, 60, 256, bs + brows)
    whole = _bits(ctx, brp, bci, values, B, bs)
    for n in (1, 7, 16, 30, 56, 64, 88, 128, 136, 192):
        assert torch.equal(_bits(ctx, brp, bci, values, B[:, :n].contiguous(), bs), whole[:, :n])
    off = torch.empty(B.numel() + 1, dtype=B.dtype, device="cuda")[1:].view(B.shape).copy_(B)
    assert torch.equal(_bits(ctx, brp, bci, torch.cat([values[:1], values])[1:], off, bs), whole)
