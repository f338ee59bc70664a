"""bf16 BSR SpMM: a block row's results are the same bits however many block rows the call has and on which of the tensor-core
kernels it runs, and its sums are no further from the exact ones than the sequential loop's where that used to run."""
import numpy as np
import pytest
import torch

import oracle

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
    """Two kinds of sums: the tensor cores' chain on aligned operands of 64 (8 x 8: 96) columns in eights and more, and sums of
    products 16 at a time added in f32."""
    brp, bci, values, B = _case(bs, brows, 60, 256, bs + brows)
    chain = _bits(ctx, brp, bci, values, B, bs)
    off = torch.empty(B.numel() + 1, dtype=B.dtype, device="cuda")[1:].view(B.shape).copy_(B)
    rounded = _bits(ctx, brp, bci, values, off, bs)
    assert torch.equal(_bits(ctx, brp, bci, torch.cat([values[:1], values])[1:], B, bs), rounded)
    for n in (1, 7, 16, 30, 56, 64, 88, 100, 128, 136, 192):
        want = chain if n % 8 == 0 and n >= (96 if bs == 8 else 64) else rounded
        assert torch.equal(_bits(ctx, brp, bci, values, B[:, :n].contiguous(), bs), want[:, :n])
    C = torch.empty(brows * bs * 256 + 1, dtype=B.dtype, device="cuda")[1:].view(brows * bs, 256)
    ctx.bsr_spmm("", brp, bci, values, B, bs, C)
    assert torch.equal(C.view(torch.int16), chain)


@pytest.mark.parametrize("bs", [8, 16, 32])
@pytest.mark.parametrize("n", [3, 32, 88, 100])
@pytest.mark.parametrize("brows", [4, 2400])
def test_sums_against_64_bits(ctx, bs, n, brows):
    """Products that cancel leave the roundings of the sums: against those of the sequential f32 loop."""
    if bs > 8 and n == 88:
        pytest.skip("the tensor cores' chain, as ever")
    for per in (4, 20, 100) if brows == 4 else (20,):
        gen = torch.Generator().manual_seed(per + n)
        order = torch.randperm(per, generator=gen)
        bci = torch.randint(40, (brows, per), generator=gen, dtype=torch.int32)
        v = torch.randn((brows, per, bs, bs), generator=gen).bfloat16()
        brp = torch.arange(0, 2 * per * brows + 1, 2 * per, dtype=torch.int32)
        bci, v = torch.cat([bci, bci[:, order]], 1).reshape(-1), torch.cat([v, -v[:, order]], 1).reshape(-1)
        B = torch.randn((40 * bs, n), generator=gen).bfloat16()
        C = ctx.bsr_spmm("", brp.cuda(), bci.cuda(), v.cuda(), B.cuda(), bs).double().cpu().numpy()
        rows = slice(0, 4 * bs)  # of the oracle: the first four block rows
        _, f32 = oracle.bsr_spmm_bf16(brp[:5].numpy(), bci[:8 * per].numpy(), v[:8 * per * bs * bs].view(torch.uint16).numpy(),
                                      B.view(torch.uint16).numpy(), bs)
        # the exact result is 0; a small sample of the loop's errors, hence the factor
        assert np.sqrt((C[rows] ** 2).mean()) <= 1.2 * np.sqrt((f32.astype(np.float64) ** 2).mean())
