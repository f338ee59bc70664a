"""The tcgen05 kernel of BSR SpMM in each of its instantiations (block size, tiles of 128 or 256 columns, status word per call or
per unit), by kernel name: the other tensor-core kernel takes small calls, so that a size alone does not say which one ran."""
import pytest
import torch

from sparsewave_b200 import api, workloads as W
from tests.helpers import assert_bf16_close, launched

pytestmark = pytest.mark.gpu

# block size, 128-column accumulators per tile, block rows, columns
INSTANTIATIONS = [(8, 1, 310, 128), (8, 2, 930, 256), (16, 1, 310, 128), (16, 1, 170, 320), (16, 2, 930, 256), (16, 2, 640, 488),
                  (32, 1, 310, 128), (32, 1, 90, 112), (32, 2, 1500, 512)]


def _ran(names, kernel):
    if names is not None:
        assert names == [kernel]


@pytest.mark.parametrize("bs,halves,brows,n", INSTANTIATIONS)
def test_values_of_other_block_rows_do_not_leak(ctx, bs, halves, brows, n):
    """NaN among the blocks of some block rows, infinities in a slab of B that some others read: neither reaches any other block
    row, through what a stage, an accumulator or the padding held before."""
    row = torch.arange(brows)
    counts = torch.tensor([0, 1, 41, 3, 64, 2, 0, 64, 4, 57, 1])[row % 11]
    brp = torch.zeros(brows + 1, dtype=torch.int32)
    brp[1:] = torch.cumsum(counts, 0)
    of_block = torch.repeat_interleave(row, counts)
    cols = 30
    gen = torch.Generator().manual_seed(brows)
    bci = torch.randint(cols - 1, (len(of_block),), generator=gen, dtype=torch.int32)
    infinite = (row % 7 == 3) & (counts > 0)
    bci[brp[1:][infinite].long() - 1] = cols - 1  # the row's last block
    poisoned = (row % 5 == 1) & (counts > 0)
    values = torch.ones((len(of_block), bs * bs), dtype=torch.bfloat16)
    values[poisoned[of_block]] = float("nan")
    B = torch.ones((cols * bs, n), dtype=torch.bfloat16)
    B[-bs:] = float("inf")
    operands = brp.cuda(), bci.cuda(), values.reshape(-1).cuda(), B.cuda()
    C, names = launched(lambda: ctx.bsr_spmm("", *operands, bs))
    _ran(names, f"bsr_spmm_tcgen05_kernel<false, {bs}, {halves}>")
    assert ctx.device_status() == 0
    want = (counts * bs).float()  # whole numbers of at most eight bits times a power of two
    want[infinite] = float("inf")
    want[poisoned] = float("nan")
    want = want.repeat_interleave(bs)[:, None].expand(-1, n)
    assert torch.equal(C.cpu().float().nan_to_num(-1.0, 1e30), want.nan_to_num(-1.0, 1e30))


@pytest.mark.parametrize("bs,halves,brows,n", INSTANTIATIONS)
@pytest.mark.parametrize("graph", [False, True])
def test_chain(ctx, bs, halves, brows, n, graph):
    """Products whose operand is the result of the one before, in two buffers that take turns, without a synchronisation: block
    rows exchanged and their rows turned, by a permutation among blocks of zeros."""
    gen = torch.Generator().manual_seed(brows + bs)
    per = 24
    brp = torch.arange(0, per * brows + 1, per, dtype=torch.int32, device="cuda")
    perm = torch.randperm(brows, generator=gen)
    bci = torch.randint(brows, (brows, per), generator=gen, dtype=torch.int32)
    values = torch.zeros((brows, per, bs, bs), dtype=torch.bfloat16)
    at = torch.randint(per, (brows,), generator=gen)
    bci[torch.arange(brows), at] = perm.int()
    values[torch.arange(brows), at] = torch.roll(torch.eye(bs), 1, 1).bfloat16()
    matrix = brp, bci.reshape(-1).cuda(), values.reshape(-1).cuda()
    B0 = torch.randint(-200, 201, (brows * bs, n), generator=gen).bfloat16().cuda()
    a, b = torch.empty_like(B0), torch.empty_like(B0)
    _ran(launched(lambda: ctx.bsr_spmm("", *matrix, B0, bs, a))[1], f"bsr_spmm_tcgen05_kernel<false, {bs}, {halves}>")

    def chain():
        a.copy_(B0)
        x, y = a, b
        for _ in range(12):
            ctx.bsr_spmm("", *matrix, x, bs, y)
            x, y = y, x
        return x

    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = chain()
        g.replay()
    else:
        got = chain()
    want = B0.view(brows, bs, n)
    for _ in range(12):
        want = want[perm.cuda()].roll(-1, 1)
    assert torch.equal(got.view(brows, bs, n), want)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("bs,brows,n,team", [(8, 40, 24, True), (16, 40, 24, True), (32, 40, 24, True), (8, 2500, 24, False),
                                             (16, 2500, 24, False), (32, 2500, 24, False)])
def test_chain_of_the_other_kernel(ctx, bs, brows, n, team):
    perm = torch.randperm(brows, generator=torch.Generator().manual_seed(brows))
    brp = torch.arange(0, 9 * brows + 1, 9, dtype=torch.int32, device="cuda")
    bci = torch.randint(brows, (brows, 9), generator=torch.Generator().manual_seed(bs), dtype=torch.int32)
    bci[:, 8] = perm.int()
    values = torch.zeros((brows, 9, bs, bs), dtype=torch.bfloat16)
    values[:, 8] = torch.roll(torch.eye(bs), 1, 1).bfloat16()
    matrix = brp, bci.reshape(-1).cuda(), values.reshape(-1).cuda()
    B0 = torch.randint(-200, 201, (brows * bs, n)).bfloat16().cuda()
    x, y = B0.clone(), torch.empty_like(B0)
    names = launched(lambda: ctx.bsr_spmm("", *matrix, B0, bs, y))[1]
    if names is not None:
        arguments = names[0].split("<")[1].rstrip(">").split(", ")  # block size, ..., several warps per block row, sums
        assert len(names) == 1 and names[0].startswith(f"bsr_spmm_mma_kernel<{bs}, ") and (arguments[4] == "true") == team
    for _ in range(12):
        ctx.bsr_spmm("", *matrix, x, bs, y)
        x, y = y, x
    want = B0.view(brows, bs, n)
    for _ in range(12):
        want = want[perm.cuda()].roll(-1, 1)
    assert torch.equal(x.view(brows, bs, n), want)


@pytest.mark.parametrize("sizes", [[(200, 256), (100, 200)], [(310, 128), (160, 488), (2400, 256)]])
def test_static_entry_point(ctx, sizes):
    """A status word per unit: the bits of the context's call, on calls in a row that share the words."""
    for brows, n in sizes:
        a = W.random_bsr(brows, 60, 16, 0.3, seed=brows, device="cuda")
        B = W.dense_normal((60 * 16, n), seed=n, device="cuda")
        want = ctx.bsr_spmm("", a.block_row_ptr, a.block_col_idx, a.block_values, B, 16)
        got, names = launched(lambda: api.bsr16_spmm_bf16_static(a.block_row_ptr, a.block_col_idx, a.block_values, B))
        _ran(names, "bsr_spmm_tcgen05_kernel<true, 16, 2>")
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
        out = torch.empty_like(want)
        api.bsr16_spmm_bf16_static(a.block_row_ptr, a.block_col_idx, a.block_values, B, out, wait=False)
        assert api.bsr16_static_status() == 0
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("bs,per_sm,per,n,here", [(32, 1, 5, 64, True), (32, 0.99, 5, 96, False), (32, 0.05, 5, 104, True), (16, 1, 1, 128, True),
                                                  (16, 0.99, 9, 128, False), (16, 1, 8, 72, True), (16, 1, 7, 120, False),
                                                  (16, 2, 12, 64, True), (16, 1.99, 12, 64, False), (16, 2, 11, 64, False),
                                                  (16, 1, 12, 136, True), (16, 1, 11, 136, False), (16, 1, 8, 144, True),
                                                  (16, 3, 30, 56, False), (8, 1, 20, 128, True), (8, 1, 19, 128, False),
                                                  (8, 4, 8, 256, True), (8, 3.99, 8, 256, False), (8, 9, 8, 384, False), (8, 1, 20, 136, False),
                                                  (16, 1, 6, 208, True), (16, 1, 5, 208, False), (16, 1, 6, 192 + 8, False),
                                                  (8, 2, 12, 448, True), (8, 2, 11, 448, False), (8, 1.99, 12, 448, False),
                                                  (8, 4, 27, 208, True), (8, 4, 26, 208, False), (8, 3.99, 27, 208, False)])
def test_line_between_the_kernels(ctx, bs, per_sm, per, n, here):
    """Both sides of each limit: block rows per SM, blocks per block row and columns."""
    brows = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count)
    gen = torch.Generator().manual_seed(brows + n)
    cols = 40
    brp = torch.arange(0, per * brows + 1, per, dtype=torch.int32)
    bci = torch.randint(cols, (per * brows,), generator=gen, dtype=torch.int32)
    values, B = W.dense_normal((per * brows * bs, bs), seed=bs).view(-1), W.dense_normal((cols * bs, n), seed=n)
    C, names = launched(lambda: ctx.bsr_spmm("", brp.cuda(), bci.cuda(), values.cuda(), B.cuda(), bs))
    if names is not None:
        assert len(names) == 1 and names[0].startswith("bsr_spmm_tcgen05_kernel" if here else "bsr_spmm_mma_kernel")
    assert ctx.device_status() == 0
    assert_bf16_close(C, brp.numpy(), bci.numpy(), values.view(torch.uint16).numpy(), B.view(torch.uint16).numpy(), bs)


@pytest.mark.parametrize("bs,cols,per,here", [(16, 2605, 4, True), (16, 2604, 4, False), (8, 6741, 8, True), (8, 6740, 8, False),
                                              (8, 5515, 9, True), (8, 5514, 9, False)])
def test_line_by_the_size_of_b(ctx, bs, cols, per, here):
    brows, n = 160, 408
    gen = torch.Generator().manual_seed(cols)
    brp = torch.arange(0, per * brows + 1, per, dtype=torch.int32)
    bci = torch.randint(cols, (per * brows,), generator=gen, dtype=torch.int32)
    values, B = W.dense_normal((per * brows * bs, bs), seed=bs).view(-1), W.dense_normal((cols * bs, n), seed=n)
    C, names = launched(lambda: ctx.bsr_spmm("", brp.cuda(), bci.cuda(), values.cuda(), B.cuda(), bs))
    if names is not None:
        assert len(names) == 1 and names[0].startswith("bsr_spmm_tcgen05_kernel" if here else "bsr_spmm_mma_kernel")
    assert_bf16_close(C, brp.numpy(), bci.numpy(), values.view(torch.uint16).numpy(), B.view(torch.uint16).numpy(), bs)
