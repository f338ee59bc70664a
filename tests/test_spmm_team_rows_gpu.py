"""wave-per-row-tile on few rows: teams of one, two and four warps per row against the oracle."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
OPTIONS = "spmm-mapping=wave-per-row-tile spmm-tile-size=32 spmm-block-size=256"


@pytest.mark.parametrize("rows,mean,n,tiles,warps", [
    (1024, 5, 5, 1, 1), (1100, 12, 19, 1, 4), (2400, 12, 33, 2, 2), (6001, 7, 9, 1, 1), (1025, 12, 511, 16, 1),
    (1100, 40, 29, 1, 4),  # a column per lane
    (1100, 30, 2, 1, 1), (1100, 40, 62, 1, 4), (3000, 31, 130, 3, 2), (8192, 3, 22, 1, 1),  # two
    (4736, 28, 40, 1, 4), (3500, 40, 12, 1, 2), (1024, 6, 68, 1, 4),  # four
    (3001, 26, 36, 1, 4), (4100, 60, 28, 1, 4)])  # two warps per row in blocks of half the size: the grid of four
def test_few_rows(ctx, rows, mean, n, tiles, warps):
    rng = np.random.default_rng(rows + n)
    lens = np.minimum(rng.geometric(1 / (mean + 1), rows) - 1, 900)
    lens[7] = 900
    lens[100:100 + max(0, mean * rows - lens.sum())] += 1  # no mean below the one named
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 1200, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (1200, n)).astype(np.float32)
    want, bound = oracle.csr_spmm(rp, ci, v, B, parallel=True), oracle.csr_abs_bound(rp, ci, v, B)
    assert ctx.launch_shape(OPTIONS, rows, int(rp[-1]), n).physical_grid == -(-rows * tiles // (8 // warps))
    a = [torch.from_numpy(t).cuda() for t in (rp, ci, v)]
    for off in (0, 1, 2):  # B that starts at an address aligned to 16, 4 and 8 bytes
        Bd = torch.empty(B.size + off, device="cuda")[off:].view(B.shape).copy_(torch.from_numpy(B))
        C = ctx.spmm(OPTIONS, *a, Bd)
        assert np.all(np.abs(C.cpu().numpy() - want) <= 900 * 2**-23 * bound + 1e-30)  # either order of up to 900 terms
    C = torch.ones((rows, n), device="cuda")
    ctx.spmm(OPTIONS + " accumulate=1", *a, torch.from_numpy(B).cuda(), C)
    assert np.all(np.abs(C.cpu().numpy() - want - 1) <= 901 * 2**-23 * (bound + 1))


@pytest.mark.parametrize("rows,mean,n,tiles,warps", [
    (2500, 5, 19, 1, 2), (6001, 7, 9, 1, 1), (1025, 2, 511, 16, 1),  # one column per lane
    (2500, 6, 50, 1, 2), (5000, 12, 50, 1, 2), (3000, 31, 130, 3, 2),  # two
    (5000, 3, 12, 1, 1), (2500, 26, 100, 1, 4), (3500, 40, 12, 1, 2), (3001, 26, 36, 1, 4)])  # four, the last in small blocks
def test_rows_far_longer_than_the_others(ctx, rows, mean, n, tiles, warps):
    """A whole block takes them: alone and several in a share of 128 rows, in the first and the last one."""
    rng = np.random.default_rng(rows + n)
    lens = np.minimum(rng.geometric(1 / (mean + 1), rows) - 1, 10 * mean)
    lens[[0, 3, 126, 400, rows - 1]] = 2500, 0, 3100, 5003, 2777
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 1200, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (1200, n)).astype(np.float32)
    want, bound = oracle.csr_spmm(rp, ci, v, B, parallel=True), oracle.csr_abs_bound(rp, ci, v, B)
    assert ctx.launch_shape(OPTIONS, rows, int(rp[-1]), n).physical_grid == -(-rows * tiles // (8 // warps))
    a = [torch.from_numpy(t).cuda() for t in (rp, ci, v, B)]
    C = ctx.spmm(OPTIONS, *a)
    assert np.all(np.abs(C.cpu().numpy() - want) <= 5003 * 2**-23 * bound + 1e-30)  # either order of up to 5,003 terms
    C = torch.ones((rows, n), device="cuda")
    ctx.spmm(OPTIONS + " accumulate=1", *a, C)
    assert np.all(np.abs(C.cpu().numpy() - want - 1) <= 5004 * 2**-23 * (bound + 1))
