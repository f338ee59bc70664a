"""wave-per-row-tile on few rows, N a power of two: more lanes per row, against the oracle."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,mean,n", [(2700, 16, 32), (6200, 30, 32), (6300, 3, 16), (12000, 5, 16), (3000, 40, 8), (50001, 3, 8),
                                         (5000, 3, 4), (3100, 9, 64)])
def test_few_rows(ctx, rows, mean, n):
    rng = np.random.default_rng(rows + n)
    lens = np.minimum(rng.geometric(1 / (mean + 1), rows) - 1, 900)
    lens[7] = 900
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 1200, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (1200, n)).astype(np.float32)
    want, bound = oracle.csr_spmm(rp, ci, v, B, parallel=True), oracle.csr_abs_bound(rp, ci, v, B)
    a = [torch.from_numpy(t).cuda() for t in (rp, ci, v, B)]
    options = "spmm-mapping=wave-per-row-tile spmm-tile-size=8 spmm-block-size=256"
    C = ctx.spmm(options, *a)
    assert np.all(np.abs(C.cpu().numpy() - want) <= 900 * 2**-23 * bound + 1e-30)  # either order of up to 900 terms
    C = torch.ones((rows, n), device="cuda")
    ctx.spmm(options + " accumulate=1", *a, C)
    assert np.all(np.abs(C.cpu().numpy() - want - 1) <= 901 * 2**-23 * (bound + 1))
