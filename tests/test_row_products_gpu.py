"""thread-per-row SpMV: products formed by the block in position order, rows summed sequentially (bit-exact)."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import dev

pytestmark = pytest.mark.gpu


# tiles hold 4096 or 2048 products, blocks 16 to 512 or 128 rows
@pytest.mark.parametrize("lens", [[1], [0, 0, 4096], [4095, 1, 4097, 0, 3], [5000] * 3 + [0] * 300 + [1] * 300, [32] * 1000,
                                  [0] * 257, [20000, 1, 20000], [2047, 1, 2048, 2049] * 600, [1, 0, 5] * 110000])
def test_row_sums_are_sequential_across_tiles(ctx, lens):
    rng = np.random.default_rng(len(lens))
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cols = 777
    ci = rng.integers(0, cols, rp[-1]).astype(np.int32)
    v, x = rng.uniform(-1, 1, rp[-1]).astype(np.float32), rng.uniform(-1, 1, cols).astype(np.float32)
    y = torch.full((len(lens),), 9.0, device="cuda")
    ctx.spmv("spmv-block-size=96", dev(rp), dev(ci), dev(v), dev(x), y)
    assert np.array_equal(y.cpu().numpy(), oracle.csr_spmv(rp, ci, v, x))
