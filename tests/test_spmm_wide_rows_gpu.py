"""wave-per-row-tile with a warp per row: products and sums rounded one by one, never fused.  From 128 columns one lane adds up
an output in position order, so the result is the sequential loop's bit for bit."""
import numpy as np
import pytest

import oracle
from tests.helpers import dev, random_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 256, 384, 512])
def test_products_and_sums_are_rounded_separately(ctx, n):
    rp, ci, v = random_csr(300, 433, 40, seed=n)
    B = np.random.default_rng(n).uniform(-1, 1, (433, n)).astype(np.float32)
    C = ctx.spmm("spmm-mapping=wave-per-row-tile spmm-tile-size=16", dev(rp), dev(ci), dev(v), dev(B))
    assert np.array_equal(C.cpu().numpy(), oracle.csr_spmm(rp, ci, v, B))
