"""Position SpMV at the sizes where the partitions per warp change, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import assert_within_bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,batch", [(7, 2), (42, 4), (243, 8)])  # partitions per SM from which a warp takes `batch`
@pytest.mark.parametrize("block", [128, 1024])
@pytest.mark.parametrize("below", [False, True])
def test_edges(ctx, per_sm, batch, block, below):
    partitions = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    groups = -(-partitions // (block // 32)) - below  # the partitions come in blocks
    nnz = groups * block - 5
    rng = np.random.default_rng(nnz)
    rows = nnz // 6
    cuts = np.sort(rng.integers(0, nnz + 1, rows - 1))
    cuts[rows // 2:rows // 2 + 9] = cuts[rows // 2]  # empty rows
    cuts = np.sort(cuts)
    rp = np.concatenate([[0], cuts, [nnz]]).astype(np.int32)
    ci = rng.integers(0, 5000, nnz).astype(np.int32)
    v, x = rng.uniform(-1, 1, nnz).astype(np.float32), rng.uniform(-1, 1, 5000).astype(np.float32)
    options = f"spmv-mapping=wave-per-position spmv-block-size={block}"
    smaller = {2: 1, 4: 2, 8: 4}[batch]
    spans = -(-groups * (block // 32) // (smaller if below else batch))
    assert ctx.launch_shape(options, rows, nnz).physical_grid == -(-spans // (block // 32))
    y = ctx.spmv(options, *(torch.from_numpy(t).cuda() for t in (rp, ci, v, x)))
    assert_within_bound(y.cpu().numpy(), oracle.csr_spmv(rp, ci, v, x), oracle.csr_abs_bound(rp, ci, v, x))
