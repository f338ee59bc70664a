"""Resident matrices stored as two column parts and cut into row panels."""
import numpy as np
import pytest

import oracle
from sparsewave_b200 import workloads as W
from tests.helpers import assert_within_bound

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,max_len", [(150001, 150001, 65536), (700000, 40, 20), (600000, 300007, 3000)])
def test_column_parts_made_on_the_device(ctx, monkeypatch, rows, cols, max_len):
    monkeypatch.setenv("SWB_RESIDENT_SPLIT_NNZ", "3000000")
    a = W.zipf_csr(rows, cols, 1.2 if cols == 40 else 1.6, 1, max_len, seed=rows, device="cuda")
    assert a.nnz > 3_000_000
    rp, ci, v = a.numpy()
    shuffled = np.random.default_rng(1).permutation(rp[1] - rp[0])  # column order within a row is not relied on
    ci[:rp[1]], v[:rp[1]] = ci[:rp[1]][shuffled], v[:rp[1]][shuffled]
    resident = ctx.csr_upload(rows, cols, rp, ci, v)
    for seed in (1, 2):
        x = np.random.default_rng(seed).uniform(-1, 1, cols).astype(np.float32)
        y = np.full(rows, 5.0, np.float32)
        resident.spmv_host("spmv-mapping=wave-per-position", x, y)
        assert_within_bound(y, oracle.csr_spmv(rp, ci, v, x, parallel=True), oracle.csr_abs_bound(rp, ci, v, x))
    resident.release()
