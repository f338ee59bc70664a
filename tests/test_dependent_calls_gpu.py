"""Calls that depend on one another, queued without a synchronisation in between: the result of each is the operand of the
next, in two buffers that take turns, so that a kernel which started before the one ahead of it had ended would read or
overwrite what is still in use.  Whole numbers: every mapping gives the same sums, exactly."""
import numpy as np
import pytest
import torch

from tests.helpers import SPMV_MAPPING_OPTIONS, dev

pytestmark = pytest.mark.gpu

SPMM_OPTIONS = ["", "spmm-mapping=wave-per-row-tile spmm-tile-size=4 spmm-block-size=64",
                "spmm-mapping=wave-per-row-tile spmm-tile-size=8 spmm-block-size=256", "spmm-mapping=thread-per-position"]


def _matrix(rows, rng):
    """Three entries per row, two of 1 and one of -1: magnitudes at most triple."""
    ci = np.sort(rng.integers(0, rows, (rows, 3)), axis=1).astype(np.int32)
    v = np.tile(np.array([1, -1, 1], np.float32), (rows, 1))
    return np.arange(0, 3 * rows + 1, 3, dtype=np.int32), ci, v


def _apply(ci, v, x):
    return np.einsum("rk,rk...->r...", v, x[ci])


@pytest.mark.parametrize("rows", [300, 5000, 200000])
@pytest.mark.parametrize("graph", [False, True])
def test_spmv_chain_through_every_mapping(ctx, rows, graph):
    rng = np.random.default_rng(rows)
    rp, ci, v = _matrix(rows, rng)
    operands = dev(rp), dev(ci.reshape(-1)), dev(v.reshape(-1))
    row_of = dev(np.repeat(np.arange(rows, dtype=np.int32), 3))
    x0 = rng.integers(-9, 10, rows).astype(np.float32)
    start, a, b = dev(x0), torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    orders = [list(rng.permutation(len(SPMV_MAPPING_OPTIONS) + 1)) for _ in range(20)]
    kept = []

    def chain():
        for order in orders:
            a.copy_(start)
            x, y = a, b
            for k in order:
                if k == len(SPMV_MAPPING_OPTIONS):
                    ctx.coo_spmv("", rows, row_of, *operands[1:], x, y)
                else:
                    ctx.spmv(SPMV_MAPPING_OPTIONS[k] + " spmv-block-size=128", *operands, x, y)
                x, y = y, x
            kept.append(x.clone())

    if graph:
        chain()
        torch.cuda.synchronize()
        kept.clear()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            chain()
        g.replay()
    else:
        chain()
    want = x0.astype(np.float64)
    for _ in range(len(orders[0])):
        want = _apply(ci, v, want)
    assert np.abs(want).max() < 2 ** 24
    for got in kept:
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("rows", [300, 5000, 60000])
@pytest.mark.parametrize("n", [3, 4, 32, 50])
def test_spmm_and_bsr_chain(ctx, rows, n):
    rng = np.random.default_rng(rows + n)
    rp, ci, v = _matrix(rows, rng)
    operands = dev(rp), dev(ci.reshape(-1)), dev(v.reshape(-1))
    # one 4 x 4 block per block row: rows of a block row exchanged with those of another
    perm = rng.permutation(rows // 4).astype(np.int32)
    turn = np.roll(np.eye(4, dtype=np.float32), 1, axis=1)
    blocks = dev(np.arange(rows // 4 + 1, dtype=np.int32)), dev(perm), dev(np.tile(turn.reshape(-1), rows // 4))
    B0 = rng.integers(-9, 10, (rows, n)).astype(np.float32)
    start, a, b = dev(B0), torch.empty((rows, n), device="cuda"), torch.empty((rows, n), device="cuda")
    kept, orders = [], [list(rng.permutation(8)) for _ in range(15)]  # each option twice, or a block product
    for order in orders:
        a.copy_(start)
        x, y = a, b
        for k in order:
            ctx.spmm(SPMM_OPTIONS[k % 4], *operands, x, y)
            x, y = y, x
            ctx.bsr_spmm("", *blocks, x, 4, y)
            x, y = y, x
        kept.append(x.clone())
    want = B0.astype(np.float64)
    for _ in range(8):
        want = _apply(ci, v, want)
        want = want.reshape(rows // 4, 4, n)[perm][:, [1, 2, 3, 0]].reshape(rows, n)
    assert np.abs(want).max() < 2 ** 24
    for got in kept:
        assert np.array_equal(got.cpu().numpy(), want)
