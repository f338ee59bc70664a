"""wave-per-row and block-per-row SpMV: a group of lanes per short row, and the stream of rows with x in shared memory."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import assert_within_bound, dev

pytestmark = pytest.mark.gpu


def _check(ctx, opts, lens, cols, seed, grid_below=None):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, cols, rp[-1]).astype(np.int32)
    v, x = rng.uniform(-1, 1, rp[-1]).astype(np.float32), rng.uniform(-1, 1, cols).astype(np.float32)
    y = torch.full((len(lens),), 9.0, device="cuda")
    ctx.spmv(opts, dev(rp), dev(ci), dev(v), dev(x), y)
    assert_within_bound(y.cpu().numpy(), oracle.csr_spmv(rp, ci, v, x, parallel=True), oracle.csr_abs_bound(rp, ci, v, x))
    if grid_below:
        assert ctx.launch_shape(opts, len(lens), int(rp[-1])).physical_grid < grid_below


@pytest.mark.parametrize("mapping", ["wave-per-row", "block-per-row"])
@pytest.mark.parametrize("mean", [1, 20, 24, 40, 50, 90])  # 4, 8 and 16 lanes per row
def test_short_rows(ctx, mapping, mean):
    rng = np.random.default_rng(mean)
    # more rows than groups of lanes in the grid; rows below, at and above what a group and a warp take at once
    lens = rng.integers(0, 2 * mean + 1, 160000 if mean < 30 else 120000)
    lens[rng.integers(0, len(lens), 40)] = [0, 1, 3, 4, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 513, 1000, 5000,
                                            8191] * 2
    lens[-1] = 3
    _check(ctx, f"spmv-mapping={mapping}", lens, 3000, mean, grid_below=148 * 8 + 1)


@pytest.mark.parametrize("mapping", ["wave-per-row", "block-per-row"])
@pytest.mark.parametrize("cols", [49153, 70001, 196608])
def test_rows_with_x_in_shared_memory(ctx, mapping, cols):
    rng = np.random.default_rng(cols)
    lens = rng.integers(0, 400, 4 * cols * 1000000 // 49152 // 200 * 5 // 4 + 100)
    lens[[0, 5, -1]] = 0, 20000, 1
    _check(ctx, f"spmv-mapping={mapping}", lens, cols, cols)


@pytest.mark.parametrize("mapping", ["wave-per-row", "block-per-row"])
@pytest.mark.parametrize("rows", [65536, 81921, 122880])
def test_square_matrices_take_the_stream_of_rows(ctx, mapping, rows):
    # one block of 1,024 threads per SM: the launch shape says that x is staged
    rng = np.random.default_rng(rows)
    lens = rng.integers(60, 200, rows)
    lens[[0, 7, -1]] = 0, 9001, 1
    opts = f"spmv-mapping={mapping}"
    assert ctx.launch_shape(opts, rows, int(lens.sum())).physical_grid == torch.cuda.get_device_properties(0).multi_processor_count
    _check(ctx, opts, lens, rows, rows)


@pytest.mark.parametrize("mapping", ["wave-per-row", "block-per-row"])
@pytest.mark.parametrize("rows,low,high", [(50000, 0, 30), (65536, 90, 170)])  # groups of lanes; stream of rows
def test_entries_outside_the_rows_belong_to_another_x(ctx, mapping, rows, low, high):
    # a range of rows of a larger matrix with spare capacity behind it: the entries around the range lie past the end of x.
    # (x is the front of a larger buffer, so that a kernel that read there all the same would do no harm.)
    rng = np.random.default_rng(rows)
    lens = rng.integers(low, high, rows)
    rp = (5 + np.concatenate([[0], np.cumsum(lens)])).astype(np.int32)
    ci = rng.integers(rows, rows + 4096, rp[-1] + 7).astype(np.int32)
    ci[rp[0]:rp[-1]] = rng.integers(0, rows, rp[-1] - rp[0])
    v = rng.uniform(-1, 1, len(ci)).astype(np.float32)
    xs = np.full(rows + 4096, np.nan, np.float32)
    xs[:rows] = rng.uniform(-1, 1, rows)
    y = ctx.spmv(f"spmv-mapping={mapping}", dev(rp), dev(ci), dev(v), dev(xs)[:rows]).cpu().numpy()
    own = slice(rp[0], rp[-1])
    want = oracle.csr_spmv(rp - rp[0], ci[own], v[own], xs[:rows], parallel=True)
    assert_within_bound(y, want, oracle.csr_abs_bound(rp - rp[0], ci[own], v[own], xs[:rows]))


@pytest.mark.parametrize("mapping", ["wave-per-row", "block-per-row"])
@pytest.mark.parametrize("rows,low,high", [(100000, 0, 8), (90000, 20, 50), (170000, 30, 80), (120000, 30, 100), (81920, 100, 160)])
def test_rows_that_the_block_takes(ctx, mapping, rows, low, high):
    # limits of 2,048 (groups of lanes) and 8,192 (stream of rows); steps of two quads per thread; several in one block
    rng = np.random.default_rng(rows)
    lens = rng.integers(low, high, rows)
    edges = [2047, 2048, 2049, 2052, 4095, 4097, 8191, 8192, 8193, 8200, 16384, 16389, 30001]
    lens[:len(edges)] = edges
    lens[rng.integers(100, rows - 1, len(edges))] = edges
    lens[-1] = 9000
    _check(ctx, f"spmv-mapping={mapping}", lens, rows, rows)


@pytest.mark.parametrize("mapping", ["wave-per-row", "block-per-row"])
def test_rows_sorted_by_length(ctx, mapping):
    # 64 rows of 65,536 in front of 500,000 of 8: as eight rows of one warp each they take 3 ms
    lens = torch.full((500000,), 8, device="cuda")
    lens[:64] = 65536
    rp = torch.nn.functional.pad(torch.cumsum(lens, 0), (1, 0)).int()
    ci = torch.randint(0, 500000, (int(rp[-1]),), device="cuda", dtype=torch.int32)
    v, x = torch.ones(ci.numel(), device="cuda"), torch.ones(500000, device="cuda")
    times = []
    for _ in range(4):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        y = ctx.spmv(f"spmv-mapping={mapping}", rp, ci, v, x)
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    assert torch.equal(y, lens.float())
    assert min(times) < 1.0  # ms


@pytest.mark.parametrize("rows,mean", [(60000, 70), (100000, 95), (110000, 95), (250000, 95), (60000, 130), (131072, 120), (140000, 120)])
def test_wave_per_row_on_both_sides_of_its_limits(ctx, rows, mean):
    # a warp per row on the reference's grid, or groups of lanes (up to eight blocks per SM) and one block per SM
    lens = np.random.default_rng(mean).integers(mean - 30, mean + 30, rows)
    nnz = int(lens.sum())
    grid = ctx.launch_shape("spmv-mapping=wave-per-row spmv-block-size=128", rows, nnz).physical_grid
    takes_others = nnz >= 10000000 if mean <= 100 else 65536 <= rows <= 131072
    assert (grid < rows // 4) == takes_others
    _check(ctx, "spmv-mapping=wave-per-row spmv-block-size=128", lens, rows, mean)
