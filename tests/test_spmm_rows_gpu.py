"""SpMM by groups of lanes that take whole rows in turn, and by staged products for up to four columns: thread-per-output
for every N, wave-per-row-tile from the sizes where it takes these kernels."""
import numpy as np
import pytest
import torch

import oracle
from tests.helpers import assert_within_bound, dev, random_csr

pytestmark = pytest.mark.gpu

# one, two and four columns per lane; 1 to 5 runs of them; the last widths without column tiles and the first with
WIDTHS = [1, 2, 3, 4, 5, 8, 31, 32, 33, 35, 63, 64, 66, 75, 96, 97, 100, 128, 129, 130, 132, 161, 187, 198, 224, 225, 256, 260, 300, 321, 512, 516]


def _spmm(ctx, opts, rp, ci, v, B, C=None):
    return ctx.spmm(opts, dev(rp), dev(ci), dev(v), B, C)


@pytest.mark.parametrize("n", WIDTHS)
@pytest.mark.parametrize("rows,mean", [(1, 70), (300, 9), (20000, 3)])
def test_thread_per_output_widths(ctx, n, rows, mean):
    rp, ci, v = random_csr(rows, 433, mean, seed=n + rows)
    B = np.random.default_rng(n).uniform(-1, 1, (433, n)).astype(np.float32)
    want = oracle.csr_spmm(rp, ci, v, B, parallel=True)
    assert np.array_equal(_spmm(ctx, "", rp, ci, v, dev(B)).cpu().numpy(), want)
    # B and C that start four bytes past a 16-byte boundary: single columns
    Bu = torch.empty(B.size + 1, device="cuda")[1:].view(B.shape).copy_(torch.from_numpy(B))
    Cu = torch.empty(rows * n + 1, device="cuda")[1:].view(rows, n)
    assert np.array_equal(_spmm(ctx, "", rp, ci, v, Bu, Cu).cpu().numpy(), want)


@pytest.mark.parametrize("n", [4, 32, 50, 147])
def test_rows_beyond_the_staged_positions(ctx, n):
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 30, 3000)
    lens[[0, 777, 2999]] = 5000, 1537, 4096
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 6000, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (6000, n)).astype(np.float32)
    assert np.array_equal(_spmm(ctx, "", rp, ci, v, dev(B)).cpu().numpy(), oracle.csr_spmm(rp, ci, v, B, parallel=True))


@pytest.mark.parametrize("rows,mean,n", [(50000, 6, 1), (50000, 6, 3), (60000, 5, 7), (200000, 5, 16), (150000, 9, 32),
                                         (40000, 12, 50), (100000, 4, 64), (110000, 16, 64), (70000, 7, 128), (20000, 8, 84),
                                         (9000, 6, 147), (3000, 5, 500)])
def test_wave_per_row_tile_takes_the_rows_kernel(ctx, rows, mean, n):
    opts = "spmm-mapping=wave-per-row-tile spmm-tile-size=8 spmm-block-size=256"
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 2 * mean + 1, rows)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 2000, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (2000, n)).astype(np.float32)
    want, bound = oracle.csr_spmm(rp, ci, v, B, parallel=True), oracle.csr_abs_bound(rp, ci, v, B)
    assert ctx.launch_shape(opts, rows, int(rp[-1]), n).physical_grid < rows
    assert np.array_equal(_spmm(ctx, opts, rp, ci, v, dev(B)).cpu().numpy(), want)
    C = torch.ones((rows, n), device="cuda")
    _spmm(ctx, opts + " accumulate=1", rp, ci, v, dev(B), C)
    assert_within_bound(C.cpu().numpy(), want + 1.0, bound + 1.0)


@pytest.mark.parametrize("n", [5, 17, 31, 32])
@pytest.mark.parametrize("mean", [10, 11, 24])  # one or several steps of 12 positions, steps of 8
def test_steps_of_many_rows(ctx, mean, n):
    rows = 40000
    rng = np.random.default_rng(mean + n)
    lens = rng.integers(0, 2 * mean + 1, rows)
    lens[:64] = np.arange(64)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 900, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (900, n)).astype(np.float32)
    Bu = torch.empty(B.size + 1, device="cuda")[1:].view(B.shape).copy_(torch.from_numpy(B))
    assert np.array_equal(_spmm(ctx, "", rp, ci, v, Bu).cpu().numpy(), oracle.csr_spmm(rp, ci, v, B, parallel=True))


@pytest.mark.parametrize("n", [5, 9, 16, 32, 35, 50, 63, 75, 66, 132, 198, 256, 300])  # 1, 2, 4 columns x 1 to 5 runs
def test_rows_that_the_block_finishes(ctx, n):
    # a group takes 1,024 positions of a row, the block the rest in tiles of up to 128: ends of both, several in a block
    lens = np.full(9000, 3)
    lens[[0, 1, 2, 3, 40, 41, 4500, 8999]] = 1024, 1025, 1151, 1153, 1026, 1280, 7000, 3333
    rng = np.random.default_rng(n)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 1300, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (1300, n)).astype(np.float32)
    want = oracle.csr_spmm(rp, ci, v, B, parallel=True)
    assert np.array_equal(_spmm(ctx, "", rp, ci, v, dev(B)).cpu().numpy(), want)
    C = torch.ones((9000, n), device="cuda")
    _spmm(ctx, "spmm-mapping=wave-per-row-tile spmm-tile-size=8 accumulate=1", rp, ci, v, dev(B), C)
    assert_within_bound(C.cpu().numpy(), want + 1.0, oracle.csr_abs_bound(rp, ci, v, B) + 1.0)


@pytest.mark.parametrize("opts", ["", "spmm-mapping=wave-per-row-tile spmm-tile-size=16 spmm-block-size=256"])
def test_a_very_long_row_is_not_one_chain(ctx, opts):
    # 64 columns, 200,000 rows of 10 and one of 65,536: as a chain of one group of lanes it takes 125 ns a position
    lens = torch.full((200000,), 10, device="cuda")
    lens[777] = 65536
    rp = torch.nn.functional.pad(torch.cumsum(lens, 0), (1, 0)).int()
    ci = torch.randint(0, 200000, (int(rp[-1]),), device="cuda", dtype=torch.int32)
    v, B = torch.rand(ci.numel(), device="cuda"), torch.rand((200000, 64), device="cuda")
    times = []
    for _ in range(4):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        ctx.spmm(opts, rp, ci, v, B)
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    assert min(times) < 65536 * 80e-6  # ms


@pytest.mark.parametrize("rows,most,n,outputs", [
    (262144, 9, 2, True), (262144, 24, 3, True), (262143, 9, 3, False), (262144, 28, 2, False), (8192, 7, 33, True),
    (8192, 7, 128, True), (8192, 7, 129, False), (8193, 7, 33, False), (8193, 7, 5, True), (32768, 8, 32, True), (32769, 7, 9, True),
    (32769, 7, 8, False), (9000, 11, 16, False), (8000, 2, 100, True)])
def test_thread_per_output_on_very_short_rows(ctx, rows, most, n, outputs):
    # a thread per output in blocks of 256, which start and end inside a row; both sides of each limit
    rng = np.random.default_rng(rows + n)
    lens = rng.integers(0, most + 1, rows)
    lens[[0, 5, -1]] = 0, 700, 5
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 800, rp[-1]).astype(np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32)
    B = rng.uniform(-1, 1, (800, n)).astype(np.float32)
    assert (ctx.launch_shape("", rows, int(rp[-1]), n).physical_grid == -(-rows * n // 256)) == outputs
    assert np.array_equal(_spmm(ctx, "", rp, ci, v, dev(B)).cpu().numpy(), oracle.csr_spmm(rp, ci, v, B, parallel=True))
