"""Element offsets past 2^31: outputs of more than 2^31 elements and column indices up to the int32 maximum.
The operands are far too large for the CPU oracle, so the expected values come from the structure of the
matrices: one nonzero per row makes every output a single rounded product (bit-exact by construction), and
the SpMV case is summed in float64 on the device and held to the same bound as everywhere else."""
import pytest
import torch

from sparsewave_b200 import workloads as W

pytestmark = pytest.mark.gpu

CHUNK = 1 << 22


def _one_per_row(rows, cols, seed, empty_every):
    g = torch.Generator(device="cuda").manual_seed(seed)
    keep = torch.ones(rows, dtype=torch.bool, device="cuda")
    keep[::empty_every] = False  # empty rows in between
    row_ptr = torch.zeros(rows + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = torch.cumsum(keep.to(torch.int32), 0, dtype=torch.int32)
    nnz = int(row_ptr[-1])
    col = torch.randint(0, cols, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    val = torch.rand(nnz, generator=g, device="cuda") * 2 - 1
    return keep, row_ptr, col, val


@pytest.mark.parametrize("opts", [
    "spmm-mapping=wave-per-row-tile spmm-tile-size=16 spmm-block-size=256",
    "spmm-mapping=wave-per-row-tile spmm-tile-size=5 spmm-block-size=64",
    "spmm-mapping=thread-per-output spmm-block-size=256",
    "spmm-mapping=thread-per-position spmm-position-chunk-size=4",
])
def test_spmm_outputs_past_2_pow_31_elements(ctx, opts):
    rows, cols, n = (1 << 25) + 77, 5000, 64  # rows * n = 2^31 + 4928 output elements (8.6 GB)
    keep, row_ptr, col, val = _one_per_row(rows, cols, 61, 1000)
    B = W.dense_uniform((cols, n), seed=62, device="cuda")
    C = ctx.spmm(opts, row_ptr, col, val, B)
    assert ctx.device_status() == 0 and C.shape == (rows, n)
    pos = row_ptr[:-1].long()
    for r0 in range(0, rows, CHUNK):
        r1 = min(rows, r0 + CHUNK)
        k = keep[r0:r1]
        p = pos[r0:r1].clamp(max=col.numel() - 1)
        expected = (val[p][:, None] * B[col[p].long()]) * k[:, None]
        assert torch.equal(C[r0:r1], expected), f"rows {r0}..{r1}"
    del C
    torch.cuda.empty_cache()


def test_spmv_column_indices_up_to_the_int32_maximum(ctx):
    from tests.helpers import SPMV_MAPPING_OPTIONS
    cols = (1 << 31) - 1  # x holds 2^31 - 1 floats (8.6 GB); the last column index is the int32 maximum - 1
    g = torch.Generator(device="cuda").manual_seed(63)
    lens = torch.randint(0, 200, (4096,), generator=g, device="cuda")
    lens[7], lens[8], lens[4095] = 70000, 0, 1025  # one long row, an empty one behind it, a ragged last row
    rows, nnz = lens.numel(), int(lens.sum())
    row_ptr = torch.zeros(rows + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = torch.cumsum(lens, 0).to(torch.int32)
    row_of = torch.repeat_interleave(torch.arange(rows, device="cuda"), lens)
    # distinct sorted columns within a row: a random start plus a strictly increasing walk over the whole range
    step = torch.randint(1, cols // 70001, (nnz,), generator=g, device="cuda")
    walk = torch.cumsum(step, 0)
    first = torch.repeat_interleave(walk[row_ptr[:-1].long().clamp(max=nnz - 1)] - step[row_ptr[:-1].long().clamp(max=nnz - 1)], lens)
    col64 = walk - first - 1
    col64[int(row_ptr[8]) - 1] = cols - 1  # the long row ends on the last column
    assert int(col64.max()) == cols - 1 and int(col64.min()) >= 0
    col = col64.to(torch.int32)
    val = torch.rand(nnz, generator=g, device="cuda") * 2 - 1
    x = torch.empty(cols, device="cuda").uniform_(-1, 1, generator=g)
    prod = val.double() * x[col64].double()
    expected = torch.zeros(rows, dtype=torch.float64, device="cuda").index_add_(0, row_of, prod)
    bound = torch.zeros(rows, dtype=torch.float64, device="cuda").index_add_(0, row_of, prod.abs())
    for opts in SPMV_MAPPING_OPTIONS:
        y = ctx.spmv(opts, row_ptr, col, val, x)
        assert ctx.device_status() == 0
        excess = (y.double() - expected).abs() - 1e-5 * bound
        assert float(excess.max()) <= 0, opts


def test_bsr16_bf16_outputs_past_2_pow_31_elements(ctx):
    grid_rows, grid_cols, n = (1 << 17) + 3, 300, 1024  # 16 * grid_rows * n = 2^31 + 49152 outputs (4.3 GB of bf16)
    keep, brp, bci, _ = _one_per_row(grid_rows, grid_cols, 64, 777)
    nb = bci.numel()
    g = torch.Generator(device="cuda").manual_seed(65)
    blocks = (torch.rand((nb, 16, 16), generator=g, device="cuda") * 2 - 1).to(torch.bfloat16)
    B = W.dense_normal((grid_cols * 16, n), seed=66, device="cuda")
    assert B.dtype == torch.bfloat16
    C = ctx.bsr_spmm("", brp, bci, blocks.reshape(-1), B, 16)
    assert ctx.device_status() == 0 and C.shape == (grid_rows * 16, n)
    Bt = B.float().view(grid_cols, 16, n)
    pos = brp[:-1].long().clamp(max=nb - 1)
    step = 4096
    for b0 in range(0, grid_rows, step):
        b1 = min(grid_rows, b0 + step)
        k = keep[b0:b1][:, None, None]
        a = blocks[pos[b0:b1]].float()
        b = Bt[bci[pos[b0:b1]].long()]
        expected = torch.bmm(a, b) * k                 # products of bf16 values are exact in fp32
        bound = torch.bmm(a.abs(), b.abs()) * k
        got = C[b0 * 16:b1 * 16].float().view(b1 - b0, 16, n)
        # one bf16 ulp around the fp32 sum, plus the slack of the accumulation order where terms cancel
        excess = (got - expected).abs() - (2.0 ** -7) * expected.abs() - 1e-2 * (2.0 ** -6) * bound
        assert float(excess.max()) <= 0, f"block rows {b0}..{b1}"


def _up_to_the_last_position(nnz, row_length):
    """Rows of `row_length` positions up to position `nnz`, columns p % 5, values 1; the sum of x = 0, 1, 2, 3, 4 over each row."""
    rows = -(-nnz // row_length)
    ends = torch.clamp(torch.arange(rows + 1, device="cuda") * row_length, max=nnz)
    col = torch.arange(nnz, dtype=torch.int32, device="cuda").remainder_(5)
    below = ends // 5 * 10 + (ends % 5) * (ends % 5 - 1) // 2  # sum of p % 5 over the positions before
    return ends.to(torch.int32), col, torch.ones(nnz, device="cuda"), (below[1:] - below[:-1]).float()


def test_row_products_up_to_the_last_position(ctx):
    # tiles of 2048 positions: the one behind the last would start past the int32 maximum.  Sums are whole numbers: exact.
    row_ptr, col, val, expected = _up_to_the_last_position((1 << 31) - 1, 2048)
    x = torch.arange(5, dtype=torch.float32, device="cuda")
    assert torch.equal(ctx.spmv("", row_ptr, col, val, x), expected)
    row_ptr[-1] -= 256  # SpMM takes up to 2^31 - 257 nonzeros
    expected[-1] -= (torch.arange((1 << 31) - 257, (1 << 31) - 1, device="cuda") % 5).sum()
    C = ctx.spmm("", row_ptr, col[:-256], val[:-256], torch.stack([x, 2 * x, 3 * x, -x], 1).contiguous())
    assert torch.equal(C, torch.stack([expected, 2 * expected, 3 * expected, -expected], 1))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("row_length", [64, 2048])  # below and above the rows that take 128-bit loads
def test_row_mappings_up_to_the_last_position(ctx, row_length):
    # strides of up to 1024 threads past the last positions of the matrix
    row_ptr, col, val, expected = _up_to_the_last_position((1 << 31) - 1, row_length)
    x = torch.arange(5, dtype=torch.float32, device="cuda")
    for opts in ("spmv-mapping=wave-per-row spmv-block-size=128", "spmv-mapping=block-per-row spmv-block-size=64",
                 "spmv-mapping=block-per-row spmv-block-size=1024"):
        assert torch.equal(ctx.spmv(opts, row_ptr, col, val, x), expected), opts
    assert ctx.device_status() == 0


def test_bsr_blocks_up_to_the_last_position(ctx):
    # 2^31 - 1 blocks of 1 x 1: block columns are read two blocks ahead of the last one
    brp, bci, bv, expected = _up_to_the_last_position((1 << 31) - 1, 2048)
    x = torch.arange(5, dtype=torch.float32, device="cuda")
    C = ctx.bsr_spmm("", brp, bci, bv, torch.stack([x, 2 * x, 3 * x, -x], 1).contiguous(), 1)
    assert torch.equal(C, torch.stack([expected, 2 * expected, 3 * expected, -expected], 1))
    assert ctx.device_status() == 0
