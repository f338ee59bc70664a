"""Performance cases of the operators: what programs built on the library call, from latency-bound to the largest.

A case is a dict of plain values.  `prepare` makes what a program has in hand before the call (operands from a seed,
the context, an uploaded matrix), `run` is one call through the public Python API with the option text such a program
passes, `work` states the bytes and operations the call cannot do without.
"""
import functools
import math

import numpy as np
import torch

from sparsewave_b200 import Context

ZIPF_EXPONENT = 1.8
ZIPF_MAX = 65536
HALF_BAND = 1024

# SpMV mappings, with the block sizes that the benchmark and the documentation use for them.
THREAD_PER_ROW = ""  # the defaults: thread-per-row, blocks of 256
WAVE_PER_ROW = "spmv-mapping=wave-per-row spmv-block-size=128"
BLOCK_PER_ROW = "spmv-mapping=block-per-row spmv-block-size=64"
ATOMIC = "spmv-mapping=thread-per-position spmv-block-size=256"
SEGMENTED = ("spmv-mapping=thread-per-position spmv-position-chunk-size=8 spmv-position-reduction=segmented "
             "spmv-block-size=256")
WAVE_PER_POSITION = "spmv-mapping=wave-per-position spmv-block-size=128"


def listed():
    return [
        # One small SpMV (the benchmark's configuration 1): launches and host work, not the GPU, decide.
        dict(name="spmv_small", op="spmv", rows=4096, mean=16, lengths="uniform", options=WAVE_PER_ROW),
        # The library's defaults on short ragged rows, an economic or circuit matrix (odd size).
        dict(name="spmv_default_ragged", op="spmv", rows=206501, mean=6, lengths="ragged", options=THREAD_PER_ROW),
        # Long equal rows, the mapping made for them (the reference's uniform-256 sweep).
        dict(name="spmv_block_per_row", op="spmv", rows=65536, mean=256, lengths="uniform", options=BLOCK_PER_ROW),
        # Power-law rows (graphs), positions dealt to threads; configuration 3 compares this mapping.
        dict(name="spmv_segmented_zipf", op="spmv", rows=1048577, mean=0, lengths="zipf", options=SEGMENTED),
        # Configuration 3 at full size: 4 M power-law rows, 92 M nonzeros.
        dict(name="spmv_power_law", op="spmv", rows=4194304, mean=0, lengths="zipf", options=WAVE_PER_POSITION),
        # Configuration 2, the one shape that an ahead-of-time bundle supports: four right-hand sides.
        dict(name="spmm_bundle_n4", op="spmm", rows=65536, mean=32, lengths="uniform", n=4,
             options="spmm-mapping=wave-per-row-tile spmm-tile-size=4 spmm-block-size=64"),
        # A graph layer of ordinary size with the library's defaults (the ca-AstroPh scale of the reference's sweep).
        dict(name="spmm_default_n32", op="spmm", rows=18772, mean=21, lengths="ragged", n=32, options=""),
        # A feature width that is no multiple of 4, ragged rows.
        dict(name="spmm_ragged_n50", op="spmm", rows=250001, mean=20, lengths="ragged", n=50,
             options="spmm-mapping=wave-per-row-tile spmm-tile-size=8 spmm-block-size=256"),
        # Configuration 4 at full size: banded-plus-random, 134 M nonzeros, 64 right-hand sides.
        dict(name="spmm_banded_n64", op="spmm", rows=2097152, mean=64, lengths="banded", n=64,
             options="spmm-mapping=wave-per-row-tile spmm-tile-size=16 spmm-block-size=256"),
        # Configuration 5: block-pruned weights, 16 x 16 bf16 blocks at 5 % density.
        dict(name="bsr_bf16_16", op="bsr", dtype="bf16", grid=1024, bs=16, blocks=52429, n=512),
        # Small f32 blocks of a finite-element kind (the block sizes of the reference's runner), 32 right-hand sides.
        dict(name="bsr_f32_4", op="bsr", dtype="f32", grid=16384, bs=4, blocks=393216, n=32),
        # Matrix resident on the device, x in and y out per call through pinned host memory.
        dict(name="resident_host_spmv", op="resident", rows=1048576, mean=0, lengths="zipf", options=WAVE_PER_POSITION),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "spmm", "spmm", "spmm", "bsr", "bsr", "resident"])
    if kind == "spmv":
        options = rng.choice([THREAD_PER_ROW, WAVE_PER_ROW, BLOCK_PER_ROW, ATOMIC, SEGMENTED, WAVE_PER_POSITION])
        if options in (ATOMIC, SEGMENTED, WAVE_PER_POSITION):  # any rows, skewed ones above all
            lengths = rng.choice(["zipf", "zipf", "ragged"])
            mean = 0 if lengths == "zipf" else _log(rng, 3, 64)
            return dict(op="spmv", rows=_log(rng, 4000, 4194304 if lengths == "zipf" else 1048576), mean=mean,
                        lengths=lengths, options=options)
        # a thread, a warp or a block per row: short, middling or long rows
        low, high = {THREAD_PER_ROW: (3, 48), WAVE_PER_ROW: (8, 256), BLOCK_PER_ROW: (64, 1024)}[options]
        mean = _log(rng, low, high)
        return dict(op="spmv", rows=_log(rng, 2048, min(1048576, 33554432 // mean)), mean=mean,
                    lengths=rng.choice(["uniform", "ragged"]), options=options)
    if kind == "spmm":
        mean = _log(rng, 4, 64)
        n = rng.choice([4, 8, 16, 32, 64, 128]) if rng.random() < 0.5 else _log(rng, 1, 200)
        rows = _log(rng, 2048, max(4096, min(1048576, 500000000 // (mean * n))))
        options = "" if rng.random() < 0.35 else "spmm-mapping=wave-per-row-tile spmm-tile-size=%d spmm-block-size=%d" % (
            rng.choice([4, 8, 16, 32]), rng.choice([64, 256]))
        return dict(op="spmm", rows=rows, mean=mean, lengths=rng.choice(["uniform", "ragged", "banded"]), n=n,
                    options=options)
    if kind == "bsr":
        dtype = rng.choice(["bf16", "f32"])
        bs = rng.choice([8, 16, 16, 32] if dtype == "bf16" else [2, 4, 8])
        n = 8 * _log(rng, 1, 64) if rng.random() < 0.75 else _log(rng, 1, 512)
        grid = _log(rng, 64, 65536 // bs)
        per_row = min(grid // 2, _log(rng, 4, 64), max(4, 1000000000 // (grid * bs * bs * n)))
        return dict(op="bsr", dtype=dtype, grid=grid, bs=bs, blocks=grid * per_row, n=n)
    return dict(op="resident", rows=_log(rng, 65536, 1048576), mean=0, lengths="zipf", options=WAVE_PER_POSITION)


# ---- sizes -------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _lengths(kind, rows, mean):
    """Row lengths of a square matrix, in ascending order: the quantiles of their distribution, so that a case has the
    same number of nonzeros whatever the seed (which decides which row gets which length)."""
    u = (np.arange(rows, dtype=np.float64) + 0.5) / rows
    if kind in ("uniform", "banded"):
        lens = np.full(rows, mean, dtype=np.int64)
    elif kind == "ragged":  # geometric: many short rows, some empty, a few of ten times the mean
        lens = np.floor(np.log1p(-u) / math.log(mean / (mean + 1.0))).astype(np.int64)
    else:
        weights = np.arange(1, min(ZIPF_MAX, rows // 2) + 1, dtype=np.float64) ** -ZIPF_EXPONENT
        cdf = np.cumsum(weights)
        lens = np.searchsorted(cdf / cdf[-1], u).astype(np.int64) + 1
        lens = np.minimum(lens, len(weights))
    return np.minimum(lens, rows // 2)


def work(case):
    if case["op"] == "bsr":
        size, elem = case["grid"] * case["bs"], 2 if case["dtype"] == "bf16" else 4
        stored = case["blocks"] * case["bs"] ** 2
        return {"bytes": elem * stored + 4 * case["blocks"] + 4 * (case["grid"] + 1) + 2 * elem * size * case["n"],
                "flops": 2 * stored * case["n"]}
    rows, n = case["rows"], case.get("n", 1)
    nnz = int(_lengths(case["lengths"], rows, case["mean"]).sum())
    return {"bytes": 8 * nnz + 4 * (rows + 1) + 8 * rows * n, "flops": 2 * nnz * n}


def tolerance(case):
    if case["op"] == "bsr" and case["dtype"] == "bf16":
        # f32 sums rounded once to bf16: another order of the sum moves some results by one unit in the last place
        return {"rel": 2e-3, "max": 1e-2}
    if case["op"] == "bsr" or case["options"] == "":
        return "exact"  # thread-per-row and thread-per-output add in position order, bit for bit the sequential loop
    return {"rel": 1e-5, "max": 1e-3}  # 32-bit sums of up to 65536 terms in any order


# ---- inputs ------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=1)
def _context():
    return Context(0)


def _uniform(shape, gen):
    return torch.rand(shape, generator=gen, device="cuda") * 2 - 1


def _pattern(lens, cols, gen, band=False):
    """CSR offsets and uniform-random strictly increasing columns for the row lengths `lens`; with `band`, every other
    column lies within HALF_BAND of the diagonal."""
    rows = lens.numel()
    row_ptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=row_ptr[1:])
    nnz = int(row_ptr[-1])
    row = torch.repeat_interleave(torch.arange(rows, device="cuda"), lens)
    slot = torch.arange(nnz, device="cuda") - row_ptr[row]  # index of an entry in its row
    span = cols - lens[row] + 1
    low = torch.zeros_like(span)
    if band:
        near = slot % 2 == 0
        low = torch.where(near, (row - HALF_BAND).clamp_(min=0), low)
        span = torch.where(near, torch.minimum(row + HALF_BAND, span) - low, span).clamp_(min=1)
        low = torch.minimum(low, cols - lens[row])
    col = low + torch.minimum((torch.rand(nnz, generator=gen, device="cuda") * span).long(), span - 1)
    key = row * cols + col
    del col, span, low
    key = torch.sort(key)[0]
    # sorted draws with repetition plus the index in the row: strictly increasing
    return row_ptr.to(torch.int32), (key - row * cols + slot).to(torch.int32)


class _Resident:
    """An uploaded matrix, released with the state that holds it."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        self.handle.release()


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    ctx = _context()
    if case["op"] == "bsr":
        grid, bs, n = case["grid"], case["bs"], case["n"]
        dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        where = torch.randint(grid, (case["blocks"],), generator=gen, device="cuda")  # blocks fall on block rows
        rp, ci = _pattern(torch.bincount(where, minlength=grid), grid, gen)
        values = torch.randn(case["blocks"] * bs * bs, generator=gen, device="cuda").to(dtype)
        B = torch.randn((grid * bs, n), generator=gen, device="cuda").to(dtype)
        return dict(op="bsr", ctx=ctx, a=(rp, ci, values, B, bs))
    rows = case["rows"]
    lens = torch.from_numpy(_lengths(case["lengths"], rows, case["mean"])).cuda()
    lens = lens[torch.randperm(rows, generator=gen, device="cuda")]
    rp, ci = _pattern(lens, rows, gen, band=case["lengths"] == "banded")
    values = _uniform(ci.numel(), gen)
    state = dict(op=case["op"], ctx=ctx, options=case["options"])
    if case["op"] == "spmm":
        return dict(state, a=(rp, ci, values, _uniform((rows, case["n"]), gen)))
    x = _uniform(rows, gen)
    if case["op"] == "spmv":  # a solver keeps its vectors
        return dict(state, a=(rp, ci, values, x, torch.zeros(rows, device="cuda")))
    matrix = _Resident(ctx.csr_upload(rows, rows, rp.cpu().numpy(), ci.cpu().numpy(), values.cpu().numpy()))
    return dict(state, matrix=matrix, x=x.cpu().pin_memory(), y=torch.zeros(rows).pin_memory())


def run(state):
    if state["op"] == "resident":
        return state["matrix"].handle.spmv_host(state["options"], state["x"], state["y"])
    if state["op"] == "spmv":
        return state["ctx"].spmv(state["options"], *state["a"])
    if state["op"] == "spmm":
        return state["ctx"].spmm(state["options"], *state["a"])
    return state["ctx"].bsr_spmm("", *state["a"])
