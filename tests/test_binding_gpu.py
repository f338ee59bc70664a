"""The native operator calls behind api.Context: option forms, operand checks and threads."""
import threading

import pytest
import torch

from sparsewave_b200 import Context, SparseWaveError, make_options
from tests.helpers import SPMV_GOLDEN, dev

pytestmark = pytest.mark.gpu


def _operands():
    g = SPMV_GOLDEN
    return [dev(g["row_ptr"], torch.int32), dev(g["col"], torch.int32), dev(g["val"], torch.float32),
            dev(g["x"], torch.float32)], g["y"]


@pytest.mark.parametrize("options", ["", None, "mapping=wave-per-row", make_options("mapping=block-per-row block-size=64")])
def test_option_forms(ctx, options):
    t, want = _operands()
    assert ctx.spmv(options, *t).cpu().tolist() == want
    y = torch.full((5,), 7.0, device="cuda")
    assert ctx.spmv(options, *t, y, rows=5) is y and y.cpu().tolist() == want


def test_operand_errors(ctx):
    t, _ = _operands()
    with pytest.raises(TypeError, match=r"col_idx must have dtype torch.int32, got torch.int64"):
        ctx.spmv("", t[0], t[1].long(), t[2], t[3])
    with pytest.raises(TypeError, match="x must be contiguous"):
        ctx.spmv("", *t[:3], torch.zeros((4, 2), device="cuda")[:, 0])
    with pytest.raises(TypeError, match="val must be a CUDA tensor"):
        ctx.spmv("", t[0], t[1], [1.0], t[3])
    with pytest.raises(IndexError):
        ctx.spmm("", *t)
    for _ in range(2):  # a text that does not parse is not kept
        with pytest.raises(SparseWaveError, match="unknown option 'colour'"):
            ctx.spmv("colour=3", *t)
    closed = Context(0)
    closed.close()
    with pytest.raises(SparseWaveError, match="context is NULL"):
        closed.spmv("", *t)


def test_threads_with_a_context_each():
    t, want = _operands()
    got = []

    def work(k):
        with Context(0) as c:
            for i in range(300):  # more option texts than are kept
                y = c.spmv(f"mapping=wave-per-row block-size={32 * (1 + (k + i) % 32)}" + " " * (i % 100), *t)
            got.append(y.cpu().tolist())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [th.start() for th in threads]
    [th.join() for th in threads]
    assert got == [want] * 4
