"""Which products the kernel for the rows of an ordinary step is given (``ops.rows_ok``); the library gets the others, as it got all of them before."""
import pytest
import torch

from return_b200.ext import ops

M, N, K = 40, 64, 128


def _forms():
    x, w, out = torch.zeros(M, K).bfloat16(), torch.zeros(N, K).bfloat16(), torch.zeros(M, N).bfloat16()
    wide = torch.zeros(M, 2 * K).bfloat16()
    yield "plain", x, w, out, True
    yield "rows apart", wide[:, :K], w, out, True
    yield "columns from an aligned place on", wide[:, 8:8 + K], w, out, True
    yield "float32 out", x, w, out.float(), True
    yield "part of a wider out", x, w, torch.zeros(M, N + 3).bfloat16()[:, 1:1 + N], True
    yield "transposed weight", x, torch.zeros(K, N).bfloat16().t(), out, False
    yield "transposed rows", torch.zeros(K, M).bfloat16().t(), w, out, False
    yield "every second column", wide[:, ::2], w, out, False
    yield "every second column of the weight", x, torch.zeros(N, 2 * K).bfloat16()[:, ::2], out, False
    yield "one row for all", x[:1].expand(M, K), w, out, False
    yield "one weight row for all", x, w[:1].expand(N, K), out, False
    yield "rows that overlap", torch.zeros(M * 8 + K).bfloat16().as_strided((M, K), (8, 1)), w, out, False
    yield "off a 16-byte boundary", wide[:, 1:1 + K], w, out, False
    yield "transposed out", x, w, torch.zeros(N, M).bfloat16().t(), False
    yield "one place for all of out", x, w, torch.zeros(1, N).bfloat16().expand(M, N), False
    yield "out of another shape", x, w, torch.zeros(M, N + 8).bfloat16(), False
    yield "no sum", x[:, :0], w[:, :0], out, False
    yield "no column", x, w[:0], out[:, :0], False
    yield "another length", x[:, :64], w, out, False
    yield "another type", x, w.float(), out, False
    yield "half precision out", x, w, out.half(), False


@pytest.mark.parametrize("name,x,w,out,taken", [pytest.param(*f, id=f[0]) for f in _forms()])
def test_forms(name, x, w, out, taken):
    assert ops.rows_ok(x, w, out, w.shape[0]) == taken
    if taken:
        assert ops.rows_ok(x, w)


def test_devices():
    w = torch.zeros(N, K).bfloat16()
    w.get_device = lambda: 1
    assert not ops.rows_ok(torch.zeros(M, K).bfloat16(), w)
