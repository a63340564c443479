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
    yield "gated", x, w, out[:, :N // 2], None
    yield "no sum", x[:, :0], w[:, :0], out, False
    yield "no column", x, w[:0], out[:, :0], False
    yield "another length", x[:, :64], w, out, False
    yield "another type", x, w.float(), out, False
    yield "half precision out", x, w, out.half(), False


@pytest.mark.parametrize("name,x,w,out,taken", [pytest.param(*f, id=f[0]) for f in _forms()])
def test_forms(name, x, w, out, taken):
    if taken is None:
        assert ops.rows_ok(x, w, out, gated=True) and not ops.rows_ok(x, w, out)
        return
    assert ops.rows_ok(x, w, out) == taken
    if taken:
        assert ops.rows_ok(x, w)


def test_devices():
    w = torch.zeros(N, K).bfloat16()
    w.get_device = lambda: 1
    assert not ops.rows_ok(torch.zeros(M, K).bfloat16(), w)


def _rows_taken(N, K, gated=False):
    """The most rows of an N x K product that the rule gives to the kernel."""
    w = torch.empty(N, K, device="meta", dtype=torch.bfloat16)
    taken = [M for M in range(9, 1100) if ops.rows_ok(torch.empty(M, K, device="meta", dtype=torch.bfloat16), w, gated=gated)]
    assert taken == list(range(9, 9 + len(taken)))            # one stretch from the first rows that the weight-streaming kernel leaves
    return taken[-1] if taken else 0


# (N, K): rows launch by launch, and captured
@pytest.mark.parametrize("gated,N,K,eager,captured", [(False, 4096, 1024, 825, 0), (False, 2048, 2048, 825, 0), (False, 1024, 3072, 1024, 64), (False, 2048, 6144, 275, 64),
                                                      (False, 4096, 12288, 128, 64), (False, 6144, 4096, 0, 0), (False, 64, 1024, 1024, 0), (False, 512, 2048, 1024, 0),
                                                      (True, 6144, 1024, 550, 64), (True, 8192, 2048, 206, 64), (True, 24576, 1024, 0, 0)])
def test_limits_at_their_edges(gated, N, K, eager, captured):
    assert _rows_taken(N, K, gated) == eager
    with ops.captured_step():
        assert _rows_taken(N, K, gated) == captured
    assert _rows_taken(N, K, gated) == eager


def test_a_layer_has_the_limit_of_its_least_product():
    limits = [ops.rows_limit(*s) for s in ((4096, 1024), (1024, 2048), (6144, 1024), (1024, 3072))]
    assert limits == [825, 1024, 550, 1024] and ops.layer_rows_limit(min(limits)) == 550
    with ops.captured_step():
        assert ops.layer_rows_limit(550) == 128 and ops.layer_rows_limit(100) == 100


def test_a_captured_step_is_its_threads_own():
    import threading
    seen = []
    with pytest.raises(ValueError):
        with ops.captured_step():
            t = threading.Thread(target=lambda: seen.append(ops.layer_rows_limit(550)))
            t.start()
            t.join()
            raise ValueError
    assert seen == [550] and ops.layer_rows_limit(550) == 550
