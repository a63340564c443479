"""The product for the rows of an ordinary step at the edges of its tiles, stages and shares of K."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ops():
    from return_b200.ext import ops
    return ops


def _inputs(M, N, K, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.empty(M, K + 8, device=DEV).normal_(generator=g).bfloat16()[:, :K]          # rows apart by more than their length
    w = torch.empty(N, K, device=DEV).normal_(std=0.05, generator=g).bfloat16()
    return x, w, x.double() @ w.double().T, x.double().abs() @ w.double().abs().T


def _close(got, exact, size, K, scale=1.0):
    """float32 sums of K products (K / 16 of them cut off), and one rounding to the output's type."""
    unit = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -24
    assert ((got.double() - exact).abs() <= scale * (exact.abs() * unit + size * (K / 16 + 4) * 2.0 ** -23)).all()


@pytest.mark.parametrize("M,N,K", [(9, 16, 8), (16, 128, 64), (17, 129, 128), (33, 96, 136), (64, 257, 192), (130, 384, 320), (255, 130, 1024), (257, 200, 512),
                                   (513, 64, 2048)])
@pytest.mark.parametrize("f32", [False, True])
def test_tiles_and_shares(M, N, K, f32):
    ops = _ops()
    x, w, exact, size = _inputs(M, N, K, M + K)
    wide = torch.full((M, N + 24), 7.0, device=DEV, dtype=torch.float32 if f32 else torch.bfloat16)
    least = (M + 255) // 256
    for tiles, ls in [(-1, -1)] + [(t, l) for t in (least, least + 1, least + 3) for l in (0, 1, 2)]:
        for shift in (0, 1):                                  # output rows of whole 16-byte pieces, and not
            wide.fill_(7.0)
            out = wide[:, 8 + shift:8 + shift + N]
            ops.gemm_rows(x, w, out, tiles=tiles, log2_split=ls)
            _close(out, exact, size, K)
            assert (wide[:, :8 + shift] == 7.0).all() and (wide[:, 8 + shift + N:] == 7.0).all()
    ops.check_status(x.device)


@pytest.mark.parametrize("gate", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("M,N,K", [(9, 32, 64), (100, 272, 320), (300, 512, 1024)])
def test_gated_unit(M, N, K, gate):
    ops = _ops()
    x, w, exact, size = _inputs(M, N, K, M)
    g, u = exact.view(M, -1, 2, 8).unbind(2)
    a = g * torch.sigmoid(g) if gate == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    want = (a * u).reshape(M, N // 2)
    bound = size.view(M, -1, 2, 8).amax(2).reshape(M, N // 2) * (1 + exact.abs().view(M, -1, 2, 8).amax(2).reshape(M, N // 2))
    for ls in (-1, 0, 2):
        out = torch.full((M, N // 2), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.gemm_rows(x, w, out, gated=True, act=gate, tiles=-1 if ls < 0 else (M + 255) // 256, log2_split=ls)
        _close(out, want, bound, K, 2.5)                      # (the unit's slope is at most 1.13 times the other factor, of each of the two sums)
    ops.check_status(x.device)


@pytest.mark.parametrize("act", ["relu2", "tanh", "gelu_tanh", "silu"])
def test_activation_on_the_sums(act):
    ops = _ops()
    x, w, exact, _ = _inputs(70, 136, 256, 4)
    f = {"relu2": lambda v: torch.relu(v) ** 2, "tanh": torch.tanh, "silu": lambda v: v * torch.sigmoid(v),
         "gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act]
    want = f(exact)
    assert ops.rows_ok(x, w)
    for product in (ops.gemm_rows, ops.linear):               # the kernel, and the way to it
        out = torch.full((70, 136), float("nan"), device=DEV, dtype=torch.bfloat16)
        product(x, w, out, act=act)
        assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()
    ops.check_status(x.device)


def test_what_the_kernel_does_not_take_goes_to_the_library():
    ops = _ops()
    x, w, exact, size = _inputs(40, 100, 100, 5)              # K is no multiple of eight
    assert not ops.rows_ok(x, w)
    out = torch.empty(40, 100, device=DEV, dtype=torch.bfloat16)
    ops.linear(x, w, out)
    _close(out, exact, size, 100)


@pytest.mark.parametrize("M,H,Q,I,offset,wdt", [(9, 96, 64, 48, 0.0, torch.float32), (33, 136, 136, 128, 1.0, torch.bfloat16), (130, 1024, 512, 200, 0.0, torch.bfloat16),
                                                (257, 264, 1024, 64, 0.5, torch.float32)])
def test_norms_and_residual_adds_inside_the_products(M, H, Q, I, offset, wdt):
    """Product + residual add, then the gated and a plain product on the rows it left, each step against 64 bits from what the step before it
    really left."""
    ops = _ops()
    o, w_o, exact, size = _inputs(M, H, Q, M + H)
    g = torch.Generator(device=DEV).manual_seed(M)
    stream0 = torch.empty(M, H, device=DEV).normal_(std=2.0, generator=g)
    norm = torch.empty(H, device=DEV).normal_(generator=g).to(wdt)
    woven = torch.empty(2 * I, H, device=DEV).normal_(std=0.05, generator=g).bfloat16()
    eps, tiles_n = 1e-5, (H + 127) // 128
    least = (M + 255) // 256
    for tiles, ls in [(-1, -1)] + [(t, l) for t in (least, least + 2) for l in (0, 1, 2)]:
        shape = dict(tiles=tiles, log2_split=ls)
        stream, rows = stream0.clone(), torch.full((M, H), float("nan"), device=DEV, dtype=torch.bfloat16)
        sums = ops.RowSums(torch.full((M, tiles_n), float("nan"), device=DEV), H)
        ops.gemm_rows_fused(o, w_o, rows, residual=(stream, (norm, offset), sums), **shape)
        only = stream0.clone()
        ops.gemm_rows_fused(o, w_o, None, residual=(only, None, None), **shape)
        assert torch.equal(only, stream)
        want = stream0.double() + exact
        assert ((stream.double() - want).abs() <= want.abs() * 2.0 ** -23 + size * (Q / 16 + 4) * 2.0 ** -23).all()
        left = stream.double() * (norm.double() + offset)
        assert ((rows.double() - left).abs() <= left.abs() * (2.0 ** -8 + 2.0 ** -21) + 1e-37).all()
        ssq = stream.double().square().sum(1)
        assert sums.count == tiles_n
        assert ((sums.parts[:, :tiles_n].double().sum(1) - ssq).abs() <= ssq * 16 * 2.0 ** -23).all()
        # the rows it left, times the norm's factor: eight products' and three more roundings of the factor
        rstd = (1.0 / (ssq / H + eps).sqrt())[:, None]
        p, psize = rows.double() @ woven.double().T * rstd, rows.double().abs() @ woven.double().abs().T * rstd
        plain = torch.full((M, 2 * I), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.gemm_rows_fused(rows, woven, plain, scale=(sums, eps), **shape)
        _close(plain, p, psize + p.abs(), H + 64)
        gate, up = p.view(M, -1, 2, 8).unbind(2)
        err = ((psize + p.abs()) * ((H + 64) / 16 + 4) * 2.0 ** -23).view(M, -1, 2, 8)
        unit = gate * torch.sigmoid(gate)
        act = torch.full((M, I), float("nan"), device=DEV, dtype=torch.bfloat16)
        ops.gemm_rows_fused(rows, woven, act, gated=True, scale=(sums, eps), **shape)
        tol = 1.1 * err[:, :, 0] * up.abs() + (unit.abs() + 1.1 * err[:, :, 0]) * err[:, :, 1] + (unit * up).abs() * (2.0 ** -8 + 2.0 ** -20) + 1e-37
        assert ((act.double() - (unit * up).reshape(M, I)).abs() <= tol.reshape(M, I)).all()
        # and a product that scales and adds at once
        again = stream.clone()
        ops.gemm_rows_fused(rows[:, :H], w_back := woven[:H] if 2 * I >= H else woven.repeat(H // (2 * I) + 1, 1)[:H].contiguous(), None,
                            scale=(sums, eps), residual=(again, None, None), **shape)
        q, qsize = rows.double() @ w_back.double().T * rstd, rows.double().abs() @ w_back.double().abs().T * rstd
        want = stream.double() + q
        assert ((again.double() - want).abs() <= want.abs() * 2.0 ** -23 + (qsize + q.abs()) * ((H + 64) / 16 + 4) * 2.0 ** -23).all()
    ops.check_status(torch.device("cuda:0"))


def test_products_refuse_what_they_cannot_take():
    """Before anything is launched: each is an error of the entry itself."""
    ops = _ops()
    x, w = torch.zeros(16, 64, device=DEV).bfloat16(), torch.zeros(128, 64, device=DEV).bfloat16()
    out, stream, norm = torch.zeros(16, 128, device=DEV).bfloat16(), torch.zeros(16, 128, device=DEV), torch.ones(128, device=DEV)
    sums = ops.RowSums(torch.zeros(16, 1, device=DEV), 128)
    ops.gemm_rows_fused(x, w, out, residual=(stream, (norm, 0.0), sums))
    def zeros(*shape):
        return torch.zeros(*shape, device=DEV).bfloat16()

    refused = [
        # a row of the stream is no whole 16-byte pieces; K is no multiple of 8; rows lie off 16-byte boundaries
        lambda: ops.gemm_rows_fused(x, zeros(130, 64), None, residual=(torch.zeros(16, 130, device=DEV), None, None)),
        lambda: ops.gemm_rows(x[:, :60], w[:, :60], out),
        lambda: ops.gemm_rows(x[:, 1:57], w[:, :56], out),
        # a tile of 300 rows; a cluster of eight CTAs; gate and up rows in no whole blocks
        lambda: ops.gemm_rows(zeros(300, 64), w, zeros(300, 128), tiles=1, log2_split=0),
        lambda: ops.gemm_rows(x, w, out, tiles=1, log2_split=3),
        lambda: ops.gemm_rows_fused(x, zeros(136, 64), out[:, :68], gated=True, scale=(sums, 1e-6)),
    ]
    for call in refused:
        with pytest.raises(ops.KernelError):
            call()
    narrow = ops.RowSums(torch.zeros(16, 1, device=DEV), 256)
    gaps = torch.zeros(16, 129, device=DEV)[:, :128]
    refused = [
        # room for one share a row instead of two; a stream with gaps; a next norm and nowhere to put its rows
        lambda: ops.gemm_rows_fused(x, zeros(256, 64), None, residual=(torch.zeros(16, 256, device=DEV), None, narrow)),
        lambda: ops.gemm_rows_fused(x, w, None, residual=(gaps, None, None)),
        lambda: ops.gemm_rows_fused(x, w, None, residual=(stream, (norm, 0.0), None)),
    ]
    for call in refused:
        with pytest.raises(AssertionError):
            call()
    ops.check_status(x.device)


def test_operands_that_only_the_library_takes():
    """Strides and sizes that go past the kernel: as ``torch.mm`` takes them."""
    ops = _ops()
    M, N, K = 40, 64, 128
    x, w, _, _ = _inputs(M, N, K, 6)
    x = x.contiguous()
    wide = torch.randn(M, 2 * K, device=DEV).bfloat16()
    row_out = torch.empty(N, M, device=DEV, dtype=torch.bfloat16).t()
    forms = [(x, w.t().contiguous().t(), None), (x.t().contiguous().t(), w, None), (wide[:, ::2], w, None), (x[:1].expand(M, K), w, None),
             (wide.reshape(-1).as_strided((M, K), (8, 1)), w, None), (x, w[:1].expand(N, K), None), (x, w, row_out), (x[:, :0], w[:, :0], None), (x, w[:0], None)]
    for i, (a, b, out) in enumerate(forms):
        for dtype in (torch.bfloat16, torch.float32) if out is None else (torch.bfloat16,):
            o = torch.full((M, b.shape[0]), 7.0, device=DEV, dtype=dtype) if out is None else out
            ops.linear(a, b, o)
            _close(o, a.double() @ b.double().T, a.double().abs() @ b.double().abs().T, K)
    unit = torch.empty(M, N // 2, device=DEV, dtype=torch.bfloat16)
    ops.gated_linear(x.t().contiguous().t(), w, unit, 8)
    want = torch.empty_like(unit)
    ops.gated_linear(x, w, want, 8)
    assert (unit.float() - want.float()).norm() <= 2e-2 * want.float().norm()       # (the library's way rounds the two sums to bfloat16 first)
    with pytest.raises(Exception):
        ops.linear(x, w, torch.empty(1, N, device=DEV, dtype=torch.bfloat16).expand(M, N))


def test_clusters_share_an_sm_only_where_all_find_tensor_memory():
    """Tiles of 144 rows hold 256 columns of tensor memory in few bytes of shared memory (one stage): more CTAs than SMs, in clusters."""
    ops = _ops()
    x, w, exact, size = _inputs(144, 128 * 400, 256, 3)
    for ls in (1, 2):
        out = torch.empty(144, 128 * 400, device=DEV)
        ops.gemm_rows(x, w, out, tiles=1, log2_split=ls)
        _close(out, exact, size, 256)
    ops.check_status(x.device)


def test_shapes_fill_the_device_once():
    """A device holds fewer CTAs in fours than it has SMs.  A product that fits it in one round of another shape does not take two of these."""
    ops = _ops()
    for N in (768, 1024, 1152, 1536, 2048, 3072, 4608):
        for K in (1024, 2048, 4096):
            for M in range(16, 257, 16):
                tiles, ls, ctas, held = ops.gemm_rows_plan(M, N, K)
                assert ctas == tiles * ((N + 127) // 128) << ls and ctas <= held, (M, N, K, tiles, ls, ctas, held)
    with pytest.raises(ops.KernelError):
        ops.gemm_rows_plan(16, 128, 0)
