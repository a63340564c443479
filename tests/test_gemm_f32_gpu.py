"""The float32 product's shapes at the edges of its tiles, runs and groups, and what numbers without parts do."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ops():
    from return_b200.ext import ops
    return ops


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (16, 129, 65), (17, 1, 511), (64, 127, 512), (65, 128, 576), (80, 256, 1024), (81, 130, 1088), (163, 384, 260),
                                   (257, 128, 3072)])
@pytest.mark.parametrize("offset", [0, 1])
def test_every_shape_gives_the_same_bits(M, N, K, offset):
    """K around whole blocks of 64, runs of two and four groups of them; M around the tiles' widths.  Three of nine products are left out (each at
    most 2^-24 of its term), a run of 128 values is cut off and not rounded (at most 8 + 5 times 2^-23 of its terms' sizes), and
    the sums of runs and groups round once each."""
    ops = _ops()
    torch.manual_seed(M * 7 + K)
    wide = torch.randn(M + N, K + 3, device=DEV)
    x, w = wide[:M, offset:offset + K], wide[M:, offset:offset + K]
    if offset == 0 and K % 4 == 0:
        x, w = x.contiguous(), w.contiguous()
    outs = []
    for kind in range(-1, 12):
        outs.append(torch.full((M, N), float("nan"), device=DEV))
        ops.gemm_f32(x, w, outs[-1], kind=kind)
        assert torch.equal(outs[-1], outs[0]), kind
    ops.check_status(x.device)
    exact = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    roundings = 3 * 2.0 ** -24 + 13 * 2.0 ** -23 + (K / 128 + 4) * 2.0 ** -24
    assert ((outs[0].double() - exact).abs() <= size * roundings).all()


@pytest.mark.parametrize("K", [40, 96, 97, 128, 200, 512, 1024])
def test_error_is_below_a_chain_of_multiply_adds(K):
    """Short sums (up to 96 values) are such a chain; the others' errors are smaller."""
    ops = _ops()
    torch.manual_seed(5)
    x, w = torch.randn(33, K, device=DEV), torch.randn(200, K, device=DEV)
    out = torch.empty(33, 200, device=DEV)
    ops.gemm_f32(x, w, out)
    exact = x.double() @ w.double().T
    acc = torch.zeros(33, 200, device=DEV)
    for k in range(K):                                        # float32(float64 product + sum): one rounding, as fused
        acc = (acc.double() + x[:, k:k + 1].double() * w[:, k].double()).float()
    if K <= 96:
        assert torch.equal(out, acc)
    else:
        assert (out.double() - exact).norm() < (acc.double() - exact).norm()


@pytest.mark.parametrize("kind", [-1, 0, 4, 8, 11])
def test_numbers_without_parts(kind):
    """Infinities, NaNs and numbers next to the largest: their rows and columns hold what a chain of float32 products and sums
    holds, and nothing else changes."""
    ops = _ops()
    torch.manual_seed(3)
    M, N, K = 40, 140, 320
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    plain = torch.empty(M, N, device=DEV)
    ops.gemm_f32(x, w, plain, kind=kind)
    inf, big = float("inf"), 3.4e38
    x[3, 17], x[7, 100], x[9, 5], x[11, 64] = inf, float("nan"), -inf, big
    w[64, 3], w[139, 200], w[2, 64] = -inf, float("nan"), 0.25
    w[5, 17] = 0.0                                            # inf * 0
    out = torch.empty(M, N, device=DEV)
    ops.gemm_f32(x, w, out, kind=kind)
    rows, cols = [3, 7, 9, 11], [64, 139]
    keep_r = [i for i in range(M) if i not in rows]
    keep_c = [i for i in range(N) if i not in cols and i not in (2, 5)]
    assert torch.equal(out[keep_r][:, keep_c], plain[keep_r][:, keep_c])
    want = x.double() @ w.double().T                          # (3.4e38 times a normal weight may pass float32's range)
    for r in rows:
        far = want[r].abs() > 3.4028235e38
        want[r] = torch.where(far & want[r].isfinite(), torch.copysign(torch.full_like(want[r], inf), want[r]), want[r])
    got = out.double()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert ((got - want).abs()[fine] <= 1e-4 * want.abs()[fine] + 1e-3).all()


@pytest.mark.parametrize("x_up,w_up", [(-120, 100), (-60, 60), (-140, 110), (-110, -25), (90, 3)])
@pytest.mark.parametrize("kind", [-1, 0, 5, 11])
def test_small_and_large_operands_keep_their_24_bits(x_up, w_up, kind):
    """Powers of two times ordinary operands, down to numbers with fewer bits than 24 and products next to the smallest.  Where nothing leaves
    the range the bits are those of the ordinary operands, and everywhere the error is theirs (and a rounding to float32's smallest
    step for a result that small)."""
    ops = _ops()
    torch.manual_seed(9)
    M, N, K = 37, 130, 260
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV).clamp(-3.9, 3.9)
    plain, out = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_f32(x, w, plain, kind=kind)
    xs, ws = (x.double() * 2.0 ** x_up).float(), (w.double() * 2.0 ** w_up).float()
    ops.gemm_f32(xs, ws, out, kind=kind)
    ops.check_status(x.device)
    if x_up > -100 and x_up + w_up < 90:
        assert torch.equal(out.double(), plain.double() * 2.0 ** (x_up + w_up))
    exact, size = xs.double() @ ws.double().T, xs.double().abs() @ ws.double().abs().T
    roundings = 3 * 2.0 ** -24 + 13 * 2.0 ** -23 + (K / 128 + 4) * 2.0 ** -24
    if x_up == 90:                                            # sums beyond 2^96: a chain of K fused multiply-adds
        roundings = K * 2.0 ** -24
    assert ((out.double() - exact).abs() <= size * roundings + 2.0 ** -149).all()
    assert exact.abs().max() > 0 and torch.isfinite(out).all()


def test_rows_far_apart():
    """32 rows times their stride pass 31 bits.  (The rows lie in 9 GB of which only they are touched.)"""
    ops = _ops()
    torch.manual_seed(1)
    M, N, K, ld = 34, 130, 128, 1 << 26
    far = torch.empty(ld * (M - 1) + K, device=DEV).as_strided((M, K), (ld, 1))
    near, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    far.copy_(near)
    out, want = torch.full((M, N), float("nan"), device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_f32(near, w, want)
    ops.gemm_f32(far, w, out)
    assert torch.equal(out, want)
    out = torch.full((N, M), float("nan"), device=DEV)
    ops.gemm_f32(w, far, out)                                 # as weight rows
    assert (out - want.t()).abs().max() <= 1e-4
    ops.check_status(far.device)


def test_more_rows_than_a_launch_has_tiles():
    ops = _ops()
    torch.manual_seed(2)
    M, K = 65535 * 16 + 19, 100
    x, w = torch.randn(M, K, device=DEV), torch.randn(3, K, device=DEV)
    for kind in (-1, 9):
        out = torch.full((M, 3), float("nan"), device=DEV)
        ops.gemm_f32(x, w, out, kind=kind)
        ends = torch.cat((torch.arange(40), torch.arange(65535 * 16 - 40, M))).to(DEV)
        want = torch.empty(len(ends), 3, device=DEV)
        ops.gemm_f32(x[ends], w, want, kind=kind)
        assert torch.equal(out[ends], want) and torch.isfinite(out).all()
    ops.check_status(x.device)


@pytest.mark.parametrize("K", [132, 188, 196, 252, 316, 1000])
def test_rows_of_whole_pieces_of_four(K):
    """They are fetched 16 bytes at a time and give the bits that they give one value at a time; what lies behind a row is not read."""
    ops = _ops()
    torch.manual_seed(K)
    M, N = 85, 140
    wide = torch.full((M + N, K + 4), float("nan"), device=DEV)
    wide[:, :K] = torch.randn(M + N, K, device=DEV)
    x, w = wide[:M, :K], wide[M:, :K]
    off = torch.empty((M + N) * (K + 4) + 1, device=DEV)[1:].view(M + N, K + 4)
    off.copy_(wide)
    for kind in (-1, 0, 4, 11):
        out, want = torch.full((M, N), float("nan"), device=DEV), torch.empty(M, N, device=DEV)
        ops.gemm_f32(x, w, out, kind=kind)
        ops.gemm_f32(off[:M, :K], off[M:, :K], want, kind=kind)
        assert torch.equal(out, want) and torch.isfinite(out).all()
    ops.check_status(x.device)
