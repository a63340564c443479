"""The experts' tcgen05 products by pairs of CTAs: runs of places at the edges of tiles, columns that do not fill one, the gated unit
in the epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
RUNS = [[1], [256], [0, 257, 0], [31, 32, 33, 0, 1, 300], [512, 513], [0, 0, 5]]


def _case(runs, N, K, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    normal = lambda *s: torch.randn(*s, generator=g, device=DEV).bfloat16()
    offsets = torch.tensor([0] + runs, device=DEV).cumsum(0).to(torch.int32)
    return normal(sum(runs), K), normal(len(runs), N, K) * K ** -0.5, offsets


def _products(x, w, offsets):
    out = torch.empty(x.shape[0], w.shape[1], dtype=torch.float64, device=DEV)
    for e, (a, b) in enumerate(zip(offsets[:-1].tolist(), offsets[1:].tolist())):
        out[a:b] = x[a:b].double() @ w[e].double().T
    return out


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("N,K,pad,act", [(256, 64, 0, None), (264, 136, 0, "relu2"), (40, 1032, 3, None), (1000, 128, 0, "silu")])
def test_moe_tc5_gemm(runs, N, K, pad, act):
    from return_b200.ext import ops
    x, w, offsets = _case(runs, N, K, N + len(runs))
    out = torch.full((x.shape[0], N + pad), float("nan"), dtype=torch.bfloat16, device=DEV)[:, :N]         # rows off 16 bytes
    ops.moe_tc5_gemm(x, w, offsets, out, act)
    ops.check_status(DEV)
    want = _products(x, w, offsets)
    want = {None: want, "relu2": want.clamp(min=0) ** 2, "silu": want * torch.sigmoid(want)}[act]
    # one rounding to bfloat16 of a float32 sum of order one
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -12).all()


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("F,K,weighed", [(128, 64, False), (72, 136, True), (200, 1032, False)])
def test_moe_tc5_gated(runs, F, K, weighed):
    from return_b200.ext import ops
    x, w, offsets = _case(runs, 2 * F, K, F + len(runs))
    n = x.shape[0]
    weight, pair_at = torch.rand(n, device=DEV), torch.randperm(n, device=DEV).to(torch.int32)
    out = torch.full((n, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.moe_tc5_gated(x, w, offsets, out, 1.5, 1.702, 1.0, weight if weighed else None, pair_at if weighed else None)
    ops.check_status(DEV)
    s = _products(x, w, offsets) * (weight[pair_at.long()].double()[:, None] if weighed else 1.0)
    g, u = s[:, :F].clamp(max=1.5), s[:, F:].clamp(-1.5, 1.5)
    want = g * torch.sigmoid(1.702 * g) * (u + 1.0)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -12).all()


def test_moe_tc5_gated_unit_keeps_float32():
    """The unit alone, of sums that are exact: rounded to bfloat16 it is the rounded 64-bit value but where that lies next to the middle
    between two bfloat16 numbers.  Four float32 roundings of 2^-24 against a spacing of 2^-8 to 2^-7: one in some 4,000 at most; an exponential
    that loses bits with the size of its argument would miss thirty times as many."""
    from return_b200.ext import ops
    F, K = 1024, 64
    g = torch.Generator(device=DEV).manual_seed(0)
    gate = (torch.rand(F, K, generator=g, device=DEV) * 67 - 60).bfloat16()
    up = torch.randn(F, K, generator=g, device=DEV).bfloat16()
    x, w = torch.eye(K, device=DEV).bfloat16(), torch.cat([gate, up])[None].contiguous()            # place k takes column k
    out = torch.empty(K, F, dtype=torch.bfloat16, device=DEV)
    ops.moe_tc5_gated(x, w, torch.tensor([0, K], dtype=torch.int32, device=DEV), out, 7.0, 1.0, 1.0)
    ops.check_status(DEV)
    a, b = gate.T.double().clamp(max=7.0), up.T.double().clamp(-7.0, 7.0)
    want = a * torch.sigmoid(a) * (b + 1.0)
    missed = (out != want.to(torch.bfloat16)).double().mean().item()
    assert missed <= 1.0 / 4000, missed
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs()).all()
