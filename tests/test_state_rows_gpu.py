"""The row kernels around a scan, four elements a lane, against the element-by-element kernels that take everything else.  The
latter are reached through operands that lie off the addresses the former need."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _ops():
    from return_b200.ext import ops
    return ops


def off_by_one(x):
    """The same numbers one element further on in a wider buffer."""
    wide = torch.zeros(x.shape[0], x.shape[1] + 3, dtype=x.dtype, device=x.device)
    wide[:, 1:1 + x.shape[1]] = x
    return wide[:, 1:1 + x.shape[1]]


# sums over a head in two orders and a rounding or two of the result
def same(a, b, dt):
    tol = 2.0 ** -17 if dt == torch.float32 else 2.0 ** -7
    return torch.allclose(a.float(), b.float(), rtol=tol, atol=tol)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,D", [(1, 8), (3, 40), (16, 128), (2, 256)])
def test_rotary_to_f32(dt, heads, D):
    ops = _ops()
    T, HD = 37, heads * D
    x = torch.randn(T, 2 * HD, device=DEV).to(dt)
    ang = torch.rand(50, D // 2, device=DEV) * 6
    pos = torch.randint(0, 50, (T,), dtype=torch.int32, device=DEV)
    outs = []
    for form in (lambda y: y, off_by_one):
        q, k = torch.empty(T, HD, device=DEV), torch.empty(T, HD, device=DEV)
        ops.rotary_to_f32(form(x), 0, HD, ang.cos().contiguous(), ang.sin().contiguous(), D, pos, q, k, heads, D, 1.0, D ** -0.5)
        outs.append((q, k))
    assert same(outs[0][0], outs[1][0], torch.float32) and same(outs[0][1], outs[1][1], torch.float32)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,V", [(1, 4), (5, 60), (16, 128), (3, 132), (2, 256)])
@pytest.mark.parametrize("mode,act", [(0, 0), (1, 1), (2, 0)])
def test_head_norm_gate(dt, H, V, mode, act):
    ops = _ops()
    T = 19
    o, gate = torch.randn(T, H * V, device=DEV), torch.randn(T, H * V, device=DEV).to(dt)
    w = (None, torch.rand(V, device=DEV), torch.rand(H * V, device=DEV).to(dt))[mode]
    outs = []
    for form in (lambda y: y, off_by_one):
        out = torch.empty(T, H * V, device=DEV, dtype=dt)
        ops.head_norm_gate(o, form(gate), w, mode, act, 1e-5, out, H, V)
        outs.append(out)
    assert same(outs[0], outs[1], dt)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", [[1, 1, 5, 2], [3, 1030], [9] * 120])
@pytest.mark.parametrize("H,G,D,V,K,head_decay", [(4, 2, 8, 12, 4, False), (2, 1, 128, 256, 2, True), (2, 2, 36, 132, 1, False), (1, 1, 256, 4, 3, True)])
def test_delta_prep(dt, lens, H, G, D, V, K, head_decay):
    """Runs of tokens that begin within a segment, at its start and over several segments, with what the state holds before them."""
    ops = _ops()
    T, n, C = sum(lens), len(lens), 2 * G * D + H * V
    x, taps = torch.randn(T, C, device=DEV).to(dt), torch.randn(C, K, device=DEV).to(dt)
    DA = 1 if head_decay else D
    a, b = torch.randn(T, H * DA, device=DEV), torch.randn(T, H, device=DEV)
    A_log, dt_bias = torch.randn(H, device=DEV).to(dt), torch.randn(H * DA, device=DEV).to(dt)
    state = torch.randn(n, 1 + C * (K - 1), device=DEV)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    batch = SimpleNamespace(cu_q=cu, seg_slot=torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEV),
                            tok_seg=torch.repeat_interleave(torch.arange(n, device=DEV), torch.tensor(lens, device=DEV)).to(torch.int32))
    outs = []
    for form in (lambda y: y, off_by_one):
        out = [torch.empty(T, w, device=DEV) for w in (G * D, G * D, H * V)] + [a.clone(), b.clone()]
        ops.delta_prep(form(x), taps, state, 1, batch, out[0], out[1], out[2], out[3], A_log, dt_bias, out[4], H, G, D, V, D ** -0.5,
                       head_decay=head_decay)
        outs.append(out)
    assert all(same(p, q, torch.float32) for p, q in zip(*outs))


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,D,V,K", [(4, 2, 8, 12, 4), (2, 1, 128, 256, 2)])
def test_delta_prep_bits_do_not_depend_on_the_step(dt, H, G, D, V, K):
    """Steps of 1,024 tokens and more take runs of tokens a warp: the same bits as a segment alone."""
    ops = _ops()
    lens, C = [531, 2, 600], 2 * G * D + H * V
    T, n = sum(lens), len(lens)
    x, taps = torch.randn(T, C, device=DEV).to(dt), torch.randn(C, K, device=DEV).to(dt)
    a, b = torch.randn(T, H * D, device=DEV), torch.randn(T, H, device=DEV)
    A_log, dt_bias = torch.randn(H, device=DEV).to(dt), torch.randn(H * D, device=DEV).to(dt)
    state = torch.randn(n, C * (K - 1), device=DEV)

    def run(segs):
        rows = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in segs]).to(DEV)
        sizes = torch.tensor([lens[i] for i in segs], device=DEV)
        batch = SimpleNamespace(cu_q=torch.nn.functional.pad(sizes.cumsum(0), (1, 0)).to(torch.int32), seg_slot=torch.tensor(segs, dtype=torch.int32, device=DEV),
                                tok_seg=torch.repeat_interleave(torch.arange(len(segs), device=DEV), sizes).to(torch.int32))
        out = [torch.empty(len(rows), w, device=DEV) for w in (G * D, G * D, H * V)] + [a[rows], b[rows]]
        ops.delta_prep(x[rows], taps, state, 0, batch, out[0], out[1], out[2], out[3], A_log, dt_bias, out[4], H, G, D, V, D ** -0.5)
        return out

    whole, apart = run([0, 1, 2]), [run([i]) for i in range(n)]
    assert all(torch.equal(w, torch.cat(parts)) for w, parts in zip(whole, zip(*apart)))


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,D,V,K", [(4, 2, 8, 12, 4), (2, 1, 128, 256, 2), (2, 2, 36, 132, 1), (1, 1, 20, 4, 3)])
def test_delta_prep_moves_conv_states_of_single_tokens(dt, H, G, D, V, K):
    """The same numbers as the two kernels one after the other, in both forms, with a slot of no request between."""
    ops = _ops()
    T, C = 7, 2 * G * D + H * V
    x, taps = torch.randn(T, C, device=DEV).to(dt), torch.randn(C, K, device=DEV).to(dt)
    a, b = torch.randn(T, H * D, device=DEV), torch.randn(T, H, device=DEV)
    A_log, dt_bias = torch.randn(H, device=DEV).to(dt), torch.randn(H * D, device=DEV).to(dt)
    state = torch.randn(T + 1, 2 + C * (K - 1), device=DEV)
    i32 = lambda y: torch.as_tensor(y, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(cu_q=i32(list(range(T + 1))), seg_slot=i32([7, 0, 3, 1, 6, 2, 5]), tok_seg=i32(list(range(T))), num_segments=T)
    for form in (lambda y: y, off_by_one):
        outs = []
        for fused in (False, True):
            out, st = [torch.empty(T, w, device=DEV) for w in (G * D, G * D, H * V)] + [a.clone(), b.clone()], state.clone()
            ops.delta_prep(form(x), taps, st, 2, batch, out[0], out[1], out[2], out[3], A_log, dt_bias, out[4], H, G, D, V, D ** -0.5,
                           update_state=fused)
            if not fused:
                ops.conv_state_update(form(x), K, st, 2, batch, C)
            outs.append(out + [st])
        assert all(torch.equal(p, q) for p, q in zip(*outs))


@pytest.mark.parametrize("mode", ["DECAY", "DELTA", "BONUS", "SSM", "DELTA_HEAD"])
@pytest.mark.parametrize("n,H,G,D,V,off", [(1, 2, 1, 128, 128, 0), (5, 4, 2, 24, 40, 4), (3, 2, 2, 100, 144, 0), (2, 3, 3, 64, 7, 8)])
def test_scan_of_single_tokens(mode, n, H, G, D, V, off):
    """The kernel for segments of one token beside the walk: the same sums of up to 128 products in another order."""
    ops = _ops()
    m = getattr(ops, "SCAN_" + mode)
    normal = lambda *s: torch.randn(*s, device=DEV)
    q, k, v = normal(n, G * D) * D ** -0.5, torch.nn.functional.normalize(normal(n, G, D), dim=-1).reshape(n, -1), normal(n, H * V).bfloat16()
    gate_a = torch.rand({"DECAY": (H,), "DELTA": (n, H * D), "BONUS": (n, H * D)}.get(mode, (n, H)), device=DEV)
    gate_b = torch.rand(n, H, device=DEV) if mode in ("DELTA", "DELTA_HEAD", "SSM") else None
    extra = normal(H, D) if mode == "BONUS" else normal(H) if mode == "SSM" else None
    state = normal(n + 1, off + (H * ((D + 7) // 8 * 8) * V + 3) // 4 * 4)
    batch = SimpleNamespace(cu_q=torch.arange(n + 1, dtype=torch.int32, device=DEV), num_segments=n,
                            seg_slot=torch.arange(n, 0, -1, dtype=torch.int32, device=DEV))
    outs = []
    for single in (False, True):
        st, out = state.clone(), torch.empty(n, H * V, device=DEV)
        ops.linear_scan(m, q, k, v, gate_a, gate_b, st, (off, 0, 0), batch, out, H, G, D, V, extra=extra, single=single)
        outs.append((out, st))
    rows = (D + 7) // 8 * 8
    if rows != D:                                             # rows that do not exist are zero in a real state; here they hold anything
        keep = torch.ones(H, rows // 8, V, 8, dtype=torch.bool, device=DEV)
        keep[:, -1, :, D % 8:] = False
        outs = [(o, s[:, off:off + keep.numel()] * keep.reshape(-1)) for o, s in outs]
    bound = 2.0 ** -17 * (1 + float(state.abs().max()))       # 128 roundings of 2^-24 of sums of the size of the state
    assert all((x - y).abs().max() <= bound for x, y in zip(*outs))


@pytest.mark.parametrize("mode", ["DECAY", "DELTA", "BONUS", "SSM", "DELTA_HEAD"])
def test_single_tokens_beside_long_segments_get_the_same_bits(mode):
    """A decoded token's output and state do not depend on whether a long portion shares its step."""
    ops = _ops()
    m, H, G, D, V = getattr(ops, "SCAN_" + mode), 4, 2, 72, 40
    lens = [1, 1, 130, 1, 64, 1]
    T, n = sum(lens), len(lens)
    normal = lambda *s: torch.randn(*s, device=DEV)
    q, k, v = normal(T, G * D) * D ** -0.5, torch.nn.functional.normalize(normal(T, G, D), dim=-1).reshape(T, -1), normal(T, H * V).bfloat16()
    gate_a = torch.rand({"DECAY": (H,), "DELTA": (T, H * D), "BONUS": (T, H * D)}.get(mode, (T, H)), device=DEV)
    gate_b = torch.rand(T, H, device=DEV) if mode in ("DELTA", "DELTA_HEAD", "SSM") else None
    extra = normal(H, D) if mode == "BONUS" else normal(H) if mode == "SSM" else None
    state = normal(n, H * D * V)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    slots = torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEV)

    def run(tokens, cu, slots, below):
        st, out = state.clone(), torch.full((len(tokens), H * V), 7.0, device=DEV)
        pick = lambda x: None if x is None else x[tokens].contiguous()
        batch = SimpleNamespace(cu_q=cu, seg_slot=slots, num_segments=len(slots))
        ops.linear_scan(m, pick(q), pick(k), pick(v), gate_a if mode == "DECAY" else pick(gate_a), pick(gate_b), st, (0, 0, 0), batch, out,
                        H, G, D, V, extra=extra, below=below, single=True)
        return out, st

    alone = [i for i, x in enumerate(lens) if x == 1]
    rows = cu[:-1][alone].long()
    out, st = run(torch.arange(T, device=DEV), cu, slots, 64)
    one, st1 = run(rows, torch.arange(len(alone) + 1, dtype=torch.int32, device=DEV), slots[alone], 0)
    assert torch.equal(out[rows], one) and torch.equal(st, st1)
    others = torch.ones(T, dtype=torch.bool, device=DEV)
    others[rows] = False
    assert (out[others] == 7.0).all()                          # long segments are left alone, their states too (st1 has the old ones)
