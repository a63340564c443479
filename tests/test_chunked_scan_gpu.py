"""The recurrences 32 tokens at a time against the plain recurrence in float64 and beside the walk token by token."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _ops():
    from return_b200.ext import ops
    return ops


def plain(mode, ops, q, k, v, gate_a, gate_b, S, extra):
    """One segment: q, k [T, H, D], v [T, H, V], S [H, D, V], all float64."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        g = gate_a[:, None, None] if mode == ops.SCAN_DECAY else gate_a[t].reshape(S.shape[0], -1, 1)
        if mode == ops.SCAN_BONUS:
            pair = k[t][:, :, None] * v[t][:, None]
            out[t] = torch.bmm(q[t][:, None], S + extra[:, :, None] * pair)[:, 0]
            S = g * S + pair
            continue
        S = g * S
        u = v[t]
        if mode in (ops.SCAN_DELTA, ops.SCAN_DELTA_HEAD):
            u = gate_b[t][:, None] * (u - torch.bmm(k[t][:, None], S)[:, 0])
        elif mode == ops.SCAN_SSM:
            u = gate_b[t][:, None] * u
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = torch.bmm(q[t][:, None], S)[:, 0]
        if mode == ops.SCAN_SSM:
            out[t] += extra[:, None] * v[t]
    return out, S


def rows(S):
    """A state [H, D, V] in a slot's order: [head][row / 8][column][row % 8], rows padded with zeros."""
    H, D, V = S.shape
    padded = torch.zeros(H, (D + 7) // 8 * 8, V, dtype=S.dtype, device=S.device)
    padded[:, :D] = S
    return padded.view(H, -1, 8, V).transpose(2, 3).reshape(-1)


@pytest.mark.parametrize("mode", ["DECAY", "DELTA", "BONUS", "SSM", "DELTA_HEAD"])
@pytest.mark.parametrize("lens,H,G,D,V,decay,form", [
    ([64, 1, 95, 96], 2, 2, 128, 16, 1.0, "float32"),          # whole chunks and remainders, a segment that is left alone
    ([70, 200], 4, 2, 24, 40, 0.1, "bfloat16"),                # few key rows, columns that do not fill a CTA
    ([97], 2, 1, 100, 24, 30.0, "unaligned"),                  # decays that underflow within a chunk; rows off 16-byte boundaries
    ([129, 65], 3, 3, 64, 17, 0.0, "bfloat16"),                # no decay at all
])
def test_chunked_scan(mode, lens, H, G, D, V, decay, form, monkeypatch):
    ops = _ops()
    m = getattr(ops, "SCAN_" + mode)
    delta = mode.startswith("DELTA")
    T, n = sum(lens), len(lens)
    gen = torch.Generator(device=DEV).manual_seed(D + V)
    normal = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    dt = torch.bfloat16 if form == "bfloat16" else torch.float32
    wide = torch.zeros(T, 2 * G * D + H * V + 5, dtype=dt, device=DEV)
    lead = 3 if form == "unaligned" else 0
    q, k, v = wide[:, lead:lead + G * D], wide[:, lead + G * D:lead + 2 * G * D], wide[:, lead + 2 * G * D:lead + 2 * G * D + H * V]
    q.copy_(normal(T, G * D) * D ** -0.5)
    k.copy_(unit(normal(T, G, D)).reshape(T, -1))
    v.copy_(normal(T, H * V))
    shape = {"DECAY": (H,), "DELTA": (T, H * D), "BONUS": (T, H * D)}.get(mode, (T, H))
    gate_a = torch.exp(-decay * torch.nn.functional.softplus(normal(*shape)))
    gate_b = torch.rand(T, H, generator=gen, device=DEV) if delta or mode == "SSM" else None
    extra = normal(H, D) if mode == "BONUS" else normal(H) if mode == "SSM" else None
    s_off, per = 1, H * ((D + 7) // 8 * 8) * V                  # a state that begins on an odd float of an odd row
    starts = [normal(H, D, V) * 0.3 for _ in lens]
    state = torch.zeros(n + 1, s_off + per + 2 - (per + s_off) % 2, device=DEV)
    for i, S in enumerate(starts):
        state[n - i, s_off:s_off + per] = rows(S)              # slots in another order than segments
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    batch = SimpleNamespace(cu_q=torch.from_numpy(cu).to(DEV), num_segments=n,
                            seg_slot=torch.tensor([n - i for i in range(n)], dtype=torch.int32, device=DEV))
    chunks = sum((x + 31) // 32 for x in lens if x >= 64)

    def run(in_chunks, scratch=None):
        st, out = state.clone(), torch.full((T, H * V), float("nan"), device=DEV)
        below = 0
        if in_chunks:
            if scratch is not None:
                monkeypatch.setattr(ops, "CHUNK_SCRATCH_BYTES", scratch)
            ops.chunked_scan(m, q, k, v, gate_a, gate_b, st, s_off, batch, chunks, 64, out, H, G, D, V, extra=extra)
            below = 64
        ops.linear_scan(m, q, k, v, gate_a, gate_b, st, (s_off, 0, 0), batch, out, H, G, D, V, extra=extra, below=below)
        return out, st

    got, walked = run(True), run(False)
    windows = run(True, scratch=1)                             # a chunk at a time: the state goes through its slot in between
    ops.check_status(DEV)
    assert torch.equal(windows[0], got[0]) and torch.equal(windows[1], got[1])
    f = lambda x: None if x is None else x.double()
    heads = lambda x, d, g: x.double().reshape(-1, g, d).repeat_interleave(H // g, 1)
    for i, (a, b) in enumerate(zip(cu[:-1], cu[1:])):
        ga = f(gate_a) if mode == "DECAY" else f(gate_a[a:b])
        want, S = plain(m, ops, heads(q[a:b], D, G), heads(k[a:b], D, G), heads(v[a:b], V, H), ga,
                        None if gate_b is None else f(gate_b[a:b]), starts[i].double(), f(extra))
        for x, y, w in ((got[0][a:b], walked[0][a:b], want.reshape(b - a, -1)),
                        (got[1][n - i, s_off:s_off + per], walked[1][n - i, s_off:s_off + per], rows(S))):
            off = lambda z: float((z.double() - w).norm() / w.norm())
            # sums of up to 128 + 32 terms rounded to 24 bits, in other orders: a few 2^-24 either way
            assert off(x) < 2.0 * off(y) + 2.0 ** -22, (i, off(x), off(y))


@pytest.mark.parametrize("lens", [[1] * 131 + [70, 1, 64, 3, 200], [100] + [1] * 40 + [65], [64] * 37 + [1] * 95 + [97]])
def test_long_segments_are_found(lens):
    """The grid of the second kernel covers the long segments alone, wherever they stand among the others; a grid that covers more
    gives the same, in windows that begin within a segment too."""
    ops = _ops()
    H, D, V, T, n = 2, 64, 24, sum(lens), len(lens)
    gen = torch.Generator(device=DEV).manual_seed(n)
    normal = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    q, k, v, state = normal(T, H * D) * D ** -0.5, normal(T, H * D) * D ** -0.5, normal(T, H * V), normal(n, H * D * V)
    gate = torch.rand(H, generator=gen, device=DEV)
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    batch = SimpleNamespace(cu_q=cu, num_segments=n, seg_slot=torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEV))
    longs, chunks = sum(x >= 64 for x in lens), sum((x + 31) // 32 for x in lens if x >= 64)
    outs = []
    for grid, scratch in ((longs, 64 << 20), (None, 64 << 20), (longs, 5 * 4 * ops.recurrent_lib().rb_chunked_scan_floats(ops.SCAN_DECAY, H, D))):
        st, out = state.clone(), torch.zeros(T, H * V, device=DEV)
        old, ops.CHUNK_SCRATCH_BYTES = ops.CHUNK_SCRATCH_BYTES, scratch
        try:
            ops.chunked_scan(ops.SCAN_DECAY, q, k, v, gate, None, st, 0, batch, chunks, 64, out, H, H, D, V, longs=grid)
        finally:
            ops.CHUNK_SCRATCH_BYTES = old
        outs.append((out, st))
    ops.check_status(DEV)
    for out, st in outs[1:]:
        assert torch.equal(out, outs[0][0]) and torch.equal(st, outs[0][1])
    walked, st = torch.zeros(T, H * V, device=DEV), state.clone()
    ops.linear_scan(ops.SCAN_DECAY, q, k, v, gate, None, st, (0, 0, 0), batch, walked, H, H, D, V)
    for i, (a, b) in enumerate(zip(cu[:-1].tolist(), cu[1:].tolist())):
        slot = n - 1 - i
        if b - a < 64:                                         # left alone
            assert not outs[0][0][a:b].any() and torch.equal(outs[0][1][slot], state[slot])
        else:                                                  # the same sums of up to 64 + 32 terms in another order
            assert torch.allclose(outs[0][0][a:b], walked[a:b], rtol=2.0 ** -18, atol=2.0 ** -18 * float(walked.abs().max()))
            assert torch.allclose(outs[0][1][slot], st[slot], rtol=2.0 ** -18, atol=2.0 ** -18 * float(st.abs().max()))


@pytest.mark.parametrize("mode", ["DECAY", "DELTA", "BONUS", "SSM", "DELTA_HEAD"])
@pytest.mark.parametrize("D,V", [(24, 40), (128, 16)])
@pytest.mark.parametrize("where,what", [("v", "inf"), ("v", "nan"), ("v", "3.4e38"), ("k", "nan"), ("k", "inf"), ("q", "nan"), ("gate_a", "nan"),
                                        ("gate_b", "inf"), ("state", "-inf"), ("state", "nan")])
def test_infinities_and_nans_reach_what_they_reach_token_by_token(mode, D, V, where, what):
    """An infinity, a NaN or a number beyond bfloat16's largest, in one token and head: no token before it, no other head or request
    and (in a value or a state) no other column sees it, and the tokens behind it hold infinities and NaNs where the walk has them."""
    ops = _ops()
    m, x = getattr(ops, "SCAN_" + mode), float(what)
    delta = mode.startswith("DELTA")
    if where == "gate_b" and not (delta or mode == "SSM") or where == "gate_a" and mode == "DECAY":
        pytest.skip("no such operand")
    lens, H, G, at = [70, 100, 40], 4, 2, 70 + 43                # the 12th token of the second segment's second chunk
    T, n = sum(lens), len(lens)
    gen = torch.Generator(device=DEV).manual_seed(D)
    normal = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    q, k, v = normal(T, G * D) * D ** -0.5, torch.nn.functional.normalize(normal(T, G, D), dim=-1).reshape(T, -1), normal(T, H * V)
    shape = {"DECAY": (H,), "DELTA": (T, H * D), "BONUS": (T, H * D)}.get(mode, (T, H))
    gate_a = torch.rand(*shape, generator=gen, device=DEV)
    gate_b = torch.rand(T, H, generator=gen, device=DEV) if delta or mode == "SSM" else None
    extra = normal(H, D) if mode == "BONUS" else normal(H) if mode == "SSM" else None
    state = normal(n, H * D * V) * 0.3
    head = 3                                                     # the head of values, gates and state; its queries and keys are the second group's
    if where == "v":
        v[at, head * V + 5] = x
    elif where == "state":
        state[1, head * D * V + (0 * V + 5) * 8 + 2] = x         # a row of column 5
    elif where in ("k", "q"):
        {"k": k, "q": q}[where][at, 1 * D + 9] = x
    elif where == "gate_b":
        gate_b[at, head] = x
    else:
        gate_a[at, head * (gate_a.shape[1] // H)] = x
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    batch = SimpleNamespace(cu_q=cu, num_segments=n, seg_slot=torch.arange(n, dtype=torch.int32, device=DEV))
    outs = []
    for chunks in (False, True):
        st, out = state.clone(), torch.zeros(T, H * V, device=DEV)
        if chunks:
            ops.chunked_scan(m, q, k, v, gate_a, gate_b, st, 0, batch, 9, 1, out, H, G, D, V, extra=extra, longs=n)
        else:
            ops.linear_scan(m, q, k, v, gate_a, gate_b, st, (0, 0, 0), batch, out, H, G, D, V, extra=extra)
        outs.append((out, st))
    ops.check_status(DEV)
    # a column's sums are of terms of its own size, in another order
    columns = [lambda y: y.view(T, H * V).amax(0).expand(T, -1), lambda y: y.view(n, H, D // 8, V, 8).amax((2, 4), keepdim=True).expand(n, H, D // 8, V, 8).reshape(n, -1)]
    for walked, got, size in zip(outs[0], outs[1], columns):
        plain = walked.isfinite()
        assert torch.equal(got.isnan(), walked.isnan()) and torch.equal(got[walked.isinf()], walked[walked.isinf()])
        bound = 2.0 ** -17 * (1.0 + size(torch.where(plain, walked.abs(), torch.zeros_like(walked))))
        assert ((got - walked).abs() <= bound)[plain].all()
    out = outs[1][0]
    first = 70 if where == "state" else at
    assert out[:first].isfinite().all() and out[170:].isfinite().all()       # the tokens before, and the third request
    if where in ("v", "state"):
        others = torch.ones(H * V, dtype=torch.bool, device=DEV)
        others[head * V + 5] = False
        assert out[:, others].isfinite().all()
    if what != "3.4e38":
        assert not out[first:170].isfinite().all()
