"""The 32-bit attention on the matrix instructions against the kernel of the CUDA cores, which takes pools that lie off 16-byte boundaries."""
import types

import pytest
import torch

from test_kernels_gpu import Paged

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _off(pool):
    """The same pool four bytes further."""
    flat = torch.empty(pool.numel() + 1, device=DEV)
    flat[1:] = pool.reshape(-1)
    return flat[1:].view(pool.shape)


def _both(pg, Hq, Hkv, D, P, **options):
    from return_b200.ext import ops
    batch = types.SimpleNamespace(pos=pg.pos, tok_seg=pg.tok_seg)
    outs = []
    for k, v in ((pg.kpool, pg.vpool), (_off(pg.kpool), _off(pg.vpool))):
        out = torch.full((pg.qkv.shape[0], Hq * D), float("nan"), device=DEV)
        ops.paged_attention(pg.qkv, k, v, batch, pg.bt, P, out, Hq, Hkv, D, D ** -0.5, **options)
        outs.append(out)
    return outs


@pytest.mark.parametrize("Hq,Hkv,D,P", [(2, 2, 32, 16), (8, 2, 64, 8), (40, 1, 96, 16), (16, 8, 128, 16)])
@pytest.mark.parametrize("options", ["plain", "window", "keep", "chunk", "softcap", "slopes", "bias", "sink"])
def test_options_and_edges(Hq, Hkv, D, P, options):
    """Rows of softmax-weighted values of size 1: a chain of FFMAs and the split products are each off by a few 2^-24 a tile of keys."""
    pg = Paged([1, 70, 200, 33, 129, 64], [1, 70, 17, 33, 3, 1], Hq, Hkv, D, P, torch.float32, seed=D)
    g = torch.Generator(device=DEV).manual_seed(D)
    given = {"plain": {}, "window": {"window": 37}, "keep": {"window": 40, "keep": 35}, "chunk": {"chunk": 48}, "softcap": {"softcap": 3.0},
             "slopes": {"slopes": torch.rand(Hq, device=DEV, generator=g)}, "sink": {"sink": torch.randn(Hq, device=DEV, generator=g)},
             "bias": {"bias": torch.randn(Hq, 50, device=DEV, generator=g)}}[options]
    got, want = _both(pg, Hq, Hkv, D, P, **given)
    assert torch.isfinite(got).all()
    assert (got - want).abs().max() <= 2e-6 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("D", [32, 64, 96, 128])
def test_error_is_no_larger_than_the_chains(D):
    pg = Paged([400, 300], [400, 60], 4, 2, D, 16, torch.float32, seed=3)
    got, chain = _both(pg, 4, 2, D, 16)
    err = [0.0, 0.0]
    row = 0
    for i, (n, ql) in enumerate(zip(pg.kv_lens, pg.q_lens)):
        q, k, v = pg.q[i].double(), pg.k[i].double().repeat_interleave(2, 1), pg.v[i].double().repeat_interleave(2, 1)
        s = torch.einsum("qhd,nhd->hqn", q, k) * D ** -0.5
        s = s.masked_fill(torch.arange(n)[None] > torch.arange(n - ql, n)[:, None], float("-inf"))
        want = torch.einsum("hqn,nhd->qhd", torch.softmax(s, -1), v).reshape(ql, -1).to(DEV)
        for j, o in enumerate((got, chain)):
            err[j] += float((o[row:row + ql].double() - want).norm() ** 2)
        row += ql
    assert err[0] <= err[1]


@pytest.mark.parametrize("window", [None, 40])
def test_infinities_and_nans_reach_who_sees_them(window):
    pg = Paged([100, 70], [100, 30], 4, 2, 64, 16, torch.float32, seed=8)
    inf, nan, big = float("inf"), float("nan"), 3.4e38
    for at, value in ((20, inf), (50, nan), (61, -inf), (80, big)):
        page, row = int(pg.bt[0, at // 16]), at % 16
        pg.vpool[page, 0, row, at % 64] = value
        pg.vpool[page, 1, row, 3] = value
    page, row = int(pg.bt[1, 2]), 9
    pg.kpool[page, 0, row, 5] = inf
    pg.kpool[page, 1, row, 7] = nan
    pg.qkv[110, 3] = inf
    got, want = _both(pg, 4, 2, 64, 16, window=window)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[want.isinf()], want[want.isinf()])
    assert want.isnan().any() and torch.isfinite(want).any()
    fine = torch.isfinite(want)
    assert ((got - want).abs()[fine] <= 1e-5 * want.abs()[fine] + 2e-6).all()


def test_rows_do_not_depend_on_their_block():
    from return_b200.ext import ops
    pg = Paged([130, 70, 200, 1], [130, 3, 17, 1], 16, 8, 128, 16, torch.float32, seed=2)
    def run(rows):
        out = torch.full((len(rows), 16 * 128), float("nan"), device=DEV)
        batch = types.SimpleNamespace(pos=pg.pos[rows].contiguous(), tok_seg=pg.tok_seg[rows].contiguous())
        ops.paged_attention(pg.qkv[rows].contiguous(), pg.kpool, pg.vpool, batch, pg.bt, 16, out, 16, 8, 128, 128 ** -0.5, 75)
        return out
    rows = torch.arange(sum(pg.q_lens))
    whole = run(rows)
    for t in (0, 15, 16, 17, 64, 129, 130, 132, 133, 149, 150):
        assert torch.equal(run(rows[t:t + 1])[0], whole[t]), t
    assert torch.equal(run(rows.flip(0)), whole.flip(0))


def test_tables_written_by_the_kernel_just_before():
    """The launch overlaps the kernel before it, so the tables are read behind the wait for that kernel."""
    from return_b200.ext import ops
    pg = Paged([130, 70, 1], [130, 3, 1], 4, 2, 64, 16, torch.float32, seed=4)
    order = torch.randperm(134, generator=torch.Generator().manual_seed(1)).to(DEV)
    sets = [(pg.qkv, pg.pos, pg.tok_seg), tuple(t[order].contiguous() for t in (pg.qkv, pg.pos, pg.tok_seg))]
    tables = types.SimpleNamespace(pos=torch.zeros_like(pg.pos), tok_seg=torch.zeros_like(pg.tok_seg))

    def run(k, out):
        qkv, pos, seg = sets[k]
        torch.add(pos, 0, out=tables.pos)
        torch.add(seg, 0, out=tables.tok_seg)
        ops.paged_attention(qkv, pg.kpool, pg.vpool, tables, pg.bt, 16, out, 4, 2, 64, 0.125)

    outs = [torch.full((134, 256), float("nan"), device=DEV) for _ in range(40)]
    for i, out in enumerate(outs):
        run(i & 1, out)
        if i < 2:
            torch.cuda.synchronize()
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[1], outs[0][order])
    for i, out in enumerate(outs):
        assert torch.equal(out, outs[i & 1]), i


@pytest.mark.parametrize("q_up,k_up,v_up", [(100, -118, 0), (0, 0, -115), (-118, 105, 60)])
def test_small_operands_keep_their_24_bits(q_up, k_up, v_up):
    """Queries, keys and values times powers of two: the same scores and the same softmax, also where an operand's last bits lie below
    bfloat16's smallest number."""
    from return_b200.ext import ops
    pg = Paged([100, 70], [100, 30], 4, 2, 64, 16, torch.float32, seed=12)
    plain, _ = _both(pg, 4, 2, 64, 16)
    q_cols = 4 * 64
    pg.qkv[:, :q_cols] *= 2.0 ** q_up
    pg.kpool *= 2.0 ** k_up
    pg.vpool *= 2.0 ** v_up
    batch = types.SimpleNamespace(pos=pg.pos, tok_seg=pg.tok_seg)
    outs = []
    for k, v in ((pg.kpool, pg.vpool), (_off(pg.kpool), _off(pg.vpool))):
        out = torch.full((130, q_cols), float("nan"), device=DEV)
        ops.paged_attention(pg.qkv, k, v, batch, pg.bt, 16, out, 4, 2, 64, 0.125 * 2.0 ** -(q_up + k_up))
        outs.append(out.double() * 2.0 ** -v_up)
    got, want = outs
    assert torch.isfinite(got).all()
    assert (got - want).abs().max() <= 2e-6 * max(1.0, float(want.abs().max()))
    assert (got - plain.double()).abs().max() <= 2e-6 * max(1.0, float(want.abs().max()))
