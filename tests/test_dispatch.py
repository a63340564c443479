"""The choices the engine makes on the host before it launches anything: how many ways keys are split,
which graph a decode step runs in.  Pure functions, no GPU."""
import pytest


def test_decode_graph_batch_sizes():
    from return_b200.engine.runner import graph_batch_size
    assert [graph_batch_size(m, 64) for m in range(1, 10)] == [1, 2, 3, 4, 5, 6, 7, 8, 12]
    assert [graph_batch_size(m, 64) for m in (12, 13, 16, 17, 24, 25, 33, 48, 49, 64)] == [12, 16, 16, 24, 24, 32, 48, 48, 64, 64]
    assert graph_batch_size(9, 10) == 10 and graph_batch_size(10, 10) == 10          # never beyond max_reside
    sizes = {graph_batch_size(m, 256) for m in range(1, 257)}
    assert len(sizes) <= 20 and all(graph_batch_size(m, 256) >= m for m in range(1, 257))
    # padding stays under half of the step
    assert all(graph_batch_size(m, 256) < 1.5 * m + 1 for m in range(9, 257))


def test_prefill_key_splits():
    """Keys are split only while blocks x heads leave SMs idle and every share keeps enough keys."""
    from return_b200.ext import ops
    assert ops.prefill_splits(256, 8192) == 1 and ops.prefill_splits(100, 8192) == 1
    assert ops.prefill_splits(64, 4096) == 2 and ops.prefill_splits(32, 4096) == 4
    assert ops.prefill_splits(32, 1024) == 2 and ops.prefill_splits(32, 600) == 1 and ops.prefill_splits(2, 100000) == 64
    for ctas in range(1, 300):
        for keys in (100, 700, 5000, 70000):
            s = ops.prefill_splits(ctas, keys)
            assert 1 <= s <= 64 and (s == 1 or (s * ctas <= ops.num_sms() and keys // s >= ops.PREFILL_SPLIT_MIN_KEYS))


def test_prefill_key_shares():
    """Shares keep enough keys, cover the longest block and stay within the scratch; even work is left alone."""
    import random
    from types import SimpleNamespace

    import numpy as np
    from return_b200.ext import ops
    assert ops.prefill_shares([4 * i for i in range(8, 0, -1)], 32, 2048, 128) == (1, 0)        # a whole prompt, 32 heads
    assert ops.prefill_shares([8], 4, 200, 128) == (1, 0)                                       # a share would have too few keys
    rng = random.Random(0)
    for _ in range(300):
        tiles = [rng.randint(1, 400) for _ in range(rng.randint(1, 40))]
        heads, rows = rng.choice((4, 16, 32)), 256 * len(tiles)
        s, share = ops.prefill_shares(tiles, heads, rows, 128)
        if s == 1:
            assert share == 0
            continue
        assert 1 < s <= 64 and share * ops.PREFILL_KEY_TILE >= ops.PREFILL_SPLIT_MIN_KEYS
        assert -(-max(tiles) // share) <= s and s * rows * heads * 130 * 4 <= ops.PREFILL_SPLIT_SCRATCH_BYTES
    # the tiles that the kernel walks for a block, counted key by key
    for _ in range(100):
        pos0, n = rng.randint(0, 600), rng.randint(2, 700)
        window, chunk, keep = rng.choice(((None, None, 0), (rng.randint(1, 300), None, 0), (rng.randint(1, 300), None, rng.randint(1, 300)),
                                          (None, rng.randint(1, 300), 0)))
        blocks = np.array([(0, r) for r in range(0, n, ops.TC5_TILE_ROWS)], np.int32)
        seen = []
        real, ops.prefill_shares = ops.prefill_shares, lambda tiles, *rest: (seen.append(tiles), (1, 0))[1]
        try:
            ops.prefill_shares_of(SimpleNamespace(host=SimpleNamespace(tiles={ops.TILES_TC5: blocks}, seg_pos0=np.array([pos0]),
                                                                       seg_kv_len=np.array([pos0 + n]), num_tokens=n)), 4, 128, window, chunk, keep)
        finally:
            ops.prefill_shares = real
        for got, (_, r0) in zip(seen[0], blocks):
            first = pos0 + r0
            last = min(first + ops.TC5_TILE_ROWS, pos0 + n) - 1
            low = max(0, first - window + 1) if window else first // chunk * chunk if chunk else 0
            walked = {j // 64 for j in range(low, last + 1)} | {j // 64 for j in range(min(keep, low // 64 * 64))}
            assert got == len(walked)


def test_prefill_key_shares_cost_little():
    """A new step pays for the choice in host time: a few sums a candidate, however many blocks there are and however uneven."""
    import random
    import sys

    from return_b200.ext import ops
    ops.num_sms()
    rng = random.Random(0)
    for n, heads in ((4, 16), (12, 4), (16, 4), (64, 4), (128, 32), (256, 32)):
        for _ in range(20):
            tiles = sorted((int(2 ** rng.uniform(0, 9)) for _ in range(n)), reverse=True)
            calls = []
            sys.setprofile(lambda frame, event, arg: calls.append(event) if event in ("call", "c_call") else None)
            try:
                ops.prefill_shares(tiles, heads, 64 * n, 128)
            finally:
                sys.setprofile(None)
            assert len(calls) <= 120, (n, heads, len(calls))


def _state_mixer(H, D, V, dtype):
    from types import SimpleNamespace
    from return_b200.parts.recurrent import _StateMixer
    m = object.__new__(_StateMixer)
    m.H, m.D, m.V, m.env = H, D, V, SimpleNamespace(act_dtype=dtype, device="cpu")
    return m


def _scan_batch(lens):
    from types import SimpleNamespace

    import numpy as np
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    host = SimpleNamespace(cu_q=cu, num_multi=sum(n > 1 for n in lens))
    return SimpleNamespace(host=host, scratch={}, num_segments=len(lens), num_tokens=int(cu[-1]))


def test_chunked_scan_is_launched_for_the_long_segments_alone(monkeypatch):
    """The scan in chunks takes an SM a CTA: decoded tokens beside a portion must not add CTAs to it."""
    from types import SimpleNamespace

    import torch
    from return_b200.ext import ops
    seen = []
    monkeypatch.setattr(ops, "chunked_scan_ok", lambda mode, heads, dim: True)
    monkeypatch.setattr(ops, "chunked_scan", lambda mode, *a, **k: seen.append(("chunks", a[8], k["longs"])))
    monkeypatch.setattr(ops, "linear_scan", lambda mode, *a, **k: seen.append(("singles" if k["single"] else "walk", k["below"])))
    m = _state_mixer(16, 128, 128, torch.bfloat16)
    least = m.CHUNKED_MIN_TOKENS
    for lens, want in (([1] * 64 + [200], [("chunks", 7, 1), ("singles", least)]), ([300, 1, least, least - 1], [("chunks", 10 + least // 32, 2), ("walk", least)]),
                       ([least], [("chunks", least // 32, 1)]), ([1, least - 1], [])):
        seen.clear()
        batch = _scan_batch(lens)
        ctx = SimpleNamespace(batch=batch, state=None, buffer=None)
        assert m._scan_in_chunks(ops.SCAN_DELTA, None, None, None, None, None, ctx, None, 4) == bool(want)
        assert seen == want


def test_which_scan_a_portion_takes(monkeypatch):
    """Chunks from CHUNKED_MIN_TOKENS on, but where a linear scan can be cut into many pieces, or into any with few key rows."""
    import torch
    from return_b200.ext import ops
    monkeypatch.setattr(ops, "num_sms", lambda: 148)
    monkeypatch.setattr(ops, "chunked_scan_ok", lambda mode, heads, dim: mode != ops.SCAN_MEMORY and dim <= 128)
    for H, D, V, mode, lens, pieces, chunks in (
            (2, 24, 40, ops.SCAN_DECAY, [992], None, 31), (2, 24, 40, ops.SCAN_DECAY, [1, 1190], [1, 9], None), (2, 64, 40, ops.SCAN_DECAY, [1190], [9], 38),
            (2, 64, 40, ops.SCAN_SSM, [2048], [16], None), (2, 64, 40, ops.SCAN_DELTA, [2048], [16], 64), (2, 24, 40, ops.SCAN_DELTA_HEAD, [1190], [9], 38),
            (16, 128, 128, ops.SCAN_BONUS, [2048], [4], 64), (16, 32, 128, ops.SCAN_BONUS, [2048], [4], None), (16, 32, 256, ops.SCAN_BONUS, [2048], None, 64),
            (16, 128, 128, ops.SCAN_DECAY, [95, 1], None, None), (16, 128, 128, ops.SCAN_DECAY, [96, 1], None, 3), (4, 200, 64, ops.SCAN_DECAY, [500], None, None)):
        m, batch = _state_mixer(H, D, V, torch.bfloat16), _scan_batch(lens)
        plan = m._chunks(mode, batch)
        assert (plan and plan[0]) == chunks, (H, D, V, mode, lens, plan)
        assert m._piece_counts(batch.host.cu_q[1:] - batch.host.cu_q[:-1]) == pieces
        assert _state_mixer(H, D, V, torch.float32)._chunks(mode, _scan_batch(lens)) is None


def test_experts_dispatch():
    from return_b200.ext import ops
    assert ops.moe_on_tc5(128, 16, 1024, 768) and not ops.moe_on_tc5(127, 16, 1024, 768)        # little weight: from 128 pairs on
    assert ops.moe_on_tc5(64, 32, 2048, 1536) and not ops.moe_on_tc5(8192, 1025, 2048, 1536)    # much: always; at most 1,024 experts


def test_decode_key_splits():
    from return_b200.ext import ops
    for base in (1, 8, 64, 296, 512, 2000):
        for keys in (1, 100, 2048, 40000):
            s = ops.decode_splits(base, keys)
            assert 1 <= s <= 64
            assert s == 1 or (keys + s - 1) // s >= 128            # a share keeps at least 128 keys
    assert ops.decode_splits(512, 2048) == 1                      # more CTAs than the GPU holds at once: no split
    assert ops.decode_splits(8, 32768) > ops.decode_splits(8, 2048) >= 2


def test_profile_buckets_know_the_engines_kernels():
    from return_b200 import benchmark
    names = {"void (anonymous namespace)::gemm_skinny_kernel<1, __nv_bfloat16, 0, 2>(...)": "gemm/matmul",
             "nvjet_tst_64x32_64x8_4x1_v_bz_TNT": "gemm/matmul",
             "void (anonymous namespace)::attn_decode_kernel<true>(...)": "decode_attn",
             "(anonymous namespace)::attn_combine_kernel(...)": "decode_attn",
             "attn_prefill_tc5_kernel": "prefill_attn",
             "void add_rmsnorm_vec_kernel<__nv_bfloat16, __nv_bfloat16, 4>(...)": "rmsnorm",
             "void qk_norm_rope_write_vec_kernel<8>(...)": "rope",
             "void swiglu_bf16x8_kernel(...)": "elementwise",
             "void sample_kernel(...)": "softmax/sample", "something_else": "other"}
    for kernel, want in names.items():
        assert benchmark.profile_bucket(kernel) == want, kernel
