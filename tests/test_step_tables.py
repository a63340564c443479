"""A step's tables against what they say entry by entry, whichever way the numbers get into them."""
import random

import numpy as np
import pytest

from return_b200.cache.manager import CacheManager, GroupSpec
from return_b200.engine.batch import StepEntry, build_host_batch
from return_b200.ext import build
from return_b200.parts.base import Tiling


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("seed", range(6))
def test_tables_entry_by_entry(monkeypatch, native, seed):
    if not native:
        monkeypatch.setattr(build, "native_module", lambda: None)
    rnd = random.Random(seed)
    n = rnd.choice((1, 2, 7, 30))
    manager = CacheManager([GroupSpec("all", 8, 600, None), GroupSpec("near", 4, 900, 9)], n)
    entries = []
    for i in range(n):
        manager.add(i)
        for _ in range(rnd.choice((0, 1, 3))):
            manager.append(i, rnd.randint(1, 12))
        new = 1 if seed % 3 == 0 else rnd.choice((1, 1, 5, 40))
        tokens = [rnd.randrange(500) for _ in range(new)]
        kind = rnd.choice((list, tuple, np.array)) if seed > 2 else list
        entries.append(StepEntry(rid=i, tokens=kind(tokens), want=[new - 1] if rnd.random() < 0.7 else [], start=manager.append(i, new)))
    h = build_host_batch(entries, manager, 500, 4096, {"t": Tiling(16, heaviest_first=True)})
    row = 0
    for i, e in enumerate(entries):
        L = len(e.tokens)
        assert h.tokens[row:row + L].tolist() == list(e.tokens) and h.pos[row:row + L].tolist() == list(range(e.start, e.start + L))
        assert (h.tok_seg[row:row + L] == i).all() and h.cu_q[i] == row and h.seg_pos0[i] == e.start and h.seg_kv_len[i] == e.start + L
        assert h.seg_slot[i] == manager.slot(i)
        for g, table in enumerate(h.block_tables):
            blocks = manager.block_table(i, g)[:table.shape[1]]
            assert table[i].tolist() == blocks + [-1] * (table.shape[1] - len(blocks))
        row += L
    assert h.cu_q[n] == row == h.num_tokens and all(getattr(h, f).dtype == np.int32 for f in (
        "tokens", "pos", "tok_seg", "seg_slot", "cu_q", "seg_pos0", "seg_kv_len", "want_rows", "decode_segs"))
    assert [t.shape[1] for t in h.block_tables] == [(int(h.seg_kv_len.max()) + p - 1) // p for p in (8, 4)]


@pytest.mark.skipif(build.native_calls_path() is None, reason="no C compiler or no Python headers")
def test_fill_says_what_it_does_not_take():
    fill = build.native_module().fill
    a = np.full(8, -1, np.int32)
    assert fill(a, [0, 5], [[1, 2, 3, 4], [2 ** 31 - 1, -2 ** 31]], 3) and a.tolist() == [1, 2, 3, -1, -1, 2 ** 31 - 1, -2 ** 31, -1]
    for places, lists in (([0], [[2 ** 31]]), ([0], [[-2 ** 31 - 1]]), ([0], [[1.0]]), ([0], [[True]]), ([0], [(1, 2)]), ([6], [[1, 2, 3]]), ([-1], [[1]]),
                          ([2 ** 70], [[1]]), ([0, 1], [[1]]), ([0], [[np.int64(3)]])):
        assert not fill(a, places, lists, 100)
    assert not fill(np.zeros(4, np.float32), [0], [[1]], 1) and not fill(np.zeros(4, np.int64), [0], [[1]], 1)
    with pytest.raises((BufferError, ValueError)):
        fill(np.zeros((4, 4), np.int32)[:, 1], [0], [[1]], 1)
