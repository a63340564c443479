"""The rows that the design benchmarks put together from the kernels' names."""
import os
import re

import pytest

from return_b200 import benchmark
from return_b200.ext import build


def _kernels(*sources):
    text = "".join(open(os.path.join(build.CSRC, name)).read() for name in sources)
    return set(re.findall(r"__global__\b[^;{]*?(\w+_kernel)\(", text))


def test_scan_rows_count_every_kernel_of_a_scan():
    found = {k for k in _kernels("recurrent.cu", "recurrent_chunks.cu") if k.startswith(("linear_", "scan_step", "chunk_"))}
    assert found == {"linear_scan_kernel", "scan_step_kernel", "chunk_prep_kernel", "chunk_serial_kernel"}
    assert benchmark._kernel_ms({f"void (anonymous namespace)::{k}<3, 128>(Args)": 1.0 for k in found}, *benchmark.SCAN_KERNELS) == len(found)
    assert benchmark._kernel_ms({"delta_prep_kernel": 1.0, "conv_state_update_kernel": 1.0, "general_delta_scan_kernel": 1.0}, *benchmark.SCAN_KERNELS) == 0


def test_expert_rows_count_every_product_of_decoded_tokens():
    found = {k for k in _kernels("moe.cu", "moe_tc5.cu") if "linear" in k or "gemm" in k or "tc5" in k}
    assert {"moe_pair_linear_kernel", "moe_grouped_gemm_kernel", "moe_tc5_kernel"} <= found
    assert all(benchmark._kernel_ms({k: 1.0}, *benchmark.DECODED_EXPERT_KERNELS) for k in found), found


@pytest.mark.gpu
@pytest.mark.parametrize("ctx,q_len,window", [(4096, 512, 0), (4096, 4096, 0), (6000, 300, 1000)])
def test_prefill_attention_is_timed_as_the_engine_launches_it(monkeypatch, ctx, q_len, window):
    from return_b200.ext import ops
    used, kernel = [], ops.attention_prefill_tc5
    monkeypatch.setattr(ops, "attention_prefill_tc5", lambda *a, **k: (used.append((k["num_splits"], k["share"])), kernel(*a, **k))[1])
    row = benchmark.kernel_attention_prefill(1, ctx, q_len, 4, 2, 64, iters=2, warmup=1, window=window)
    tiles = []
    for first in range(ctx - q_len, ctx, ops.TC5_TILE_ROWS):
        low = max(0, first - window + 1) if window else 0
        tiles.append((min(ctx, first + ops.TC5_TILE_ROWS) - 1) // 64 - low // 64 + 1)
    assert set(used) == {ops.prefill_shares(tiles[::-1], 4, q_len, 64)} == {(row["splits"], row["share"])}
