"""The rows that the design benchmarks put together from the kernels' names."""
import os
import re

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
