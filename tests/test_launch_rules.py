"""What the sources of kernels that overlap the kernel before them keep to (csrc/common.cuh): nothing that a kernel may have written is read in front
of ``pdl_wait()``."""
import os
import re

import pytest

import return_b200

CSRC = os.path.join(os.path.dirname(return_b200.__file__), "csrc")


def _body(source, kernel):
    """The text of a kernel from its opening brace on, comments taken out."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, source)).read())
    return text[text.index("{", re.search(r"\b" + kernel + r"\(const [^;{]*\)", text).start()):]


# kernel, and how it spells what other kernels write
@pytest.mark.parametrize("source,kernel,written", [
    ("attention_f32.cu", "attention_f32_kernel", r"\ba\.(q|kpool|vpool|pos|tok_seg|block_table|out)\b"),
    ("gemm_f32.cu", "gemm_f32_kernel", r"\bg\.(A|C)\b"),
    ("gemm_rows.cu", "gemm_rows_kernel", r"\bg\.(ssq_in|stream|ssq_out|out)\b|load_box\("),
    ("elementwise.cu", "swiglu_f32x4_kernel", r"\b(gu|out) \+"),
])
def test_nothing_is_read_in_front_of_the_wait(source, kernel, written):
    body = _body(source, kernel)
    wait = body.index("pdl_wait()")
    first = re.search(written, body)
    assert first is not None and first.start() > wait, body[first.start():first.start() + 60]
