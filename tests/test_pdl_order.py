"""Decode attention reads positions, lengths and cache rows of earlier steps before it waits for its predecessor.  That needs the
kernels that begin a step to launch their dependents only behind their own wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "doppler_b200", "csrc")


def body(file, kernel):
    with open(os.path.join(CSRC, file)) as f:
        text = f.read()
    at = re.search(r"__global__[^;{]*\b" + kernel + r"\(", text).end()
    return text[text.index("{", at):text.index("\n}\n", at)]


@pytest.mark.parametrize("file,kernel", [("small_ops.cu", "gather_f16_kernel"), ("streams.cu", "stream_embed_kernel")])
def test_first_kernels_of_a_step_wait_before_they_launch(file, kernel):
    b = body(file, kernel)
    assert b.count("pdl_launch();") == 1 and 0 < b.index("pdl_wait();") < b.index("pdl_launch();")


@pytest.mark.parametrize("file,kernel", [("gemm_q4k_int.cu", "gemm_q4k_int_kernel"), ("gemm_q4k_tc.cu", "gemm_q4k_tc2_kernel"), ("gemm_bf16.cu", "gemm_bf16_tc_kernel")])
def test_launches_of_clusters_launch_no_dependents_early(file, kernel):
    """Dependents of such a launch, which carries no programmatic attribute, were seen to read rows that it had not stored yet."""
    b = body(file, kernel).replace("if constexpr (!PAIR) pdl_launch();", "")
    assert "pdl_launch();" not in b and b.count("pdl_wait();") == 1
