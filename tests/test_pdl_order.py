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
