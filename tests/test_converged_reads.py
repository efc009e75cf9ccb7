"""Reads of tensor memory (tcgen05.ld.sync.aligned) are the whole warp's: a loop whose lanes store under conditions of their own joins them
before the next read, and no lane leaves a round early."""
import os

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "doppler_b200", "csrc")


def loop_around(text, at):
    """the body of the innermost for loop around a place, and the place in it"""
    depth, i = 0, at
    while True:
        i -= 1
        if text[i] == "}":
            depth += 1
        elif text[i] == "{":
            depth -= 1
            if depth < 0:
                if text.rindex("\n", 0, i) < text.rfind("for (", 0, i):
                    break
                depth = 0
    end, depth = i, 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[i:end], at - i


@pytest.mark.parametrize("file", ["gemm_bf16.cu", "gemm_f16w_rows.cu"])
def test_lanes_meet_before_they_read(file):
    with open(os.path.join(CSRC, file)) as f:
        text = f.read()
    body, at = loop_around(text, text.index("tmem_ld16("))
    assert "__syncwarp();" in body[:at] and "continue;" not in body
