"""Which call of a runner a scheduler's step becomes."""
import os

import numpy as np
import pytest

from doppler_b200 import scheduler
from doppler_b200.scheduler import Scheduler


class Runner:
    max_batch, tp_size = 2, 1

    def __init__(self):
        self.cfg, self.calls = {"vocab": 5, "max_seq": 64}, []

    def release(self, seq):
        pass

    def extend(self, tokens, want=(), seq=0):
        self.calls.append(("extend", len(tokens), seq))
        return np.zeros((len(want), 5), np.float32)

    def decode(self, tokens, steps):
        self.calls.append(("decode", tuple(tokens), steps))
        return np.zeros((steps, 1), np.int32)

    def advance(self, token):
        self.calls.append(("advance", token))

    def read_logits(self, n):
        self.calls.append(("read_logits", n))
        return np.arange(n, dtype=np.float32)


class Sharded(Runner):
    tp_size = 2


class Plain(Runner):
    advance = property()


@pytest.mark.parametrize("runner", [Runner, Sharded, Plain])
def test_one_token_of_the_only_sequence(runner):
    """On one GPU the table is left to the read of the logits, which comes where they are wanted."""
    m = runner()
    s = Scheduler(m)
    assert np.array_equal(s.step("a", [3], [0, 0]), np.arange(5, dtype=np.float32) * np.ones((2, 1)))
    one = [("advance", 3) if runner is Runner else ("decode", (3,), 1)]
    assert m.calls == one + [("read_logits", 5)]
    assert s.step("a", [3]).shape == (0, 5)
    assert m.calls[2:] == one


def test_everything_else_is_a_portion():
    m = Runner()
    s = Scheduler(m)
    s.step("a", [1, 2], [1])
    s.step("b", [3])
    s.step("a", [4], [0])
    assert m.calls == [("extend", 2, 0), ("extend", 1, 1), ("extend", 1, 0)]


def test_a_failed_step_leaves_no_hidden_row():
    """dp_model_advance: the row that logits may still be computed from is given up when the step's graph is launched, and there again
    only behind the last thing that can fail."""
    with open(os.path.join(os.path.dirname(scheduler.__file__), "csrc", "model.cu")) as f:
        text = f.read()
    at = text.index('extern "C" dp_status dp_model_advance')
    body = text[at:text.index("\n}\n", at)]
    launch, gone, back = (body.index(x) for x in ("dp_graph_launch(", "m->head_row = nullptr;", "m->head_row = m->h;"))
    assert launch < gone < back
    assert not any(x in body[launch:gone].split(";", 1)[1] for x in ("DP_TRY", "DP_CUDA")) and not any(x in body[back:] for x in ("DP_TRY", "DP_CUDA"))
