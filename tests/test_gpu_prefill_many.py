"""Prompts that share passes over the layers against the same prompts one by one."""
import numpy as np
import pytest

from doppler_b200 import synthetic
from doppler_b200.model import DecoderModel
from model_util import gaussian_model_weights

pytestmark = pytest.mark.gpu

CFG = dict(synthetic.MODEL_CONFIGS["small"], n_layers=2)
_weights = []


def weights():
    if not _weights:
        _weights.append(gaussian_model_weights(CFG, 7))
    return _weights[0]


def close(got, want):
    # the same f32-exact products in kernels for other row counts: 22 bits of activations and weights, a few hundred sums
    assert np.sqrt(np.mean((got - want) ** 2)) < 1e-4 * want.std()


@pytest.mark.parametrize("lengths", [[1, 1], [2, 64, 1, 65, 129], [24] * 30, [300, 400, 5, 512, 200, 513, 3]])
def test_same_as_one_by_one(dev, lengths):
    """(activation rows: 768 at this longest sequence, so the last list needs several passes)"""
    n = len(lengths)
    rng = np.random.default_rng(n)
    prompts = [rng.integers(0, CFG["vocab"], k).tolist() for k in lengths]
    more = [rng.integers(0, CFG["vocab"], 1 + k % 7).tolist() for k in lengths]
    seqs = rng.permutation(n).tolist()
    m = DecoderModel(dev, CFG, max_seq=600, max_batch=n)
    m.load_all(weights())
    seen = []
    for many in (False, True):
        m.reset()
        got = []
        for part in (prompts, more):  # a second portion of every sequence starts behind the first
            got.append(m.prefill_many(part, seqs) if many else [m.prefill(p, seq=s) for p, s in zip(part, seqs)])
            got += [m.read_logits(), m.read_hidden(1)]
        got.append([m.seq_len(s) for s in range(n)])
        first = np.empty(n, np.int32)
        first[seqs] = got[3]
        got.append(m.decode(first, 8))
        got.append(m.read_logits(n * CFG["vocab"]))
        seen.append(got)
    one, many = seen
    assert one[0] == many[0] and one[3] == many[3] and one[6] == many[6] and np.array_equal(one[7], many[7])
    for i in (1, 2, 4, 5, 8):
        close(many[i], one[i])
    m.destroy()


def test_nothing_runs_where_a_prompt_is_invalid(dev):
    m = DecoderModel(dev, CFG, max_seq=64, max_batch=3)
    for prompts, seqs in (([[1], []], [0, 1]), ([[1], [CFG["vocab"]]], [0, 1]), ([[1], [2] * 65], [0, 1]), ([[1], [2]], [0, 0]), ([[1], [2]], [0, 3]), ([[1]] * 4, [0, 1, 2, 0])):
        with pytest.raises(RuntimeError):
            m.prefill_many(prompts, seqs)
    for prompts, seqs in (([[1], [2], [3]], [0, 1]), ([[1]], [0, 1]), ([[1]], [])):
        with pytest.raises(ValueError):
            m.prefill_many(prompts, seqs)
    assert [m.seq_len(s) for s in range(3)] == [0, 0, 0]
    m.destroy()
