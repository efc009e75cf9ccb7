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


def test_logits_behind_a_shared_pass(dev):
    """The head after a shared pass is the one-row head: f32 products and sums, not f16 halves."""
    m = DecoderModel(dev, CFG, max_seq=64, max_batch=5)
    m.load_all(weights())
    H, V, last = CFG["hidden"], CFG["vocab"], 30
    m.prefill_many([np.arange(k) * 7 % V for k in (5, 9, 2, 33, last)], range(5))
    x = m.read_hidden(last)[-1].astype(np.float64)  # (the last prompt's rows come first)
    w = weights()
    want = (x / np.sqrt(np.mean(x * x) + CFG["eps"]) * w["final_norm"]) @ w["lm_head"].astype(np.float64).T
    got = m.read_logits(V)
    # 1024 products in f32: 1.2e-7 with lanes that add 32 of them each, and the rounding of the normalised row
    assert np.linalg.norm(got - want) < 4e-7 * np.linalg.norm(want)
    m.destroy()


@pytest.mark.parametrize("lengths", [[3, 2, 1], [1, 1], [1, 4, 1, 5, 1], [64, 1, 300, 1]])
def test_prompts_of_one_token(dev, lengths):
    """A prompt of one token is computed as by itself, bit for bit."""
    m = DecoderModel(dev, CFG, max_seq=320, max_batch=len(lengths))
    m.load_all(weights())
    prompts = [(np.arange(k) * 11 + 3 * i) % CFG["vocab"] for i, k in enumerate(lengths)]
    n = len(lengths) - 1
    one = [m.prefill(p, seq=i) for i, p in enumerate(prompts)]
    logits, hidden = m.read_logits(CFG["vocab"]), m.read_hidden()
    m.reset()
    assert m.prefill_many(prompts, range(n + 1)) == one
    assert [m.seq_len(i) for i in range(n + 1)] == lengths
    if lengths[-1] == 1:
        assert np.array_equal(m.read_logits(CFG["vocab"]), logits) and np.array_equal(m.read_hidden(), hidden)
    # every sequence goes on from its own state
    follow = [m.extend([5], [0], i) for i in range(n + 1)]
    m.reset()
    for i, p in enumerate(prompts):
        m.prefill(p, seq=i)
    for i, k in enumerate(lengths):
        want = m.extend([5], [0], i)
        assert np.array_equal(follow[i], want) if k == 1 else np.sqrt(np.mean((follow[i] - want) ** 2)) < 1e-4 * want.std()
    m.destroy()


@pytest.mark.parametrize("batch", [65, 71, 96])
def test_steps_of_more_sequences_than_the_small_batch_kernel_takes(dev, batch):
    """Decode steps beyond 64 sequences (another GEMM inside the step's graph): the same step after step, and the logits of the
    same sequences in smaller groups."""
    rng = np.random.default_rng(batch)
    prompts = [rng.integers(0, CFG["vocab"], 2 + i % 3).tolist() for i in range(batch)]
    V, rows = CFG["vocab"], []
    for most in (batch, batch, 32):
        out = []
        m = DecoderModel(dev, CFG, max_seq=16, max_batch=most)
        m.load_all(weights())
        for i in range(0, batch, most):
            part = prompts[i:i + most]
            m.reset()
            m.decode(m.prefill_many(part, range(len(part))), 5)
            out.append(m.read_logits(len(part) * V).reshape(len(part), V))
        m.destroy()
        rows.append(np.concatenate(out))
    assert np.array_equal(rows[0], rows[1])
    # f32-exact products in another kernel, and cache entries on the other side of a rounding boundary
    assert (np.linalg.norm(rows[0] - rows[2], axis=1) < 2e-3 * np.linalg.norm(rows[2], axis=1)).all()
