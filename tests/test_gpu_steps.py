"""Single steps without logits (dp_model_advance) against decode steps: the same state, the same logits whenever they are asked for."""
import numpy as np
import pytest

import fenorax_util as fu
import virolorn_util as vu
from doppler_b200 import _lib as L
from doppler_b200 import synthetic
from doppler_b200.model import DecoderModel
from doppler_b200.scheduler import Scheduler
from model_util import gaussian_model_weights

pytestmark = pytest.mark.gpu
MAX_SEQ = 40


def dense(dev):
    cfg = dict(synthetic.MODEL_CONFIGS["tiny"])
    m = DecoderModel(dev, cfg, max_seq=MAX_SEQ)
    m.load_all(gaussian_model_weights(cfg, 7))
    return m


def fenorax(dev):
    cfg = fu.config([fu.mamba(), fu.attention()])
    return fu.build(dev, cfg, fu.weights(cfg), MAX_SEQ)


def fenorax_one_stream(dev):
    cfg = fu.config([fu.mamba(), fu.attention()], streams=1)
    return fu.build(dev, cfg, fu.weights(cfg), MAX_SEQ, dtype="bfloat16")


def virolorn(dev):
    cfg = vu.config([vu.delta(mlp={"kind": "dense", "ff": 40}), vu.lightning(), vu.latent()])
    return vu.build(dev, cfg, vu.weights(cfg), MAX_SEQ)


def close(a, b):
    """Equal but for the order of a few f32 sums in front of the table (the residual's end in a kernel of its own)."""
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    assert np.abs(a - b).max() <= 2e-5 * np.sqrt((b * b).mean()), np.abs(a - b).max()


@pytest.mark.parametrize("model", [dense, fenorax, fenorax_one_stream, virolorn])
def test_steps_without_logits(dev, model):
    m = model(dev)
    t = np.random.default_rng(5).integers(0, m.cfg["vocab"], 24).tolist()
    want, hidden = [], []
    m.extend(t[:6])
    for x in t[6:]:
        m.decode([x], 1)
        want.append(m.read_logits())
        hidden.append(m.read_hidden())
    m.release(0)
    m.extend(t[:6])
    for i, x in enumerate(t[6:]):
        m.advance(x)
        close(m.read_hidden(), hidden[i])
        if i % 3 == 0:
            close(m.read_logits(), want[i])
            close(m.read_logits(), want[i])  # and again
    assert m.seq_len() == len(t)
    # what overwrites the hidden row first puts it aside, or has logits of its own
    rows = []
    for step in (lambda x: m.decode([x], 1), m.advance):
        m.release(0)
        m.extend(t[:6])
        step(t[6])
        m.extend(t[7:8])
        m.extend(t[8:9])
        rows.append([m.read_logits()])
        step(t[9])
        rows[-1].append(m.extend(t[10:12], [1])[0])
        rows[-1].append(m.read_logits())
        step(t[12])
        m.decode([t[13]], 1)
        rows[-1].append(m.read_logits())
    close(rows[1], rows[0])
    # through the scheduler, some steps wanted
    m.release(0)
    s = Scheduler(m)
    s.step("a", t[:6])
    for i, x in enumerate(t[6:]):
        rows = s.step("a", [x], [0] if i % 4 == 1 else [])
        assert rows.shape == (1 if i % 4 == 1 else 0, m.cfg["vocab"])
        if len(rows):
            close(rows[0], want[i])
    s.finish("a")
    m.destroy()


@pytest.mark.parametrize("model", [dense, fenorax])
def test_new_weights_behind_a_step(dev, model):
    """The logits of a step are those of the weights that it ran with."""
    m = model(dev)
    m.extend([1, 2, 3])
    m.decode([4], 1)
    want = m.read_logits()
    for load in range(2):
        m.release(0)
        m.extend([1, 2, 3])
        m.advance(4)
        if model is dense:
            rows = np.zeros((m.cfg["vocab"], m.cfg["hidden"]), np.float16)
            m.load_final_norm(np.zeros(m.cfg["hidden"], np.float32)) if load else m.load_lm_head(rows)
        else:
            shape = (m.cfg["hidden"],) if load else (m.cfg["vocab"], m.cfg["hidden"])
            m.load_tensor(-1, L.T_FINAL_NORM if load else L.T_EMBED, np.zeros(shape, np.uint16))
        close(m.read_logits(), want)
        m.destroy()
        m = model(dev)
    m.destroy()


def test_errors(dev):
    m = fenorax(dev)
    m.extend([1] * (MAX_SEQ - 1))
    m.advance(2)
    for bad in (2, -1, m.cfg["vocab"]):  # no room; outside the vocabulary
        with pytest.raises(Exception, match="advance"):
            m.advance(bad)
    assert m.seq_len() == MAX_SEQ
    m.destroy()
