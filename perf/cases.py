"""The work that is timed: what programs have this library do, through its public entry points.

``listed()`` names the cases, ``draw()`` gives more of the same ranges.  Four kinds:

  matmul     one ``run_matmul`` (Q4_K or f16 weights), as a host pipeline issues it
  attention  one ``run_attention`` over an f16 K/V cache, decode (one query a sequence) or a causal portion
  decoder    ``Scheduler.generate`` of the dense Q4_K decoder: prompts and greedy steps, then the last step's logits
  stack      ``Scheduler.step`` of a decoder described layer by layer: a portion of a prompt with the logits of some of its
             places, then tokens one by one, as a trace of token ids is replayed

Weights and inputs are random, from the seed alone.  Q4_K blocks hold zero-mean weights; the LM head of a decoder is its
embedding with the rows in another order, so that a step's choice stands out as a trained model's does and does not hang
on rounding.
"""
import math

import numpy as np
import torch

from doppler_b200 import fenorax, ops, virolorn
from doppler_b200.model import DecoderModel, StackModel
from doppler_b200.scheduler import Scheduler

GPU = torch.device("cuda")

# layer shapes of the dense decoder (Qwen3-0.6B- and 9B-shaped, and one in between)
SHAPES = {
    "0.6b": dict(hidden=1024, n_heads=16, n_kv_heads=8, head_dim=128, inter=3072),
    "2b": dict(hidden=2048, n_heads=16, n_kv_heads=8, head_dim=128, inter=6144),
    "9b": dict(hidden=4096, n_heads=32, n_kv_heads=8, head_dim=128, inter=12288),
}
# the same widths for the layer-by-layer decoders
FENORAX = {
    "0.6b": dict(width=1024, groups=2, mamba2=dict(heads=32, vdim=64, state=128, groups=2, conv=4, norm_groups=2),
                 attention=dict(heads=16, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5, mask={"size": 2048}), ff=3072),
    "9b": dict(width=4096, groups=4, mamba2=dict(heads=128, vdim=64, state=128, groups=8, conv=4, norm_groups=8),
               attention=dict(heads=32, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5, mask={"size": 8192}), ff=12288),
}
VIROLORN = {"0.6b": dict(width=1024, heads=8, ff=1536, kv_rank=256, q_rank=768, rank=64),
            "9b": dict(width=4096, heads=32, ff=6144, kv_rank=512, q_rank=1536, rank=128)}


def listed():
    return [
        # the smallest call of a host pipeline: one token through one projection of the Qwen3-0.6B shape
        dict(name="matvec small", kind="matmul", M=1, N=3072, K=1024, weights="q4k", act="f32", out="f32", f16_weights=False),
        # a prompt's rows through the gate projection of the 9B shape, f16 activations, default numerics
        dict(name="prompt matmul", kind="matmul", M=512, N=12288, K=4096, weights="q4k", act="f16", out="f16", f16_weights=False),
        # a decode step's attention of a loaded server: 32 sequences at context 8192
        dict(name="batch attention", kind="attention", batch=32, seq=1, kv=8192, heads=32, kv_heads=8, dim=128),
        # a chat turn on the whole Qwen3-0.6B-shaped decoder: prompt, then tokens one by one
        dict(name="chat 0.6b", kind="decoder", shape="0.6b", layers=28, vocab=151936, batch=1, prompt=512, new=64),
        # single-user decoding at the 9B shape (four of its layers; the vocabulary cut by about as much)
        dict(name="decode 9b", kind="decoder", shape="9b", layers=4, vocab=32000, batch=1, prompt=200, new=96),
        # many users at once at the 9B shape: short ragged prompts, then batched steps
        dict(name="batch 9b", kind="decoder", shape="9b", layers=4, vocab=32000, batch=64, prompt=24, new=32),
        # a long prompt at the 9B shape, one answer token (classification, scoring, cache filling)
        dict(name="prompt 9b", kind="decoder", shape="9b", layers=4, vocab=32000, batch=1, prompt=2048, new=1),
        # hybrid decoder: a long prompt
        dict(name="fenorax prompt", kind="stack", arch="Fenorax", size="9b", layers=4, vocab=32000, dtype="bfloat16", prompt=2048, want=1, steps=0),
        # hybrid decoder: tokens one by one behind a short prompt
        dict(name="fenorax steps", kind="stack", arch="Fenorax", size="0.6b", layers=8, vocab=32000, dtype="bfloat16", prompt=100, want=1, steps=64),
        # mixed linear / latent attention decoder: a prompt whose logits are looked at in places (scoring)
        dict(name="virolorn prompt", kind="stack", arch="Virolorn", size="9b", layers=4, vocab=32000, dtype="bfloat16", prompt=1500, want=32, steps=0),
        # the same decoder, tokens one by one
        dict(name="virolorn steps", kind="stack", arch="Virolorn", size="9b", layers=4, vocab=32000, dtype="bfloat16", prompt=60, want=1, steps=48),
        # 32-bit mode (reference runs of a checkpoint): a prompt and a few tokens
        dict(name="fenorax f32", kind="stack", arch="Fenorax", size="0.6b", layers=4, vocab=32000, dtype="float32", prompt=700, want=4, steps=4),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: sizes over their whole ranges, about half of the matrices with the odd sizes that no tile divides."""
    kind = rng.choice(["matmul", "matmul", "matmul", "attention", "attention", "decoder", "decoder", "stack", "stack", "stack"])
    if kind == "matmul":
        while True:
            m, n, k = _log(rng, 1, 1024), _log(rng, 256, 12288), _log(rng, 256, 12288)
            if rng.random() < 0.6:
                n, k = (n + 127) // 128 * 128, (k + 255) // 256 * 256
            if m * n * k <= 512 * 12288 * 4096:
                break
        m = 1 if rng.random() < 0.2 else m
        act = "f32" if m == 1 else rng.choice(["f32", "f16"])
        q4k = m > 64 or rng.random() < 0.8
        return dict(kind=kind, M=m, N=n, K=k, weights="q4k" if q4k else "f16", act=act, out=rng.choice([act, "f32"]),
                    f16_weights=act == "f16" and q4k and rng.random() < 0.3)
    if kind == "attention":
        kv_heads, group, dim = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 8]), rng.choice([64, 128, 128, 256])
        if rng.random() < 0.6:
            kv, most = _log(rng, 16, 16384), 32 * 8192 * 8 * 128
            batch = _log(rng, 1, 64)
            while batch > 1 and batch * kv * kv_heads * dim > most:
                batch //= 2
            return dict(kind=kind, batch=batch, seq=1, kv=kv, heads=kv_heads * group, kv_heads=kv_heads, dim=dim)
        seq = _log(rng, 16, 2048)
        return dict(kind=kind, batch=1, seq=seq, kv=seq + rng.choice([0, _log(rng, 1, 2048)]), heads=kv_heads * group, kv_heads=kv_heads, dim=dim)
    if kind == "decoder":
        shape = rng.choice(sorted(SHAPES))
        batch = rng.choice([1, 1, _log(rng, 2, 96)])
        layers = rng.randint(2, 4 if shape == "9b" else 8)
        return dict(kind=kind, shape=shape, layers=layers, vocab=rng.choice([4096, 32000, 32001]), batch=batch,
                    prompt=_log(rng, 1, 2048) if batch == 1 else _log(rng, 1, 48), new=_log(rng, 1, 64))
    arch, size, dtype = rng.choice(["Fenorax", "Virolorn"]), rng.choice(["0.6b", "9b"]), rng.choice(["bfloat16", "bfloat16", "float32"])
    prompt = _log(rng, 1, 2048 if dtype == "bfloat16" else 700)
    return dict(kind=kind, arch=arch, size=size, layers=4, vocab=rng.choice([4096, 32000]), dtype=dtype, prompt=prompt,
                want=min(prompt, _log(rng, 1, 32)), steps=rng.choice([0, _log(rng, 1, 48)]))


# ------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device=GPU).manual_seed(seed * 1000003 + salt)


def _normal(g, *shape, sigma=1.0, dtype=torch.float32):
    return torch.randn(*shape, generator=g, device=GPU).mul_(sigma).to(dtype)


def q4k_blocks(g, n, k, gain=1.0):
    """[n, blocks of a row, 144] bytes: weights d * sc * q - dmin * m around zero, about gain / sqrt(k) in size."""
    bpr = -(-k // 256)
    d = (gain / math.sqrt(k) / 190.0) * (0.75 + 0.5 * torch.rand(n, bpr, generator=g, device=GPU))
    sc = torch.randint(16, 64, (n, bpr, 8), generator=g, device=GPU, dtype=torch.uint8)
    mn = (sc + torch.randint(0, 5, (n, bpr, 8), generator=g, device=GPU, dtype=torch.uint8) - 2).clamp_(max=63)
    out = torch.empty(n, bpr, 144, dtype=torch.uint8, device=GPU)
    out[:, :, 0:4] = torch.stack([d, 7.5 * d], -1).half().view(torch.uint8)
    out[:, :, 4:8] = sc[..., :4] | (sc[..., 4:] >> 4 << 6)
    out[:, :, 8:12] = mn[..., :4] | (mn[..., 4:] >> 4 << 6)
    out[:, :, 12:16] = (sc[..., 4:] & 15) | ((mn[..., 4:] & 15) << 4)
    out[:, :, 16:] = torch.randint(0, 256, (n, bpr, 128), generator=g, device=GPU, dtype=torch.uint8)
    return out


def q4k_values(blocks, k):
    """The weights of packed blocks, [n, k] in 64 bits."""
    n, bpr, _ = blocks.shape
    d = blocks[:, :, 0:4].contiguous().view(torch.float16).double()
    b = blocks[:, :, 4:16]
    sc = torch.cat([b[..., 0:4] & 63, (b[..., 8:12] & 15) | (b[..., 0:4] >> 6 << 4)], -1).double()
    mn = torch.cat([b[..., 4:8] & 63, (b[..., 8:12] >> 4) | (b[..., 4:8] >> 6 << 4)], -1).double()
    qs = blocks[:, :, 16:].reshape(n, bpr, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], 3).reshape(n, bpr, 8, 32).double()
    w = q * (d[..., :1] * sc).unsqueeze(-1) - (d[..., 1:] * mn).unsqueeze(-1)
    return w.reshape(n, bpr * 256)[:, :k]


_TYPES = {"f32": (torch.float32, "<f4"), "f16": (torch.float16, "<f2"), "q4k": (torch.uint8, "|u1")}


class Owned:
    """A buffer of the pool; it goes back when nothing refers to it any more."""

    def __init__(self, shape, dtype, values=None):
        self.shape, self.typestr = tuple(shape), _TYPES[dtype][1]
        self.buffer = device().acquire_buffer(math.prod(shape) * torch.empty(0, dtype=_TYPES[dtype][0]).element_size())
        if values is not None:
            self.tensor().copy_(values)

    @property
    def __cuda_array_interface__(self):
        return {"data": (self.buffer.device_ptr, False), "shape": self.shape, "typestr": self.typestr, "version": 3}

    def tensor(self):
        """The same memory as a torch tensor, which keeps the buffer."""
        return torch.as_tensor(self, device=GPU)

    def __del__(self):
        if "buffer" in self.__dict__:
            device().release_buffer(self.buffer)
            device().pool_trim()


class Held:
    """What a program keeps between its passes."""

    model = None

    def __del__(self):
        if self.model is not None:
            self.model.destroy()
            device().pool_trim()


_device = None


def device():
    """The program's one open device."""
    global _device
    if _device is None:
        _device = ops.Device(0)
    return _device


# ---- matmul -------------------------------------------------------------------
def matmul_inputs(c, seed):
    g = _gen(seed)
    a = _normal(g, c["M"], c["K"], dtype=_TYPES[c["act"]][0])
    if c["weights"] == "q4k":
        return a, q4k_blocks(g, c["N"], c["K"])
    return a, _normal(g, c["N"], c["K"], sigma=c["K"] ** -0.5, dtype=torch.float16)


def prepare_matmul(c, seed):
    a, w = matmul_inputs(c, seed)
    s = Held()
    s.held = [Owned(a.shape, c["act"], a), Owned(w.shape, c["weights"], w), Owned((c["M"], c["N"]), c["out"])]
    s.A = ops.create_tensor(s.held[0].buffer, c["act"], [c["M"], c["K"]])
    s.B = ops.create_weight_buffer(s.held[1].buffer, c["weights"], "row", [c["N"], c["K"]])
    s.out, s.seen, s.case = s.held[2].buffer, s.held[2].tensor(), c
    return s


def run_matmul(s):
    c = s.case
    ops.run_matmul(s.A, s.B, c["M"], c["N"], c["K"], output_buffer=s.out, output_dtype=c["out"], f16_weights=c["f16_weights"])
    return s.seen


def exact_matmul(c, seed):
    a, w = matmul_inputs(c, seed)
    if c["weights"] == "q4k":
        w = q4k_values(w, c["K"])
        if c["f16_weights"]:
            w = w.float().half()
    return a.double() @ w.double().T


# ---- attention ----------------------------------------------------------------
def attention_inputs(c, seed):
    g = _gen(seed)
    return (_normal(g, c["batch"], c["seq"], c["heads"], c["dim"]), _normal(g, c["batch"], c["kv"], c["kv_heads"], c["dim"], dtype=torch.float16),
            _normal(g, c["batch"], c["kv"], c["kv_heads"], c["dim"], dtype=torch.float16))


def prepare_attention(c, seed):
    q, k, v = attention_inputs(c, seed)
    s = Held()
    s.held = [Owned(q.shape, "f32", q), Owned(k.shape, "f16", k), Owned(v.shape, "f16", v), Owned(q.shape, "f32")]
    s.Q, s.K, s.V = (ops.create_tensor(h.buffer, dtype, [h.shape[0] * h.shape[1], h.shape[2], h.shape[3]]) for h, dtype in zip(s.held, ("f32", "f16", "f16")))
    s.out, s.seen, s.case = s.held[3].buffer, s.held[3].tensor(), c
    return s


def run_attention(s):
    c = s.case
    ops.run_attention(s.Q, s.K, s.V, None, c["heads"], c["dim"], seq_len=c["seq"], kv_len=c["kv"], num_kv_heads=c["kv_heads"], causal=c["seq"] > 1,
                      start_pos=c["kv"] - c["seq"], batch=c["batch"], kv_batch_stride=c["kv"] * c["kv_heads"] * c["dim"], output_buffer=s.out)
    return s.seen


def attend(q, k, v, scale, see=None):
    """q [T, H, D], k [S, G, D], v [S, G, V] in 64 bits; see [T, S] says which keys a query may look at."""
    T, H, D = q.shape
    S, G, V = v.shape
    s = torch.einsum("tgrd,sgd->grts", q.reshape(T, G, H // G, D), k) * scale
    if see is not None:
        s.masked_fill_(~see, -math.inf)
    return torch.einsum("grts,sgv->tgrv", torch.softmax(s, -1), v).reshape(T, H, V)


def causal(T, S, chunk=0):
    """Rows at the last T of S positions."""
    i, j = torch.arange(S - T, S, device=GPU)[:, None], torch.arange(S, device=GPU)[None]
    return (j <= i) & (i // chunk == j // chunk) if chunk else j <= i


def exact_attention(c, seed):
    q, k, v = attention_inputs(c, seed)
    see = causal(c["seq"], c["kv"]) if c["seq"] > 1 else None
    return torch.stack([attend(q[b].double(), k[b].double(), v[b].double(), c["dim"] ** -0.5, see) for b in range(c["batch"])])


# ---- dense decoder ----------------------------------------------------------------
def decoder_config(c):
    return dict(SHAPES[c["shape"]], n_layers=c["layers"], vocab=c["vocab"], eps=1e-6, rope_theta=1e6)


def decoder_matrices(z):
    q, kv, h, i = z["n_heads"] * z["head_dim"], z["n_kv_heads"] * z["head_dim"], z["hidden"], z["inter"]
    return {"wq": (q, h, 1.0), "wk": (kv, h, 1.0), "wv": (kv, h, 1.0), "wo": (h, q, 0.5), "wgate": (i, h, 1.0), "wup": (i, h, 1.0), "wdown": (h, i, 0.7)}


def decoder_layer(c, seed, layer):
    z, g = decoder_config(c), _gen(seed, 10 + layer)
    w = {name: q4k_blocks(g, n, k, gain) for name, (n, k, gain) in decoder_matrices(z).items()}
    for name in ("in_norm", "post_norm", "q_norm", "k_norm"):
        w[name] = 1.0 + _normal(g, z["head_dim"] if name in ("q_norm", "k_norm") else z["hidden"], sigma=0.1)
    return w


def decoder_tables(c, seed):
    """embedding, LM head (the embedding in another order), final norm"""
    z, g = decoder_config(c), _gen(seed, 1)
    embed = _normal(g, c["vocab"], z["hidden"], dtype=torch.float16)
    head = (embed[torch.randperm(c["vocab"], generator=g, device=GPU)] * 0.05).half()
    return embed, head, 1.0 + _normal(g, z["hidden"], sigma=0.1)


def decoder_prompts(c, seed):
    """Prompts of a batch are ragged: half to all of the length."""
    rng = np.random.default_rng(seed)
    lengths = [c["prompt"]] + [int(rng.integers((c["prompt"] + 1) // 2, c["prompt"] + 1)) for _ in range(c["batch"] - 1)]
    return [rng.integers(0, c["vocab"], n).tolist() for n in lengths]


def prepare_decoder(c, seed):
    s = Held()
    s.model = DecoderModel(device(), decoder_config(c), c["prompt"] + c["new"], c["batch"])
    for i in range(c["layers"]):
        s.model.load_layer(i, {name: w.cpu().numpy() for name, w in decoder_layer(c, seed, i).items()})
    embed, head, norm = decoder_tables(c, seed)
    s.model.load_embed(embed.cpu().numpy())
    s.model.load_lm_head(head.cpu().numpy())
    s.model.load_final_norm(norm.cpu().numpy())
    s.scheduler, s.prompts, s.case = Scheduler(s.model), decoder_prompts(c, seed), c
    return s


def run_decoder(s):
    c = s.case
    tokens = s.scheduler.generate(s.prompts, c["new"])
    rows = c["batch"] if c["new"] > 1 else 1
    return {"tokens": np.asarray(tokens, np.int64), "logits": s.model.read_logits(rows * c["vocab"]).reshape(rows, c["vocab"])}


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def rotate(x, pos, base, single=False):
    """x [T, ..., R], dimension i turned with dimension i + R / 2; ``single``: frequencies are numbers of 32 bits."""
    half = x.shape[-1] // 2
    f = base ** (-2.0 * torch.arange(half, device=GPU, dtype=torch.float64) / x.shape[-1])
    a = pos.double()[:, None] * (f.float().double() if single else f)
    a = a.reshape((x.shape[0],) + (1,) * (x.dim() - 2) + (half,))
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def exact_decoder(c, seed):
    z, B, D = decoder_config(c), c["batch"], 128
    H, G, eps = z["n_heads"], z["n_kv_heads"], z["eps"]
    layers = []
    for i in range(c["layers"]):
        w, m = decoder_layer(c, seed, i), decoder_matrices(z)
        layers.append({n: q4k_values(x, m[n][1]) if n in m else x.double() for n, x in w.items()})
    embed, head, norm = decoder_tables(c, seed)
    norm = norm.double()
    cache = [[[None, None] for _ in range(B)] for _ in layers]

    def forward(ids, spans):
        """Rows of several sequences; spans: (sequence, first row, end, position of the first row)."""
        x = embed[ids].double()
        pos = torch.cat([torch.arange(p, p + e - a, device=GPU) for _, a, e, p in spans])
        for w, kv in zip(layers, cache):
            h = rms(x, eps) * w["in_norm"]
            q, k, v = ((h @ w[n].T).reshape(len(ids), -1, D) for n in ("wq", "wk", "wv"))
            q, k = (rotate(rms(t, eps) * w[n], pos, z["rope_theta"], True) for t, n in ((q, "q_norm"), (k, "k_norm")))
            o = torch.empty_like(q)
            for b, a, e, p in spans:
                for j, t in ((0, k), (1, v)):
                    new = t[a:e].float().half().double()  # the cache holds 16-bit numbers
                    kv[b][j] = new if p == 0 else torch.cat([kv[b][j], new])
                o[a:e] = attend(q[a:e], kv[b][0], kv[b][1], D ** -0.5, causal(e - a, p + e - a))
            x = x + o.reshape(len(ids), H * D) @ w["wo"].T
            h = rms(x, eps) * w["post_norm"]
            x = x + (torch.nn.functional.silu(h @ w["wgate"].T) * (h @ w["wup"].T)) @ w["wdown"].T
        return x

    def logits(x):
        h = rms(x, eps) * norm
        return torch.cat([h @ part.double().T for part in head.split(16384)], -1)

    held, done = [], []
    for b, prompt in enumerate(decoder_prompts(c, seed)):
        x = forward(torch.tensor(prompt, device=GPU), [(b, 0, len(prompt), 0)])
        last = logits(x[-1:])
        held.append(len(prompt))
        done.append([int(last.argmax())])
    for _ in range(c["new"] - 1):
        x = forward(torch.tensor([d[-1] for d in done], device=GPU), [(b, b, b + 1, held[b]) for b in range(B)])
        last = logits(x)
        for b, t in enumerate(last.argmax(-1).tolist()):
            done[b].append(t)
            held[b] += 1
    return {"tokens": np.asarray(done, np.int64), "logits": last}


# ---- decoders described layer by layer ----------------------------------------------
def stack_config(c):
    if c["arch"] == "Fenorax":
        z = FENORAX[c["size"]]
        entry = lambda i: ({"type": "attention", "mixer": z["attention"], "mlp": {"kind": "dense", "ff": z["ff"], "limit": 7.0}} if i % 4 == 3  # noqa: E731
                           else {"type": "mamba2", "mixer": z["mamba2"], "mlp": None})
        return {"architecture": "Fenorax", "width": z["width"], "vocab": c["vocab"], "streams": 4, "canon": {"taps": 4},
                "norm": {"groups": z["groups"], "eps": 1e-6}, "embedding": {"scale": 1.0}, "layers": [entry(i) for i in range(c["layers"])]}
    z = VIROLORN[c["size"]]
    H, mlp = z["heads"], {"kind": "dense", "ff": z["ff"]}
    delta = {"type": "channel_delta", "mixer": {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4}, "mlp": mlp}
    lightning = {"type": "lightning", "mixer": {"heads": H, "dim": 128, "vdim": 128, "decay": [math.exp(-2.0 ** (-8.0 * (h + 1) / H)) for h in range(H)]}, "mlp": mlp}
    latent = {"type": "latent_attention", "mlp": mlp,
              "mixer": {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": z["kv_rank"], "q_rank": z["q_rank"], "scale": 192.0 ** -0.5,
                        "rot": {"base": 1e6, "dims": 64}}}
    return {"architecture": "Virolorn", "width": z["width"], "vocab": c["vocab"], "norm": {"eps": 1e-6}, "residual_mult": 0.5,
            "layers": [(delta, lightning, delta, latent)[i % 4] for i in range(c["layers"])]}


def stack_weights(c, seed):
    """name -> bfloat16 tensor"""
    cfg, g, w = stack_config(c), _gen(seed, 2), {}
    W = cfg["width"]

    def put(name, x):
        w[name] = x.bfloat16()

    def lin(name, n, k, gain=1.0):
        put(name, _normal(g, n, k, sigma=gain / math.sqrt(k)))

    def near_one(name, n):
        put(name, 1.0 + _normal(g, n, sigma=0.1))

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, device=GPU)

    put("embed", _normal(g, c["vocab"], W))
    near_one("final.norm", W)
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}."
        H, V = m["heads"], m["vdim"]
        if c["arch"] == "Fenorax":
            S = cfg["streams"]
            for q in ("1", "2") if layer["mlp"] else ("1",):
                near_one(p + "norm" + q, W)
                put(p + "canon" + q, _normal(g, W, cfg["canon"]["taps"], sigma=0.2))
                put(p + f"hc{q}.in", uniform(0.2, 0.4, S))
                put(p + f"hc{q}.out", uniform(0.3, 0.7, S))
                put(p + f"hc{q}.mix", torch.eye(S, device=GPU) * 0.85 + uniform(0.0, 0.08, S, S))
        else:
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                near_one(p + n, W)
        lin(p + "mix.o", W, H * V)
        if layer["type"] == "mamba2":
            ch = H * V + 2 * m["groups"] * m["state"]
            lin(p + "mix.in", H * V + ch + H, W)
            put(p + "mix.conv", _normal(g, ch, m["conv"], sigma=0.5))
            put(p + "mix.conv.b", _normal(g, ch, sigma=0.1))
            put(p + "mix.dt_bias", uniform(-2.5, 0.5, H))
            put(p + "mix.A_log", uniform(-2.5, 1.0, H))
            put(p + "mix.D", _normal(g, H))
            near_one(p + "mix.norm", H * V)
        elif layer["type"] == "attention":
            lin(p + "mix.q", H * m["dim"], W)
            lin(p + "mix.k", m["kv_heads"] * m["dim"], W)
            lin(p + "mix.v", m["kv_heads"] * V, W)
            lin(p + "mix.g", H, W)
        elif layer["type"] == "lightning":
            for t, n in (("q", H * m["dim"]), ("k", H * m["dim"]), ("v", H * V), ("g", H * V)):
                lin(p + "mix." + t, n, W)
            near_one(p + "mix.norm", H * V)
        elif layer["type"] == "channel_delta":
            QK, rank = m["kv_heads"] * m["dim"], VIROLORN[c["size"]]["rank"]
            for t, n in (("q", QK), ("k", QK), ("v", H * V)):
                lin(p + "mix." + t, n, W)
                put(p + f"mix.{t}.conv", _normal(g, n, m["conv"], sigma=0.5))
            lin(p + "mix.b", H, W)
            put(p + "mix.A_log", uniform(-3.0, 1.0, H))
            put(p + "mix.dt_bias", uniform(-3.0, 0.5, H * m["dim"]))
            lin(p + "mix.a1", rank, W)
            lin(p + "mix.a2", H * m["dim"], rank)
            lin(p + "mix.g1", rank, W)
            lin(p + "mix.g2", H * V, rank)
            near_one(p + "mix.norm", V)
        else:
            R, K, Q = m["rot_dim"], m["kv_rank"], m["q_rank"]
            lin(p + "mix.dq", Q, W)
            near_one(p + "mix.dq.norm", Q)
            lin(p + "mix.uq", H * (m["dim"] + R), Q)
            lin(p + "mix.dkv", K + R, W)
            near_one(p + "mix.dkv.norm", K)
            lin(p + "mix.uk", H * m["dim"], K)
            lin(p + "mix.uv", H * V, K)
            lin(p + "mix.g", H, W)
        if layer["mlp"]:
            lin(p + "mlp.gate", layer["mlp"]["ff"], W)
            lin(p + "mlp.up", layer["mlp"]["ff"], W)
            lin(p + "mlp.down", W, layer["mlp"]["ff"])
    return w


def stack_tokens(c, seed):
    """the prompt, the places whose logits are wanted, the tokens behind it"""
    t = np.random.default_rng(seed).integers(0, c["vocab"], c["prompt"] + c["steps"])
    want = sorted({c["prompt"] - 1 - (c["prompt"] * j) // c["want"] for j in range(c["want"])})
    return t[:c["prompt"]].tolist(), want, t[c["prompt"]:].tolist()


def prepare_stack(c, seed):
    s, w, cfg = Held(), stack_weights(c, seed), stack_config(c)
    design = fenorax if c["arch"] == "Fenorax" else virolorn
    shape = {n: tuple(x.shape) for n, x in w.items()}.get
    stack, layers = design.stack_config(cfg) if design is fenorax else design.stack_config(cfg, shape)
    s.model = StackModel(device(), stack, layers, c["prompt"] + c["steps"], 1, c["dtype"])
    design.load_weights(s.model, lambda n: w[n].view(torch.int16).cpu().numpy().view(np.uint16))
    s.scheduler, s.case = Scheduler(s.model), c
    s.prompt, s.want, s.tokens = stack_tokens(c, seed)
    return s


def run_stack(s):
    rows = [s.scheduler.step("trace", s.prompt, s.want)]
    for i, t in enumerate(s.tokens):
        rows.append(s.scheduler.step("trace", [t], [0] if i == len(s.tokens) - 1 else []))
    s.scheduler.finish("trace")
    return np.concatenate(rows)


def short_conv(x, w, b=None):
    """x [T, C], w [C, taps]: the last column multiplies the row itself."""
    T, taps = x.shape[0], w.shape[1]
    pad = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(pad[j:j + T] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def group_rms(x, w, groups, eps):
    return rms(x.reshape(x.shape[0], groups, -1), eps).reshape(x.shape) * w


def decayed_states(a, k, v, q):
    """S <- a S + k v', o = S' q over time; a [T, H] or [H], k and q [T, H, N], v [T, H, V]"""
    S, o = k.new_zeros(k.shape[1], k.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(k.shape[0]):
        S = S * (a[t] if a.dim() == 2 else a)[:, None, None] + k[t][:, :, None] * v[t][:, None]
        o[t] = torch.einsum("hnv,hn->hv", S, q[t])
    return o


def mamba2(h, m, w, eps):
    T, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    gate, xbc, dt = (h @ w["in"].T).split([H * P, H * P + 2 * G * N, H], -1)
    x, B, C = torch.nn.functional.silu(short_conv(xbc, w["conv"], w["conv.b"])).split([H * P, G * N, G * N], -1)
    x, B, C = x.reshape(T, H, P), B.reshape(T, G, N).repeat_interleave(H // G, 1), C.reshape(T, G, N).repeat_interleave(H // G, 1)
    dt = torch.nn.functional.softplus(dt + w["dt_bias"], threshold=1e9)
    y = decayed_states(torch.exp(-torch.exp(w["A_log"]) * dt), B * dt[:, :, None], x, C) + w["D"][:, None] * x
    return group_rms(y.reshape(T, H * P) * torch.nn.functional.silu(gate), w["norm"], m["norm_groups"], eps)


def chunk_attention(h, m, w, eps):
    T = h.shape[0]
    q, k = rms((h @ w["q"].T).reshape(T, -1, m["dim"]), eps), rms((h @ w["k"].T).reshape(T, -1, m["dim"]), eps)
    o = attend(q, k, (h @ w["v"].T).reshape(T, -1, m["vdim"]), m["scale"], causal(T, T, m["mask"]["size"]))
    return (o * torch.sigmoid(h @ w["g"].T)[:, :, None]).reshape(T, -1)


def lightning(h, m, w, eps):
    T, H = h.shape[0], m["heads"]
    q, k, v = (torch.nn.functional.silu(h @ w[n].T).reshape(T, H, -1) for n in ("q", "k", "v"))
    o = decayed_states(torch.tensor(m["decay"], dtype=torch.float64, device=GPU), k, v, q).reshape(T, -1)
    return rms(o, eps) * w["norm"] * torch.sigmoid(h @ w["g"].T)


def channel_delta(h, m, w, eps):
    T, H, D = h.shape[0], m["heads"], m["dim"]
    q, k, v = (torch.nn.functional.silu(short_conv(h @ w[n].T, w[n + ".conv"])) for n in ("q", "k", "v"))
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q, k = (unit(x.reshape(T, m["kv_heads"], D)).repeat_interleave(H // m["kv_heads"], 1) for x in (q, k))
    q, v = q / math.sqrt(D), v.reshape(T, H, -1)
    a = (h @ w["a1"].T) @ w["a2"].T + w["dt_bias"]
    g = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a, threshold=1e9).reshape(T, H, D))
    beta = torch.sigmoid(h @ w["b"].T)
    S, o = v.new_zeros(H, D, v.shape[2]), torch.empty_like(v)
    for t in range(T):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        o[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return (rms(o, eps) * w["norm"]).reshape(T, -1) * torch.sigmoid((h @ w["g1"].T) @ w["g2"].T)


def latent_attention(h, m, w, eps):
    T, H, D, K, base = h.shape[0], m["heads"], m["dim"], m["kv_rank"], m["rot"]["base"]
    pos = torch.arange(T, device=GPU)
    q = ((rms(h @ w["dq"].T, eps) * w["dq.norm"]) @ w["uq"].T).reshape(T, H, -1)
    down = h @ w["dkv"].T
    lat = rms(down[:, :K], eps) * w["dkv.norm"]
    turned = rotate(down[:, K:], pos, base)[:, None].expand(T, H, -1)
    q = torch.cat([q[..., :D], rotate(q[..., D:], pos, base)], -1)
    k = torch.cat([(lat @ w["uk"].T).reshape(T, H, D), turned], -1)
    o = attend(q, k, (lat @ w["uv"].T).reshape(T, H, -1), m["scale"], causal(T, T))
    return (o * torch.sigmoid(h @ w["g"].T)[:, :, None]).reshape(T, -1)


MIXERS = {"mamba2": mamba2, "attention": chunk_attention, "lightning": lightning, "channel_delta": channel_delta, "latent_attention": latent_attention}


def exact_stack(c, seed):
    cfg, held = stack_config(c), stack_weights(c, seed)
    prompt, want, tail = stack_tokens(c, seed)
    eps, fen = cfg["norm"]["eps"], c["arch"] == "Fenorax"
    x = held["embed"][torch.tensor(prompt + tail, device=GPU)].double()
    if fen:
        xs = x.expand(cfg["streams"], -1, -1)
    for i, layer in enumerate(cfg["layers"]):
        w = {n[len(f"l{i}."):]: v.double() for n, v in held.items() if n.startswith(f"l{i}.")}
        mix = {n[4:]: v for n, v in w.items() if n.startswith("mix.")}
        for q in ("1", "2") if layer["mlp"] else ("1",):
            if fen:
                h = group_rms(torch.einsum("s,stc->tc", w[f"hc{q}.in"], xs), w["norm" + q], cfg["norm"]["groups"], eps)
                h = h + short_conv(h, w["canon" + q])
            else:
                h = rms(x, eps) * w["norm" + q]
            if q == "1":
                y = MIXERS[layer["type"]](h, layer["mixer"], mix, eps) @ mix["o"].T
            elif fen:
                a, b = (h @ w["mlp.gate"].T).clamp(max=layer["mlp"]["limit"]), (h @ w["mlp.up"].T).clamp(-layer["mlp"]["limit"], layer["mlp"]["limit"])
                y = (a * torch.sigmoid(1.702 * a) * (b + 1.0)) @ w["mlp.down"].T
            else:
                y = (torch.nn.functional.silu(h @ w["mlp.gate"].T) * (h @ w["mlp.up"].T)) @ w["mlp.down"].T
            if fen:
                xs = torch.einsum("st,snc->tnc", w[f"hc{q}.mix"], xs) + w[f"hc{q}.out"][:, None, None] * y
            else:
                x = x + cfg["residual_mult"] * rms(y, eps) * w[f"norm{q}b"]
    rows = want + ([len(prompt) + len(tail) - 1] if tail else [])
    x = xs.sum(0)[rows] if fen else x[rows]
    h = group_rms(x, held["final.norm"].double(), cfg["norm"]["groups"] if fen else 1, eps)
    return h @ held["embed"].double().T


# ------------------------------------------------------------------------------
# one pass, what it cannot do without, how far another implementation may be off
# ------------------------------------------------------------------------------
_PREPARE = {"matmul": prepare_matmul, "attention": prepare_attention, "decoder": prepare_decoder, "stack": prepare_stack}
_RUN = {"matmul": run_matmul, "attention": run_attention, "decoder": run_decoder, "stack": run_stack}
_EXACT = {"matmul": exact_matmul, "attention": exact_attention, "decoder": exact_decoder, "stack": exact_stack}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state.case["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def _q4k_bytes(n, k):
    return n * -(-k // 256) * 144


def _stack_counts(c):
    """(bytes of the layers' matrices, operations of one token through them, bytes of recurrent state, bytes of one cached row)"""
    cfg = stack_config(c)
    W, weights, ops_, state, row = cfg["width"], 0, 0, 0, 0
    elem = 2 if c["dtype"] == "bfloat16" else 4
    for layer in cfg["layers"]:
        m, t = layer["mixer"], layer["type"]
        H, V = m["heads"], m["vdim"]
        n = W * H * V
        if t == "mamba2":
            n += W * (2 * H * V + 2 * m["groups"] * m["state"] + H)
            state += 4 * H * V * m["state"]
            ops_ += 4 * H * V * m["state"]
        elif t == "attention":
            n += W * (H * m["dim"] + m["kv_heads"] * (m["dim"] + V) + H)
            row += elem * m["kv_heads"] * (m["dim"] + V)
        elif t == "lightning":
            n += W * (2 * H * m["dim"] + 2 * H * V)
            state += 4 * H * V * m["dim"]
            ops_ += 4 * H * V * m["dim"]
        elif t == "channel_delta":
            rank = VIROLORN[c["size"]]["rank"]
            n += W * (2 * m["kv_heads"] * m["dim"] + H * V + H + 2 * rank) + rank * H * (m["dim"] + V)
            state += 4 * H * V * m["dim"]
            ops_ += 6 * H * V * m["dim"]
        else:
            n += W * (m["q_rank"] + m["kv_rank"] + m["rot_dim"] + H) + m["q_rank"] * H * (m["dim"] + m["rot_dim"]) + m["kv_rank"] * H * (m["dim"] + V)
            row += elem * (m["kv_rank"] + m["rot_dim"])
        if layer["mlp"]:
            n += 3 * W * layer["mlp"]["ff"]
        weights += 2 * n
        ops_ += 2 * n
    return weights, ops_, state, row


def work(case):
    c = case
    if c["kind"] == "matmul":
        size = {"f32": 4, "f16": 2}
        w = _q4k_bytes(c["N"], c["K"]) if c["weights"] == "q4k" else 2 * c["N"] * c["K"]
        return {"bytes": w + c["M"] * (c["K"] * size[c["act"]] + c["N"] * size[c["out"]]), "flops": 2 * c["M"] * c["N"] * c["K"]}
    if c["kind"] == "attention":
        pairs = c["kv"] if c["seq"] == 1 else c["seq"] * (2 * c["kv"] - c["seq"] + 1) // 2
        return {"bytes": c["batch"] * (4 * c["kv"] * c["kv_heads"] * c["dim"] + 8 * c["seq"] * c["heads"] * c["dim"]),
                "flops": 4 * c["batch"] * pairs * c["heads"] * c["dim"]}
    if c["kind"] == "decoder":
        z = decoder_config(c)
        weights = c["layers"] * sum(_q4k_bytes(n, k) for n, k, _ in decoder_matrices(z).values())
        per_token = 2 * c["layers"] * sum(n * k for n, k, _ in decoder_matrices(z).values())
        head, row = 2 * c["vocab"] * z["hidden"], 4 * c["layers"] * z["n_kv_heads"] * z["head_dim"]
        pair = 4 * c["layers"] * z["n_heads"] * z["head_dim"]
        B, T, n = c["batch"], c["prompt"], c["new"]
        # prompts: the weights once each; steps: weights once, every sequence's cached rows
        rows = sum(T + s + 1 for s in range(n - 1))
        return {"bytes": (B + n - 1) * (weights + head) + B * (rows + T) * row,
                "flops": B * ((T + n - 1) * per_token + n * head + pair * (T * (T + 1) // 2 + rows))}
    weights, per_token, state, row = _stack_counts(c)
    cfg = stack_config(c)
    head, T, n = 2 * c["vocab"] * cfg["width"], c["prompt"], c["steps"]
    heads = [l["mixer"] for l in cfg["layers"] if l["type"] in ("attention", "latent_attention")]
    pair = sum(2 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"]) for m in heads)
    rows = sum(T + s + 1 for s in range(n))
    return {"bytes": (1 + n) * weights + (2 if n else 1) * head + (1 + 2 * n) * state + (rows + T) * row,
            "flops": (T + n) * per_token + (c["want"] + (1 if n else 0)) * head + pair * (T * (T + 1) // 2 + rows)}


def tolerance(case):
    """About four times what is seen against ``exact``: f32 sums, f16 or bf16 roundings where the types have them."""
    c = case
    if c["kind"] == "matmul":
        return {"rel": 9e-4, "max": 5e-3} if c["out"] == "f16" or c["f16_weights"] else {"rel": 2.5e-5, "max": 1e-4}
    if c["kind"] == "attention":  # more than four heads a group: the weights of a decode step enter as 16-bit numbers
        return {"rel": 7e-4, "max": 3e-3} if c["heads"] > 4 * c["kv_heads"] else {"rel": 7e-6, "max": 5e-5}
    if c["kind"] == "decoder":
        return {"rel": 2e-4, "max": 2e-3, "differ": 0.005}
    return {"rel": 1.4e-2 if c["dtype"] == "bfloat16" else 5e-6, "max": 0.1 if c["dtype"] == "bfloat16" else 5e-5}
