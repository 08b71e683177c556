"""Performance cases: what programs have this library do, through its public entry points.

Eight kinds of work, each over a range of sizes:

  llama_decode      greedy decode steps of a Llama-shaped quantised model, one sequence or a batch (Model.begin_decode, decode_step)
  llama_prefill     a prompt through the same model (Model.forward)
  windowed_decode   one decode step of the windowed attention / delta rule design ("Bidonex"), bf16
  windowed_prefill  a prompt through that design
  latent_decode     one decode step of the latent attention / gated delta design ("Tetilorn"), bf16
  latent_prefill    a prompt through that design
  layer             one decoder layer of a decode step by the five fused operators of the C interface, on the caller's buffers
  kquant            activations times a weight kept as K-quant super-blocks (greta_cuda_gemv_kquant)

Every weight, token and cache value comes from the seed.  Models are cut to a few layers of their full width: the layers are alike.
"""
import ctypes
import json
import math
import os
import tempfile

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
ffi = pkg.ffi
DEV = "cuda"
F64 = torch.float64
FMT = {"q4_0": ffi.FMT_Q4_0, "q8_0": ffi.FMT_Q8_0}
BLOCK = {"q4_0": 18, "q8_0": 34}              # bytes of a block of 32 weights
SUPER = {"q4_k": (12, 144), "q6_k": (14, 210)}  # GGML type, bytes of a super-block of 256 weights
WINDOW, KEEP = 1024, 64
LATENT_DIM, LATENT_ROT, LATENT_RANK, LOW = 128, 64, 512, 128
RMS_EPS, HYBRID_EPS = 1e-5, 1e-6
GAP = 2e-3  # of the logits' rms


# ---------------------------------------------------------------------------------------------------------------- the cases
def listed():
    llama7b = dict(dim=4096, heads=32, kv_heads=32, head_dim=128, ffn=11008, vocab=32000, rope=10000.0)
    return [
        # a small model on short prompts (drafting, tests, edge use): launches and latency count
        dict(name="llama_decode_small", kind="llama_decode", fmt="q4_0", layers=2, dim=256, heads=4, kv_heads=2, head_dim=64, ffn=768, vocab=1000,
             rope=10000.0, batch=1, context=12, steps=8),
        # a chat's answer behind a 512-token prompt, one sequence, 7B shape: the headline workload
        dict(name="llama_decode_7b", kind="llama_decode", fmt="q4_0", layers=4, batch=1, context=512, steps=8, **llama7b),
        # a long document behind the answer, 8-bit weights, grouped-query heads
        dict(name="llama_decode_long", kind="llama_decode", fmt="q8_0", layers=2, dim=4096, heads=32, kv_heads=8, head_dim=128, ffn=14336, vocab=32000,
             rope=500000.0, batch=1, context=3001, steps=8),
        # sixteen users at a time on the 70B shape, prompts of up to 4096 tokens
        dict(name="llama_decode_70b_b16", kind="llama_decode", fmt="q4_0", layers=1, dim=8192, heads=64, kv_heads=8, head_dim=128, ffn=28672, vocab=32000,
             rope=500000.0, batch=16, context=4096, steps=4),
        # the 512-token prompt of the headline workload
        dict(name="llama_prefill_7b", kind="llama_prefill", fmt="q4_0", layers=4, tokens=512, **llama7b),
        # a longer prompt of no round length, 8-bit weights, grouped-query heads
        dict(name="llama_prefill_long", kind="llama_prefill", fmt="q8_0", layers=2, dim=4096, heads=32, kv_heads=8, head_dim=128, ffn=14336, vocab=32000,
             rope=500000.0, tokens=1531),
        # the windowed design: a prompt of one portion; eight sequences decoding
        dict(name="windowed_prefill", kind="windowed_prefill", layers=4, width=2048, delta_heads=32, heads=32, kv_heads=8, head_dim=64, ffn=8192, vocab=8192,
             tokens=2048),
        dict(name="windowed_decode_b8", kind="windowed_decode", layers=4, width=2048, delta_heads=32, heads=32, kv_heads=8, head_dim=64, ffn=8192, vocab=8192,
             batch=8, context=2048),
        # the latent design: a prompt of no round length; one sequence decoding
        dict(name="latent_prefill", kind="latent_prefill", layers=4, width=2048, heads=16, q_rank=768, delta_heads=16, ffn=8576, vocab=8192, tokens=1337),
        dict(name="latent_decode", kind="latent_decode", layers=4, width=2048, heads=16, q_rank=768, delta_heads=16, ffn=8576, vocab=8192, batch=1,
             context=2048),
        # a host program that calls the operators itself: one 7B layer over a cache of 2048 positions
        dict(name="layer_7b", kind="layer", fmt="q4_0", dim=4096, heads=32, kv_heads=32, head_dim=128, ffn=11008, rope=10000.0, context=2048),
        # a projection of a K-quant file, multiplied as it lies in the file
        dict(name="kquant_q4_k", kind="kquant", ggml="q4_k", rows=1, n=11008, k=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _llama_shape(rng, lo, hi):
    head_dim = rng.choice((64, 128, 128))
    dim = 256 * max(1, _log(rng, lo, hi) // 256)
    heads = dim // head_dim
    groups = [g for g in (1, 1, 2, 4, 8) if heads % g == 0]
    return dict(fmt=rng.choice(("q4_0", "q4_0", "q8_0")), dim=dim, heads=heads, kv_heads=heads // rng.choice(groups), head_dim=head_dim,
                ffn=32 * int(dim * rng.uniform(2.0, 4.0) / 32), vocab=_log(rng, 1000, 32000), rope=rng.choice((10000.0, 500000.0)))


def _windowed_shape(rng):
    head_dim, kv = rng.choice((64, 64, 128)), rng.choice((2, 4, 8))
    return dict(layers=rng.choice((2, 4)), width=8 * _log(rng, 64, 256), delta_heads=_log(rng, 8, 32), heads=kv * rng.choice((1, 2, 4)), kv_heads=kv,
                head_dim=head_dim, ffn=8 * _log(rng, 128, 1024), vocab=_log(rng, 1000, 8192))


def _latent_shape(rng):
    return dict(layers=rng.choice((2, 4)), width=8 * _log(rng, 64, 256), heads=_log(rng, 4, 16), q_rank=8 * _log(rng, 32, 96), delta_heads=_log(rng, 4, 16),
                ffn=8 * _log(rng, 128, 1072), vocab=_log(rng, 1000, 8192))


def draw(rng):
    kind = rng.choice(("llama_decode", "llama_decode", "llama_decode", "llama_prefill", "llama_prefill", "windowed_prefill", "windowed_decode",
                       "latent_prefill", "latent_decode", "layer", "kquant"))
    if kind == "llama_decode":
        if rng.random() < 0.5:  # one sequence
            return dict(kind=kind, layers=rng.choice((1, 2)), batch=1, context=_log(rng, 12, 4096), steps=8, **_llama_shape(rng, 256, 4096))
        batch = _log(rng, 2, 32)
        return dict(kind=kind, layers=1, batch=batch, context=_log(rng, 12, min(4096, 32768 // batch)), steps=4, **_llama_shape(rng, 512, 8192))
    if kind == "llama_prefill":
        return dict(kind=kind, layers=2, tokens=_log(rng, 8, 2048), **_llama_shape(rng, 512, 4096))
    if kind == "windowed_prefill":
        return dict(kind=kind, tokens=_log(rng, 16, 2048), **_windowed_shape(rng))
    if kind == "windowed_decode":
        return dict(kind=kind, batch=_log(rng, 1, 16), context=_log(rng, 16, 2048), **_windowed_shape(rng))
    if kind == "latent_prefill":
        return dict(kind=kind, tokens=_log(rng, 16, 2048), **_latent_shape(rng))
    if kind == "latent_decode":
        return dict(kind=kind, batch=_log(rng, 1, 16), context=_log(rng, 16, 2048), **_latent_shape(rng))
    if kind == "layer":
        c = dict(kind=kind, context=_log(rng, 12, 4096), **_llama_shape(rng, 1024, 4096))
        del c["vocab"]
        return c
    return dict(kind=kind, ggml=rng.choice(("q4_k", "q6_k")), rows=rng.choice((1, 1, 2, 8)), n=_log(rng, 1024, 28672), k=256 * _log(rng, 4, 32))


# ------------------------------------------------------------------------------------------------------------ random weights
def _gen(seed, stream=0):
    g = torch.Generator(DEV)
    g.manual_seed((int(seed) * 1000003 + stream) & 0x7FFFFFFFFFFF)
    return g


def _normal(g, *shape, sigma=1.0, mean=0.0):
    return torch.randn(*shape, generator=g, device=DEV) * sigma + mean


def _blocks(g, fmt, n, k):
    """GGUF blocks of an [n x k] weight: uniform quants, scale |N(0, 0.02)| / 8 (4 bits) or / 127 (8 bits), in fp16."""
    nb = n * (k // 32)
    out = torch.randint(0, 256, (nb, BLOCK[fmt]), generator=g, device=DEV, dtype=torch.uint8)
    if fmt == "q8_0":
        out[:, 2:][out[:, 2:] == 128] = 0  # -128 is never written
    out[:, :2] = (_normal(g, nb, sigma=0.02).abs() / (8 if fmt == "q4_0" else 127)).half().view(torch.uint8).reshape(nb, 2)
    return out


def _values(fmt, blocks, n, k):
    """The weights those blocks stand for, in float64."""
    d = blocks[:, :2].contiguous().view(torch.float16).to(F64)
    if fmt == "q8_0":
        q = blocks[:, 2:].contiguous().view(torch.int8).to(F64)
    else:
        q = torch.cat([blocks[:, 2:] & 15, blocks[:, 2:] >> 4], 1).to(F64) - 8
    return (q * d).reshape(n, k)


def _super_blocks(g, ggml, n, k):
    ns = n * (k // 256)
    out = torch.randint(0, 256, (ns, SUPER[ggml][1]), generator=g, device=DEV, dtype=torch.uint8)
    scale = _normal(g, ns, sigma=0.02).abs()
    if ggml == "q4_k":
        out[:, 0:2] = (scale / 256).half().view(torch.uint8).reshape(ns, 2)
        out[:, 2:4] = (scale / 32).half().view(torch.uint8).reshape(ns, 2)
    else:
        out[:, 208:210] = (scale / 2048).half().view(torch.uint8).reshape(ns, 2)
    return out


def _super_values(ggml, b, n, k):
    if ggml == "q4_k":
        d, dmin = (b[:, i:i + 2].contiguous().view(torch.float16).to(F64) for i in (0, 2))
        sc = b[:, 4:16].to(torch.int64)
        s, m = [sc[:, j] & 63 for j in range(4)], [sc[:, 6 + j] & 63 for j in range(4)]
        for j in range(4):
            shift = 4 * (j & 1)
            s.append((sc[:, j] >> 6) | (((sc[:, 4 + j // 2] >> shift) & 15) << 2))
            m.append((sc[:, 6 + j] >> 6) | (((sc[:, 10 + j // 2] >> shift) & 15) << 2))
        q = b[:, 16:]
        q = torch.stack([q & 15, q >> 4], 2).reshape(-1, 8, 32).to(F64)
        w = (d * torch.stack(s, 1))[:, :, None] * q - (dmin * torch.stack(m, 1))[:, :, None]
    else:
        low = torch.stack([b[:, :128] & 15, b[:, :128] >> 4], 2).reshape(-1, 256)
        high = torch.stack([(b[:, 128:192] >> (2 * i)) & 3 for i in range(4)], 2).reshape(-1, 256)
        q = (low | (high << 4)).to(F64) - 32
        sc = b[:, 192:208].contiguous().view(torch.int8).to(F64).repeat_interleave(16, 1)
        w = b[:, 208:210].contiguous().view(torch.float16).to(F64) * q * sc
    return w.reshape(n, k)


# ------------------------------------------------------------------------------------------------- Llama-shaped quantised models
def _llama_matrices(c):
    q, kv = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    return {"wq": (q, c["dim"]), "wk": (kv, c["dim"]), "wv": (kv, c["dim"]), "wo": (c["dim"], q), "w1": (c["ffn"], c["dim"]), "w2": (c["dim"], c["ffn"]),
            "w3": (c["ffn"], c["dim"])}


def _llama_weights(c, seed):
    layers = []
    for l in range(c["layers"]):
        g = _gen(seed, 10 + l)
        w = {n: _blocks(g, c["fmt"], *s) for n, s in _llama_matrices(c).items()}
        w["attn_norm"], w["ffn_norm"] = _normal(g, c["dim"], sigma=0.1, mean=1.0), _normal(g, c["dim"], sigma=0.1, mean=1.0)
        layers.append(w)
    g = _gen(seed, 1)
    return {"layers": layers, "tok_embd": _normal(g, c["vocab"], c["dim"], sigma=0.02).half(), "out_norm": _normal(g, c["dim"], sigma=0.1, mean=1.0),
            "out_weight": _normal(g, c["vocab"], c["dim"], sigma=0.02).half()}


def _llama_model(c, seed, positions, batch=1):
    w = _llama_weights(c, seed)
    cfg = dict(dim=c["dim"], num_heads=c["heads"], num_heads_kv=c["kv_heads"], num_layers=c["layers"], vocab=c["vocab"], hidden_dim=c["ffn"],
               head_dim=c["head_dim"], max_seq=positions, rope_base=c["rope"], rms_eps=RMS_EPS)
    m = pkg.model.Model(cfg, weight_fmt=FMT[c["fmt"]], batch=batch)
    host = {n: (t.view(torch.int16) if t.dtype == torch.float16 else t).cpu().numpy() for n, t in w.items() if n != "layers"}
    m.load({"layers": [{n: t.reshape(-1).cpu().numpy() for n, t in lw.items()} for lw in w["layers"]], **host})
    return m


def _prompts(c, seed):
    """Token ids per sequence.  A batch's prompts have lengths of their own, from half of `context` up to it."""
    rng = np.random.default_rng([int(seed), 7])
    n = [c["context"]] if c["batch"] == 1 else [int(v) for v in rng.integers((c["context"] + 1) // 2, c["context"] + 1, c["batch"])]
    return [rng.integers(0, c["vocab"], k).astype(np.int32) for k in n], rng.integers(0, c["vocab"], c["batch"]).astype(np.int32)


def _prefilled(m, c, prompts):
    for b, p in enumerate(prompts):
        if c["batch"] > 1:
            m.set_sequence(b)
        m.forward(p, 0)


def _logits(m, n):
    out = np.empty(n, np.float32)
    if m.h.greta_model_get_logits(m.handle, out.ctypes.data, out.size) != 0:
        raise RuntimeError("greta_model_get_logits failed")
    return out


def _rms(x, w, eps=RMS_EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rope(x, pos, base):
    """x [T, heads, d], halves turned together."""
    h = x.shape[-1] // 2
    a = pos.to(F64)[:, None] * base ** (-2.0 * torch.arange(h, device=DEV, dtype=F64) / x.shape[-1])
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    return torch.cat([x[..., :h] * c - x[..., h:] * s, x[..., :h] * s + x[..., h:] * c], -1)


def _causal(q, k, v, scale, first):
    """q [T, H, d] at positions first .., k, v [S, G, d]."""
    T, H, S, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    out = torch.empty_like(q)
    hidden = torch.arange(S, device=DEV)[None] > first + torch.arange(T, device=DEV)[:, None]
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T * scale).masked_fill_(hidden, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h // (H // G)]
    return out


class _Llama64:
    """The Llama-shaped model in float64; one sequence at a time."""

    def __init__(self, c, seed):
        w = _llama_weights(c, seed)
        shapes = _llama_matrices(c)
        self.c = c
        self.layers = [{n: _values(c["fmt"], t, *shapes[n]) if n in shapes else t.to(F64) for n, t in lw.items()} for lw in w["layers"]]
        self.embd, self.norm, self.head = w["tok_embd"], w["out_norm"].to(F64), w["out_weight"].to(F64)

    def run(self, tokens, cache, last_only):
        """Logits of the last token; `cache` (a list of (k, v) per layer, or None) grows.  last_only None: only the cache is wanted."""
        c, pos0 = self.c, cache[0][0].shape[0] if cache else 0
        x = self.embd[torch.as_tensor(tokens, device=DEV).long()].to(F64)
        pos = pos0 + torch.arange(len(tokens), device=DEV)
        grown = []
        for l, w in enumerate(self.layers):
            h = _rms(x, w["attn_norm"])
            k = _rope((h @ w["wk"].T).view(-1, c["kv_heads"], c["head_dim"]), pos, c["rope"])
            v = (h @ w["wv"].T).view(-1, c["kv_heads"], c["head_dim"])
            if cache:
                k, v = torch.cat([cache[l][0], k]), torch.cat([cache[l][1], v])
            grown.append((k, v))
            if l + 1 == len(self.layers):
                if last_only is None:
                    return None, grown
                h, x, pos = h[-1:], x[-1:], pos[-1:]
            q = _rope((h @ w["wq"].T).view(-1, c["heads"], c["head_dim"]), pos, c["rope"])
            x = x + _causal(q, k, v, c["head_dim"] ** -0.5, int(pos[0])).reshape(len(x), -1) @ w["wo"].T
            h = _rms(x, w["ffn_norm"])
            x = x + (torch.nn.functional.silu(h @ w["w1"].T) * (h @ w["w3"].T)) @ w["w2"].T
        return _rms(x[-1], self.norm) @ self.head.T, grown

    def decode(self, prompt, first, steps):
        """Logits of the last step, and the smallest gap between the two best ids on the way there (in units of the logits' rms)."""
        _, cache = self.run(prompt, None, None)
        token, gap = int(first), math.inf
        for i in range(steps):
            z, cache = self.run([token], cache, True)
            if i + 1 < steps:
                top = torch.topk(z, 2).values
                gap = min(gap, float((top[0] - top[1]) / z.square().mean().sqrt()))
                token = int(z.argmax())
        return z, gap


class LlamaDecode:
    @staticmethod
    def prepare(c, seed):
        m = _llama_model(c, seed, c["context"] + c["steps"], c["batch"])
        prompts, first = _prompts(c, seed)
        _prefilled(m, c, prompts)
        if c["batch"] == 1:
            return m, int(first[0]), len(prompts[0])
        return m, first, np.array([len(p) for p in prompts], np.uint32)

    @staticmethod
    def run(c, s):
        m, first, pos = s
        m.begin_decode(first, pos)
        for _ in range(c["steps"]):
            m.decode_step()
        return {"ids": np.asarray(m.read_generated(c["steps"]), np.int32), "logits": _logits(m, c["batch"] * c["vocab"])}

    @staticmethod
    def exact(c, seed):
        m = _Llama64(c, seed)
        got = [m.decode(p, t, c["steps"]) for p, t in zip(*_prompts(c, seed))]
        # The cache is fp16 and the prompt went through fp16 products, so the greedy path is certain only where no two ids came that close.
        return {"ids": None, "logits": torch.cat([z for z, _ in got])} if min(g for _, g in got) > GAP else None

    @staticmethod
    def work(c):
        prompts, _ = _prompts(c, 0)
        rows = c["steps"] * c["batch"]
        weights = sum(n * k for n, k in _llama_matrices(c).values()) * c["layers"]
        passes = c["steps"] if weights + 2 * c["vocab"] * c["dim"] > 100e6 else 1  # what fits the caches need not be read again
        heads = c["head_dim"] * sum(len(p) for p in prompts) * c["layers"]
        return {"bytes": passes * (weights * BLOCK[c["fmt"]] / 32 + 2 * c["vocab"] * c["dim"] + 4 * c["kv_heads"] * heads) + 4 * c["batch"] * c["vocab"],
                "flops": 2 * rows * (weights + c["vocab"] * c["dim"]) + 4 * c["steps"] * c["heads"] * heads}

    @staticmethod
    def tolerance(c):
        return {"rel": 2e-3, "max": 2e-2, "differ": 0.01}


class LlamaPrefill:
    @staticmethod
    def prepare(c, seed):
        tokens = np.random.default_rng([int(seed), 7]).integers(0, c["vocab"], c["tokens"]).astype(np.int32)
        return _llama_model(c, seed, c["tokens"]), tokens

    @staticmethod
    def run(c, s):
        return s[0].forward(s[1], 0)

    @staticmethod
    def exact(c, seed):
        tokens = np.random.default_rng([int(seed), 7]).integers(0, c["vocab"], c["tokens"])
        return _Llama64(c, seed).run(tokens, None, True)[0]

    @staticmethod
    def work(c):
        T = c["tokens"]
        weights = sum(n * k for n, k in _llama_matrices(c).values()) * c["layers"]
        return {"bytes": weights * BLOCK[c["fmt"]] / 32 + 2 * c["vocab"] * c["dim"] + 4 * c["layers"] * T * c["kv_heads"] * c["head_dim"] + 4 * c["vocab"],
                "flops": 2 * T * weights + 2 * c["vocab"] * c["dim"] + 2 * c["layers"] * T * (T + 1) * c["heads"] * c["head_dim"]}

    @staticmethod
    def tolerance(c):
        return {"rel": 4e-3, "max": 4e-2}


# ------------------------------------------------------------------------------------------------------ the two bf16 designs
def _ff(c):
    return {"kind": "dense", "ff": c["ffn"]}


def _windowed_config(c, positions):
    attention = {"type": "attention", "mlp": _ff(c),
                 "mixer": {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": c["head_dim"], "vdim": c["head_dim"], "conv": 4,
                           "scale": c["head_dim"] ** -0.5, "softcap": 30.0, "mask": {"size": WINDOW, "keep_first": KEEP}}}
    delta = {"type": "general_delta", "mlp": _ff(c), "mixer": {"heads": c["delta_heads"], "dim": 64, "rank": 64}}
    return {"architecture": "Bidonex", "width": c["width"], "vocab": c["vocab"], "max_positions": positions, "norm": {"eps": HYBRID_EPS},
            "layers": [delta if i % 2 == 0 else attention for i in range(c["layers"])]}


def _latent_config(c):
    mix = {"heads": c["heads"], "dim": LATENT_DIM, "rot_dim": LATENT_ROT, "vdim": LATENT_DIM, "kv_rank": LATENT_RANK, "scale": (LATENT_DIM + LATENT_ROT) ** -0.5}
    yarn = {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    first = {"type": "latent_attention", "mlp": _ff(c), "mixer": dict(mix, q_rank=c["q_rank"], rot={"base": 10000.0, "dims": LATENT_ROT, "scaling": yarn})}
    second = {"type": "latent_attention_2", "mlp": _ff(c), "mixer": dict(mix, rot={"base": 10000.0, "dims": LATENT_ROT})}
    delta = {"type": "channel_delta", "mlp": _ff(c), "mixer": {"heads": c["delta_heads"], "kv_heads": c["delta_heads"], "dim": 128, "vdim": 128, "conv": 4,
                                                               "decay_rank": LOW, "gate_rank": LOW}}
    return {"architecture": "Tetilorn", "width": c["width"], "vocab": c["vocab"], "embedding": {"scale": 1.0}, "norm": {"eps": HYBRID_EPS},
            "layers": [(delta, first, delta, second)[i % 4] for i in range(c["layers"])]}


def _hybrid_weights(cfg, seed):
    """Tensors as a model folder holds them (values of bf16), matrices scaled by their fan-in."""
    g = _gen(seed, 3)
    D, V = cfg["width"], cfg["vocab"]
    windowed = cfg["architecture"] == "Bidonex"
    w = {}

    def mat(name, rows, cols, gain=1.0):
        w[name] = _normal(g, rows, cols, sigma=gain / math.sqrt(cols))

    def vec(name, *shape, sigma, mean=0.0):
        w[name] = _normal(g, *shape, sigma=sigma, mean=mean)

    def norm(name, n):
        vec(name, n, sigma=0.2, mean=1.0)
        if windowed:
            vec(name + ".b", n, sigma=0.1)

    mat("embed", V, D, gain=math.sqrt(D))
    if windowed:
        mat("pos", cfg["max_positions"], D, gain=0.5 * math.sqrt(D))
        mat("head", V, D)
    norm("final.norm", D)
    for i, l in enumerate(cfg["layers"]):
        m, p = l["mixer"], f"l{i}.mix."
        H, d = m["heads"], m["dim"]
        norm(f"l{i}.norm1", D)
        if l["type"] == "attention":
            for n, rows in (("q", H * d), ("k", m["kv_heads"] * d), ("v", m["kv_heads"] * m["vdim"])):
                mat(p + n, rows, D)
                vec(p + n + ".conv", rows, m["conv"], sigma=0.5)
            for n, lo in (("temp", 0.5), ("r1", 0.2), ("r2", 0.05)):
                w[p + n] = lo + torch.rand(H, generator=g, device=DEV)
            vec(p + "sink", H, sigma=1.0)
            mat(p + "o", D, H * m["vdim"])
        elif l["type"] == "general_delta":
            for n in "rkvga":
                mat(p + n, H * d, D)
            vec(p + "a.b", H * d, sigma=0.5)
            mat(p + "w1", m["rank"], D)
            mat(p + "w2", H * d, m["rank"], gain=2.0)
            vec(p + "w0", H * d, sigma=1.5, mean=-2.0)
            vec(p + "norm", H * d, sigma=0.2, mean=1.0)
            mat(p + "o", D, H * d)
        elif l["type"] == "channel_delta":
            for n, rows in (("q", H * d), ("k", H * d), ("v", H * m["vdim"])):
                mat(p + n, rows, D)
                vec(p + n + ".conv", rows, m["conv"], sigma=0.5)
            mat(p + "b", H, D)
            mat(p + "a1", m["decay_rank"], D)
            mat(p + "a2", H * d, m["decay_rank"])
            vec(p + "A_log", H, sigma=1.0, mean=-1.0)
            vec(p + "dt_bias", H * d, sigma=1.0, mean=-2.0)
            mat(p + "g1", m["gate_rank"], D)
            mat(p + "g2", H * m["vdim"], m["gate_rank"])
            norm(p + "norm", m["vdim"])
            mat(p + "o", D, H * m["vdim"])
        else:
            rows = H * (d + m["rot_dim"])
            if "q_rank" in m:
                mat(p + "dq", m["q_rank"], D)
                norm(p + "dq.norm", m["q_rank"])
                mat(p + "uq", rows, m["q_rank"])
                vec(p + "sink", H, sigma=1.0)
                mat(p + "g", H * m["vdim"], D)
            else:
                mat(p + "q", rows, D)
            mat(p + "dkv", m["kv_rank"] + m["rot_dim"], D)
            norm(p + "dkv.norm", m["kv_rank"])
            mat(p + "uk", H * d, m["kv_rank"])
            mat(p + "uv", H * m["vdim"], m["kv_rank"])
            mat(p + "o", D, H * m["vdim"])
        if not windowed:
            norm(f"l{i}.norm2", D)
        mat(f"l{i}.mlp.up", l["mlp"]["ff"], D)
        mat(f"l{i}.mlp.down", D, l["mlp"]["ff"])
    return {n: t.to(torch.bfloat16) for n, t in w.items()}


def _config_of(c, positions):
    return _windowed_config(c, positions) if c["kind"].startswith("windowed") else _latent_config(c)


def _hybrid_model(c, seed, positions, batch=1):
    cfg = _config_of(c, positions)
    with tempfile.TemporaryDirectory(dir="/dev/shm" if os.path.isdir("/dev/shm") else None) as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(cfg, f)
        bits = {n: t.view(torch.int16).cpu().numpy().view(np.uint16) for n, t in _hybrid_weights(cfg, seed).items()}
        pkg.model.write_safetensors(os.path.join(folder, "model.safetensors"), bits)
        return pkg.model.Model.open(folder, batch=batch, max_seq=positions)


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _rms_plain(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _conv(u, w):
    """y[t, c] = sum_j w[c, j] u[t - taps + 1 + j, c]."""
    taps = w.shape[1]
    padded = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return sum(w[:, j] * padded[j:j + len(u)] for j in range(taps))


def _windowed64(h, w, p, m):
    T, H, G, d, eps = len(h), m["heads"], m["kv_heads"], m["dim"], HYBRID_EPS
    q, k, v = (_conv(h @ w[p + n].T, w[p + n + ".conv"]) for n in "qkv")
    q, k, v = _rms_plain(q.view(T, H, d), eps), _rms_plain(k.view(T, G, d), eps), v.view(T, G, m["vdim"])
    far = (torch.arange(T, device=DEV)[:, None] - torch.arange(T, device=DEV)[None]).to(F64)
    hidden = (far < 0) | ((far >= m["mask"]["size"]) & (torch.arange(T, device=DEV) >= m["mask"]["keep_first"])[None])
    out = []
    for i in range(H):
        s = q[:, i] @ k[:, i // (H // G)].T * (m["scale"] * w[p + "temp"][i])
        s = m["softcap"] * torch.tanh(s / m["softcap"]) - w[p + "r1"][i] * torch.log1p(w[p + "r2"][i] * far.clamp(min=0))
        s = torch.cat([s.masked_fill(hidden, -math.inf), w[p + "sink"][i].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[:, i // (H // G)])
    return torch.stack(out, 1).reshape(T, -1) @ w[p + "o"].T


def _general_delta64(h, w, p, m):
    T, H, d = len(h), m["heads"], m["dim"]
    r, k, v = ((h @ w[p + n].T).view(T, H, d) for n in "rkv")
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w[p + "w1"].T) @ w[p + "w2"].T + w[p + "w0"])).view(T, H, d)
    a = torch.sigmoid(h @ w[p + "a"].T + w[p + "a.b"]).view(T, H, d)
    u = _unit(k)
    au, S, o = a * u, h.new_zeros(H, d, d), []
    for t in range(T):
        S = decay[t][:, :, None] * S - au[t][:, :, None] * (u[t][:, None] @ S) + k[t][:, :, None] * v[t][:, None]
        o.append((r[t][:, None] @ S)[:, 0])
    o = _rms_plain(torch.stack(o), HYBRID_EPS).reshape(T, -1) * w[p + "norm"]
    return (o * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def _channel_delta64(h, w, p, m):
    T, H, d, vd = len(h), m["heads"], m["dim"], m["vdim"]
    q, k, v = (torch.nn.functional.silu(_conv(h @ w[p + n].T, w[p + n + ".conv"])) for n in "qkv")
    q, k, v = _unit(q.view(T, H, d)) * d ** -0.5, _unit(k.view(T, H, d)), v.view(T, H, vd)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    z = (h @ w[p + "a1"].T @ w[p + "a2"].T).view(T, H, d) + w[p + "dt_bias"].view(H, d)
    decay = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * torch.nn.functional.softplus(z, threshold=700.0))
    S, o = h.new_zeros(H, d, vd), []
    for t in range(T):
        S = decay[t][:, :, None] * S
        S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0]))[:, None]
        o.append((q[t][:, None] @ S)[:, 0])
    o = (_rms_plain(torch.stack(o), HYBRID_EPS) * w[p + "norm"]).reshape(T, -1)
    return (o * torch.sigmoid(h @ w[p + "g1"].T @ w[p + "g2"].T)) @ w[p + "o"].T


def _turned(x, rot, halves):
    """x [T, n, dims] turned by its positions, neighbours or halves apart."""
    dims, base, y = rot["dims"], rot["base"], rot.get("scaling")
    i = torch.arange(dims // 2, device=DEV, dtype=F64)
    f, amp = base ** (-2.0 * i / dims), 1.0
    if y:
        lo, hi = (dims * math.log(y["original"] / (2 * math.pi * y[n])) / (2 * math.log(base)) for n in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, amp = f / y["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(y["factor"]) + 1
    a = torch.arange(len(x), device=DEV, dtype=F64)[:, None] * f
    c, s = (torch.cos(a) * amp)[:, None], (torch.sin(a) * amp)[:, None]
    u, v = (x[..., :dims // 2], x[..., dims // 2:]) if halves else (x[..., 0::2], x[..., 1::2])
    u, v = u * c - v * s, v * c + u * s
    return torch.cat([u, v], -1) if halves else torch.stack([u, v], -1).reshape(x.shape)


def _latent64(h, w, p, m):
    T, H, d, r, vd, R = len(h), m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    first = "q_rank" in m
    q = _rms(h @ w[p + "dq"].T, w[p + "dq.norm"], HYBRID_EPS) @ w[p + "uq"].T if first else h @ w[p + "q"].T
    q = q.view(T, H, d + r)
    down = h @ w[p + "dkv"].T
    lat = _rms(down[:, :R], w[p + "dkv.norm"], HYBRID_EPS)
    qr, kr = _turned(q[..., d:], m["rot"], first), _turned(down[:, None, R:], m["rot"], first)[:, 0]
    k, v = (lat @ w[p + "uk"].T).view(T, H, d), (lat @ w[p + "uv"].T).view(T, H, vd)
    hidden = torch.arange(T, device=DEV)[None] > torch.arange(T, device=DEV)[:, None]
    out = []
    for i in range(H):
        s = ((q[:, i, :d] @ k[:, i].T + qr[:, i] @ kr.T) * m["scale"]).masked_fill_(hidden, -math.inf)
        if first:
            s = torch.cat([s, w[p + "sink"][i].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[:, i])
    o = torch.stack(out, 1).reshape(T, -1)
    if first:
        o = o * torch.sigmoid(h @ w[p + "g"].T)
    return o @ w[p + "o"].T


_MIXERS64 = {"attention": _windowed64, "general_delta": _general_delta64, "channel_delta": _channel_delta64, "latent_attention": _latent64,
             "latent_attention_2": _latent64}


def _hybrid64(cfg, w, tokens):
    """Logits of the last position, in float64."""
    windowed = cfg["architecture"] == "Bidonex"

    def norm(x, name):
        if not windowed:
            return _rms(x, w[name], HYBRID_EPS)
        x = x - x.mean(-1, keepdim=True)
        return _rms(x, w[name], HYBRID_EPS) + w[name + ".b"]

    x = w["embed"][torch.as_tensor(tokens, device=DEV).long()] * (1.0 if windowed else cfg["embedding"]["scale"])
    if windowed:
        x = x + w["pos"][:len(tokens)]
    for i, l in enumerate(cfg["layers"]):
        h = norm(x, f"l{i}.norm1")
        y = _MIXERS64[l["type"]](h, w, f"l{i}.mix.", l["mixer"])
        if windowed:
            x = x + y + torch.nn.functional.gelu(h @ w[f"l{i}.mlp.up"].T) @ w[f"l{i}.mlp.down"].T
        else:
            x = x + y
            x = x + torch.relu(norm(x, f"l{i}.norm2") @ w[f"l{i}.mlp.up"].T) ** 2 @ w[f"l{i}.mlp.down"].T
    return norm(x[-1:], "final.norm")[0] @ w["head" if windowed else "embed"].T


def _hybrid_work(c, rows, past, prompt):
    """rows tokens in all; past: keys that attention reads per decode step (0: a prompt, whose rows see one another)."""
    D, L = c["width"], c["layers"]
    if c["kind"].startswith("windowed"):
        H, d, Hd = c["heads"], c["head_dim"], c["delta_heads"] * 64
        attn = D * d * (H + 2 * c["kv_heads"]) + D * H * d
        delta = D * (5 * Hd + 64) + Hd * 64 + D * Hd
        key, seen, state = 4 * c["kv_heads"] * d, WINDOW + KEEP, 64 * Hd
        pairs, per_pair = sum(min(t + 1, seen) for t in range(rows)) if prompt else past, 4 * H * d
        weights = L // 2 * (attn + delta) + L * 2 * D * c["ffn"]
        attention_layers = L // 2
    else:
        H, Hd = c["heads"], c["delta_heads"] * 128
        up = LATENT_RANK * H * 2 * LATENT_DIM
        first = D * (c["q_rank"] + LATENT_RANK + LATENT_ROT + H * LATENT_DIM) + c["q_rank"] * H * (LATENT_DIM + LATENT_ROT) + up + D * H * LATENT_DIM
        second = D * (H * (LATENT_DIM + LATENT_ROT) + LATENT_RANK + LATENT_ROT) + up + D * H * LATENT_DIM
        delta = D * (3 * Hd + c["delta_heads"] + 2 * LOW) + 2 * LOW * Hd + D * Hd
        key, state = 2 * (LATENT_RANK + LATENT_ROT), 128 * Hd
        pairs = rows * (rows + 1) // 2 if prompt else past
        per_pair = 2 * H * (2 * LATENT_DIM + LATENT_ROT if prompt else 2 * LATENT_RANK + LATENT_ROT)
        weights = L // 2 * delta + sum((first, second)[i // 2 % 2] for i in range(1, L, 2)) + L * 2 * D * c["ffn"]
        attention_layers = L // 2
    head = D * c["vocab"]
    sequences = 1 if prompt else rows
    return {"bytes": 2 * (weights + head) + attention_layers * key * (rows if prompt else past) + (L - attention_layers) * 4 * state * sequences * (1 if prompt else 2) +
            4 * c["vocab"] * sequences,
            "flops": 2 * rows * weights + 2 * sequences * head + attention_layers * per_pair * pairs + (L - attention_layers) * 8 * state * rows}


class HybridPrefill:
    @staticmethod
    def _tokens(c, seed):
        return np.random.default_rng([int(seed), 7]).integers(0, c["vocab"], c["tokens"]).astype(np.int32)

    @staticmethod
    def prepare(c, seed):
        return _hybrid_model(c, seed, c["tokens"]), HybridPrefill._tokens(c, seed)

    @staticmethod
    def run(c, s):
        return s[0].forward(s[1], 0)

    @staticmethod
    def exact(c, seed):
        cfg = _config_of(c, c["tokens"])
        return _hybrid64(cfg, {n: t.to(F64) for n, t in _hybrid_weights(cfg, seed).items()}, HybridPrefill._tokens(c, seed))

    @staticmethod
    def work(c):
        return _hybrid_work(c, c["tokens"], 0, True)

    @staticmethod
    def tolerance(c):
        return {"rel": 0.015, "max": 0.15}


class HybridDecode:
    @staticmethod
    def prepare(c, seed):
        m = _hybrid_model(c, seed, c["context"] + 1, c["batch"])
        prompts, first = _prompts(c, seed)
        _prefilled(m, c, prompts)
        if c["batch"] == 1:
            return m, int(first[0]), len(prompts[0])
        return m, first, np.array([len(p) for p in prompts], np.uint32)

    @staticmethod
    def run(c, s):
        m, first, pos = s
        m.begin_decode(first, pos)
        m.decode_step()
        m.read_generated(1)  # waits for the step; the ids are the logits' maxima, which bf16 leaves open between close ones
        return _logits(m, c["batch"] * c["vocab"])

    @staticmethod
    def exact(c, seed):
        cfg = _config_of(c, c["context"] + 1)
        w = {n: t.to(F64) for n, t in _hybrid_weights(cfg, seed).items()}
        return torch.cat([_hybrid64(cfg, w, np.append(p, t)) for p, t in zip(*_prompts(c, seed))])

    @staticmethod
    def work(c):
        prompts, _ = _prompts(c, 0)
        seen = WINDOW + KEEP if c["kind"].startswith("windowed") else 1 << 30
        return _hybrid_work(c, c["batch"], sum(min(len(p) + 1, seen) for p in prompts), False)

    @staticmethod
    def tolerance(c):
        return {"rel": 0.015, "max": 0.15}


# ------------------------------------------------------------------------------------------- the operators of the C interface
def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ok(rc, what):
    ffi.check(rc, what)


def _planes(fmt, blocks, n, k):
    """The two device planes the operators read."""
    lib = ffi.cuda()
    qs = torch.empty(lib.greta_cuda_qs_bytes(FMT[fmt], n, k), dtype=torch.uint8, device=DEV)
    d = torch.empty(lib.greta_cuda_d_bytes(FMT[fmt], n, k), dtype=torch.uint8, device=DEV)
    _ok(lib.greta_cuda_repack_gguf(_stream(), FMT[fmt], blocks.data_ptr(), qs.data_ptr(), d.data_ptr(), n, k), "repack_gguf")
    return qs, d


class Layer:
    @staticmethod
    def _inputs(c, seed):
        """The layer's raw weights, the residual stream, and a cache filled in front of position `context`."""
        g = _gen(seed, 5)
        w = {n: _blocks(g, c["fmt"], *s) for n, s in _llama_matrices(c).items()}
        w["attn_norm"], w["ffn_norm"] = _normal(g, c["dim"], sigma=0.1, mean=1.0), _normal(g, c["dim"], sigma=0.1, mean=1.0)
        cache = [_normal(g, c["kv_heads"], c["context"] + 1, c["head_dim"]).half() for _ in range(2)]
        return w, _normal(g, c["dim"]), cache

    @staticmethod
    def prepare(c, seed):
        w, x, (k, v) = Layer._inputs(c, seed)
        shapes = _llama_matrices(c)
        s = {n: _planes(c["fmt"], t, *shapes[n]) if n in shapes else t for n, t in w.items()}
        s.update(x=x, k=k, v=v, pos=torch.tensor([c["context"]], dtype=torch.int32, device=DEV))
        for n, size in (("q", c["heads"] * c["head_dim"]), ("att", c["heads"] * c["head_dim"]), ("mid", c["dim"]), ("gate", c["ffn"]), ("y", c["dim"])):
            s[n] = torch.empty(size, device=DEV)
        s["scratch"] = torch.zeros(ffi.cuda().greta_cuda_attn_decode_scratch_bytes(c["heads"], c["head_dim"]), dtype=torch.uint8, device=DEV)
        return s

    @staticmethod
    def run(c, s):
        lib, st, fmt = ffi.cuda(), _stream(), FMT[c["fmt"]]
        at = {n: t.data_ptr() if isinstance(t, torch.Tensor) else tuple(p.data_ptr() for p in t) for n, t in s.items()}
        D, H, G, d, F, S = c["dim"], c["heads"], c["kv_heads"], c["head_dim"], c["ffn"], c["context"] + 1
        _ok(lib.greta_cuda_fused_rmsnorm_qkv_rope_kv(st, fmt, at["x"], at["attn_norm"], RMS_EPS, *at["wq"], *at["wk"], *at["wv"], at["q"], None, None, at["k"],
                                                     at["v"], at["pos"], H, G, d, S, c["rope"], D), "qkv")
        _ok(lib.greta_cuda_attn_decode(st, at["q"], at["k"], at["v"], at["att"], at["pos"], 0, H, G, d, S, d ** -0.5, at["scratch"], s["scratch"].numel()), "attn")
        _ok(lib.greta_cuda_gemv_residual(st, fmt, at["att"], *at["wo"], at["x"], at["mid"], D, H * d), "wo")
        _ok(lib.greta_cuda_fused_ffn_front(st, fmt, at["mid"], at["ffn_norm"], RMS_EPS, *at["w1"], *at["w3"], at["gate"], D, F), "ffn_front")
        _ok(lib.greta_cuda_gemv_residual(st, fmt, at["gate"], *at["w2"], at["mid"], at["y"], D, F), "w2")
        return {"y": s["y"], "k_row": s["k"][:, c["context"]], "v_row": s["v"][:, c["context"]]}  # the cache rows that the step adds

    @staticmethod
    def exact(c, seed):
        w, x, (kc, vc) = Layer._inputs(c, seed)
        shapes = _llama_matrices(c)
        w = {n: _values(c["fmt"], t, *shapes[n]) if n in shapes else t.to(F64) for n, t in w.items()}
        x, pos = x.to(F64)[None], torch.tensor([c["context"]], device=DEV)
        h = _rms(x, w["attn_norm"])
        q, k = (_rope((h @ w[n].T).view(1, -1, c["head_dim"]), pos, c["rope"]) for n in ("wq", "wk"))
        v = (h @ w["wv"].T).view(1, -1, c["head_dim"])
        keys, values = (torch.cat([t[:, :-1].transpose(0, 1).to(F64), n]) for t, n in ((kc, k), (vc, v)))
        x = x + _causal(q, keys, values, c["head_dim"] ** -0.5, c["context"]).reshape(1, -1) @ w["wo"].T
        h = _rms(x, w["ffn_norm"])
        y = x + (torch.nn.functional.silu(h @ w["w1"].T) * (h @ w["w3"].T)) @ w["w2"].T
        return {"y": y[0], "k_row": k[0], "v_row": v[0]}

    @staticmethod
    def work(c):
        weights = sum(n * k for n, k in _llama_matrices(c).values())
        return {"bytes": weights * BLOCK[c["fmt"]] / 32 + 4 * (c["context"] + 1) * c["kv_heads"] * c["head_dim"] + 16 * c["dim"],
                "flops": 2 * weights + 4 * (c["context"] + 1) * c["heads"] * c["head_dim"]}

    @staticmethod
    def tolerance(c):
        return {"rel": 1e-3, "max": 1e-2}  # the cache rows are fp16


class KQuant:
    @staticmethod
    def _inputs(c, seed):
        g = _gen(seed, 6)
        return _super_blocks(g, c["ggml"], c["n"], c["k"]), _normal(g, c["rows"], c["k"])

    @staticmethod
    def prepare(c, seed):
        w, x = KQuant._inputs(c, seed)
        return w, x, torch.empty(c["rows"], c["n"], device=DEV)

    @staticmethod
    def run(c, s):
        w, x, y = s
        _ok(ffi.cuda().greta_cuda_gemv_kquant(_stream(), SUPER[c["ggml"]][0], x.data_ptr(), w.data_ptr(), y.data_ptr(), c["rows"], c["n"], c["k"]), "gemv_kquant")
        return y

    @staticmethod
    def exact(c, seed):
        w, x = KQuant._inputs(c, seed)
        return x.to(F64) @ _super_values(c["ggml"], w, c["n"], c["k"]).T

    @staticmethod
    def work(c):
        return {"bytes": c["n"] * c["k"] / 256 * SUPER[c["ggml"]][1] + 4 * c["rows"] * (c["k"] + c["n"]), "flops": 2 * c["rows"] * c["n"] * c["k"]}

    @staticmethod
    def tolerance(c):
        return {"rel": 1e-5, "max": 1e-4}


# ------------------------------------------------------------------------------------------------------------------ interface
KINDS = {"llama_decode": LlamaDecode, "llama_prefill": LlamaPrefill, "windowed_prefill": HybridPrefill, "windowed_decode": HybridDecode,
         "latent_prefill": HybridPrefill, "latent_decode": HybridDecode, "layer": Layer, "kquant": KQuant}


def prepare(case, seed):
    return case, KINDS[case["kind"]].prepare(case, seed)


def run(state):
    case, s = state
    return KINDS[case["kind"]].run(case, s)


def work(case):
    return KINDS[case["kind"]].work(case)


def tolerance(case):
    return KINDS[case["kind"]].tolerance(case)


def exact(case, seed):
    with torch.no_grad():
        return KINDS[case["kind"]].exact(case, seed)
