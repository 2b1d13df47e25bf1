"""The workloads whose speed is tracked: what a program that uses this library has it do, through its public entry points.

  gemv      one weight matrix times one vector through the kernel-launcher boundary (kernels.launch_gemv), any GGUF format
  layer     one decoder layer of one decoded token, as the launcher boundary's host code issues it: fifteen launches
  decode    attention of one decoded token over the F16 cache (kernels.launch_attention_decode)
  prompt    causal attention of a run of prompt tokens over the cache (kernels.launch_attention_prefill)
  model     Model.forward: one token or a prompt in, the last token's logits on the host out.  The model has the layers of its shape
            (Llama-3 8B, 70B and smaller ones), fewer of them: a stack of random layers amplifies round-off, and time goes with depth
  family    Model.forward_logits of a model folder's family (Zelunex, BF16 tensors): one token or a prompt

A case is a dict of plain values; prepare() makes the inputs from the seed, on the GPU; run() is one pass; exact() is the same in 64 bits.
"""
from __future__ import annotations

import math

import torch

from ntransformer_b200 import kernels
from ntransformer_b200.dtypes import DType
from ntransformer_b200.engine import Model
from ntransformer_b200.model_spec import LlamaConfig

_TYPES = {"Q4_0": DType.Q4_0, "Q8_0": DType.Q8_0, "Q4_K": DType.Q4_K_M, "Q5_K": DType.Q5_K, "Q6_K": DType.Q6_K, "F16": DType.F16}
_BLOCK = {"Q4_0": (32, 18), "Q8_0": (32, 34), "Q4_K": (256, 144), "Q5_K": (256, 176), "Q6_K": (256, 210), "F16": (1, 2)}   # weights, bytes
_EPS = 1e-5


# ---- the cases ----------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # the key or value projection of an 8B model kept in 8 bits: the smallest call, all launch and latency
        {"name": "gemv_q8_0_small", "kind": "gemv", "type": "Q8_0", "rows": 1024, "cols": 4096},
        # the down projection of a 7B model in Q6_K: 43 blocks to a row, rows of 9030 bytes that start at any even address
        {"name": "gemv_q6_k_ragged", "kind": "gemv", "type": "Q6_K", "rows": 4096, "cols": 11008},
        # the output head over a 128k vocabulary: the largest matrix of a decode step
        {"name": "gemv_q6_k_head", "kind": "gemv", "type": "Q6_K", "rows": 128256, "cols": 4096},
        # a layer of the 8B model in Q4_K_M, driven launch by launch from a host program behind the launcher boundary
        {"name": "layer_q4_k_m", "kind": "layer", "mix": "Q4_K_M", "hidden": 4096, "inter": 14336, "heads": 32, "kv_heads": 8, "dim": 128, "ctx": 777},
        # a decoded token of a 70B model deep in a conversation
        {"name": "decode_attention", "kind": "decode", "heads": 64, "kv_heads": 8, "dim": 128, "ctx": 4000},
        # the second half of a long prompt, 8B heads
        {"name": "prompt_attention", "kind": "prompt", "heads": 32, "kv_heads": 8, "dim": 128, "tokens": 1000, "start": 1023},
        # the decode step, 8B shape (the reference's own benchmark is this step)
        {"name": "step_8b_q4_k_m", "kind": "model", "mix": "Q4_K_M", "hidden": 4096, "inter": 14336, "heads": 32, "kv_heads": 8, "dim": 128,
         "layers": 6, "vocab": 128256, "start": 511, "tokens": 1},
        # the decode step, 70B shape: the headline workload
        {"name": "step_70b_q4_k_m", "kind": "model", "mix": "Q4_K_M", "hidden": 8192, "inter": 28672, "heads": 64, "kv_heads": 8, "dim": 128,
         "layers": 4, "vocab": 128256, "start": 63, "tokens": 1},
        # a user's next turn in a chat: a few tokens behind what the cache holds
        {"name": "turn_8b_q4_k_m", "kind": "model", "mix": "Q4_K_M", "hidden": 4096, "inter": 14336, "heads": 32, "kv_heads": 8, "dim": 128,
         "layers": 4, "vocab": 128256, "start": 300, "tokens": 21},
        # a prompt of ordinary length into a quantised model
        {"name": "prompt_8b_q4_k_m", "kind": "model", "mix": "Q4_K_M", "hidden": 4096, "inter": 14336, "heads": 32, "kv_heads": 8, "dim": 128,
         "layers": 2, "vocab": 128256, "start": 0, "tokens": 500},
        # a long prompt into an F16 model
        {"name": "prompt_8b_f16", "kind": "model", "mix": "F16", "hidden": 4096, "inter": 14336, "heads": 32, "kv_heads": 8, "dim": 128,
         "layers": 2, "vocab": 128256, "start": 0, "tokens": 2048},
        # the decode step of a model folder in BF16, windowed attention
        {"name": "family_step_bf16", "kind": "family", "width": 4096, "ff": 14336, "heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128, "window": 1024,
         "layers": 2, "vocab": 32000, "start": 600, "tokens": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "gemv", "layer", "decode", "prompt", "model", "model", "model", "family"])
    if kind == "gemv":
        t = rng.choice(sorted(_TYPES))
        cols = 256 * _log(rng, 4, 112)
        rows = _log(rng, 256, 128256)
        return {"kind": kind, "type": t, "rows": max(17, min(rows, int(128256 * 4096 / cols * 0.82 / (_BLOCK[t][1] / _BLOCK[t][0])))), "cols": cols}
    dim = rng.choice([64, 128, 128])
    kv = rng.choice([2, 4, 8, 8])
    heads = kv * rng.choice([1, 2, 4, 4, 8])
    if kind == "decode":
        return {"kind": kind, "heads": heads, "kv_heads": kv, "dim": dim, "ctx": _log(rng, 1, 8000)}
    if kind == "prompt":
        return {"kind": kind, "heads": heads, "kv_heads": kv, "dim": dim, "tokens": _log(rng, 17, 1500), "start": rng.choice([0, _log(rng, 1, 1500)])}
    heads = rng.choice([16, 24, 32])
    shape = {"hidden": 128 * heads, "inter": 256 * rng.randint(16, 56), "heads": heads, "kv_heads": rng.choice([4, 8]), "dim": 128}
    if kind == "layer":
        return {"kind": kind, "mix": rng.choice(["Q4_0", "Q8_0", "Q4_K_M", "Q5_K", "Q6_K", "F16"]), **shape, "ctx": _log(rng, 1, 4000)}
    vocab = rng.choice([32000, 50257, 128256])
    if kind == "model":
        mode = rng.choice(["step", "step", "turn", "prompt", "prompt"])
        tokens = {"step": 1, "turn": _log(rng, 2, 31), "prompt": _log(rng, 32, 1100)}[mode]
        start = _log(rng, 1, 1900) if mode != "prompt" else rng.choice([0, 0, _log(rng, 1, 900)])
        return {"kind": kind, "mix": rng.choice(["Q4_0", "Q8_0", "Q4_K_M", "Q4_K_M", "Q5_K", "Q6_K", "F16"]), **shape, "layers": rng.randint(1, 2),
                "vocab": vocab, "start": start, "tokens": tokens}
    return {"kind": kind, "width": 1024 * rng.randint(1, 4), "ff": 1024 * rng.randint(2, 12), "heads": 16, "kv_heads": rng.choice([4, 8]), "dim": 128,
            "vdim": rng.choice([64, 128]), "window": 256 * rng.randint(1, 4), "layers": rng.randint(1, 2), "vocab": 32000, "start": _log(rng, 1, 900),
            "tokens": rng.choice([1, 1, _log(rng, 2, 700)])}


# ---- inputs -------------------------------------------------------------------------------------------------------------------

# (d, dmin) that give weights of deviation about 1 with uniform codes: w = d * sc * q - dmin * m (Q4_K, Q5_K), d * sc * (q - 32) (Q6_K), d * q
_UNIT = {"Q4_K": (1 / 160.0, 7.5 / 160.0), "Q5_K": (1 / 330.0, 15.5 / 330.0), "Q6_K": (1 / 170.0, 0.0), "Q8_0": (1 / 73.6, 0.0), "Q4_0": (1 / 4.6, 0.0)}


class _Source:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0):
        return torch.randn(shape, generator=self.g, device="cuda") * std

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.g, device="cuda")

    def activations(self, n):
        """A residual stream's vector: a few channels are ten times the others."""
        return self.normal(n) * (1 + 9 * (self.uniform(n) < 0.01))

    def tokens(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.g, device="cuda").tolist()

    def weights(self, t, rows, cols, std):
        """Rows of GGUF blocks: uint8 [rows, bytes]."""
        if t == "F16":
            return (self.normal(rows, cols) * std).half().view(torch.uint8).reshape(rows, -1)
        w, size = _BLOCK[t]
        nb = cols // w
        b = torch.randint(0, 256, (rows, nb, size), generator=self.g, device="cuda", dtype=torch.uint8)
        jitter = self.uniform(rows, nb) + 0.5
        two = lambda u: (jitter * (u * std)).half().view(torch.uint8).reshape(rows, nb, 2)   # noqa: E731
        d, dmin = _UNIT[t]
        if t == "Q6_K":
            b[:, :, 192:208] = torch.randint(-16, 16, (rows, nb, 16), generator=self.g, device="cuda", dtype=torch.int8).view(torch.uint8)
            b[:, :, 208:210] = two(d)
        else:
            b[:, :, 0:2] = two(d)
            if dmin:
                b[:, :, 2:4] = two(dmin)
        return b.reshape(rows, nb * size)


def _mix_type(mix, name, layer, layers):
    if mix != "Q4_K_M":
        return mix
    if name == "output":
        return "Q6_K"
    more = layer < layers // 8 or layer >= 7 * layers // 8 or (layer - layers // 8) % 3 == 2       # llama.cpp's rule for this mix
    return "Q6_K" if name in ("attn_v", "ffn_down") and more else "Q4_K"


def _layer_weights(src, c, layer, layers):
    h, q, kv, f = c["hidden"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["inter"]
    w = {}
    for name, rows, cols in (("attn_q", q, h), ("attn_k", kv, h), ("attn_v", kv, h), ("attn_output", h, q), ("ffn_gate", f, h), ("ffn_up", f, h), ("ffn_down", h, f)):
        t = _mix_type(c["mix"], name, layer, layers)
        w[name] = (src.weights(t, rows, cols, cols ** -0.5), t)
    for name in ("attn_norm", "ffn_norm"):
        w[name] = (1 + 0.1 * src.normal(h), "F32")
    return w


def _model_weights(c, seed):
    src = _Source(seed)
    w = {"token_embd": (src.weights(_mix_type(c["mix"], "token_embd", 0, 1), c["vocab"], c["hidden"], 1.0), _mix_type(c["mix"], "token_embd", 0, 1)),
         "output_norm": (1 + 0.1 * src.normal(c["hidden"]), "F32"),
         "output": (src.weights(_mix_type(c["mix"], "output", 0, 1), c["vocab"], c["hidden"], c["hidden"] ** -0.5), _mix_type(c["mix"], "output", 0, 1))}
    for i in range(c["layers"]):
        for name, v in _layer_weights(src, c, i, c["layers"]).items():
            w["blk.%d.%s" % (i, name)] = v
    return w, src.tokens(c["start"], c["vocab"]), src.tokens(c["tokens"], c["vocab"])


def _family_config(c):
    mixer = {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": c["dim"], "vdim": c["vdim"], "scale": c["dim"] ** -0.5, "softcap": 30.0,
             "mask": {"size": c["window"], "keep_first": 4}}
    return {"architecture": "Zelunex", "vocab": c["vocab"], "width": c["width"], "norm": {"eps": _EPS}, "residual_mult": 0.5,
            "layers": [{"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": c["ff"]}} for _ in range(c["layers"])]}


def _family_weights(c, seed):
    src = _Source(seed)
    W, q, k, v, f = c["width"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["kv_heads"] * c["vdim"], c["ff"]
    mat = lambda rows, cols, std: src.normal(rows, cols, std=std).bfloat16()   # noqa: E731
    vec = lambda n: 1 + 0.1 * src.normal(n)   # noqa: E731
    t = {"embed": mat(c["vocab"], W, 1.0), "final.norm": vec(W), "head": mat(c["vocab"], W, W ** -0.5)}
    for i in range(c["layers"]):
        p = "l%d." % i
        t.update({p + "norm1": vec(W), p + "mix.q": mat(q, W, W ** -0.5), p + "mix.k": mat(k, W, W ** -0.5), p + "mix.v": mat(v, W, W ** -0.5),
                  p + "mix.q.norm": vec(q), p + "mix.k.norm": vec(k), p + "mix.o": mat(W, c["heads"] * c["vdim"], (c["heads"] * c["vdim"]) ** -0.5),
                  p + "ls1": vec(W), p + "mlp.gate": mat(f, W, W ** -0.5), p + "mlp.up": mat(f, W, W ** -0.5), p + "mlp.down": mat(W, f, f ** -0.5),
                  p + "ls2": vec(W)})
    return t, src.tokens(c["start"], c["vocab"]), src.tokens(c["tokens"], c["vocab"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "model":
        w, before, now = _model_weights(c, seed)
        cfg = LlamaConfig(vocab_size=c["vocab"], hidden_size=c["hidden"], intermediate_size=c["inter"], n_layers=c["layers"], n_heads=c["heads"],
                          n_kv_heads=c["kv_heads"], head_dim=c["dim"], max_seq_len=4096, norm_eps=_EPS, rope_theta=500000.0)
        m = Model.from_device_tensors(cfg, {n + ".weight": (t, DType.F32 if d == "F32" else _TYPES[d]) for n, (t, d) in w.items()})
        if before:
            m.forward(before, 0, want_logits=False)
        return {"case": c, "model": m, "tokens": now}
    if kind == "family":
        t, before, now = _family_weights(c, seed)
        m = Model.from_config_json(_family_config(c), t, max_context=2048)
        m.forward_logits(before, 0, [])
        return {"case": c, "model": m, "tokens": now}
    src = _Source(seed)
    if kind == "gemv":
        return {"case": c, "W": src.weights(c["type"], c["rows"], c["cols"], c["cols"] ** -0.5), "x": src.activations(c["cols"]),
                "y": torch.empty(c["rows"], device="cuda")}
    keys = {"layer": c.get("ctx", 0), "decode": c.get("ctx", 0), "prompt": c.get("start", 0) + c.get("tokens", 0)}[kind]
    cache = (max(keys, 4096), c["kv_heads"], c["dim"])
    s = {"case": c, "k_cache": src.normal(*cache).half(), "v_cache": src.normal(*cache).half()}
    n = c.get("tokens", 1)
    if kind == "layer":
        s.update(weights=_layer_weights(src, c, 0, 8), hidden=src.activations(c["hidden"]), pos=torch.tensor([c["ctx"] - 1], dtype=torch.int32, device="cuda"))
        for name, size in (("x", c["hidden"]), ("norm", c["hidden"]), ("q", c["heads"] * c["dim"]), ("k", c["kv_heads"] * c["dim"]), ("v", c["kv_heads"] * c["dim"]),
                           ("attn", c["heads"] * c["dim"]), ("proj", c["hidden"]), ("gate", c["inter"]), ("up", c["inter"])):
            s[name] = torch.empty(size, device="cuda")
        return s
    s.update(q=src.normal(n, c["heads"], c["dim"]), out=torch.empty(n, c["heads"], c["dim"], device="cuda"))
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------------------

def _layer_pass(s):
    """The launch sequence of a decoder layer behind the launcher boundary."""
    c, w, K = s["case"], s["weights"], kernels
    h, f, nh, nkv, hd, pos = c["hidden"], c["inter"], c["heads"], c["kv_heads"], c["dim"], c["ctx"] - 1

    def gemv(y, name, x, rows, cols):
        K.launch_gemv(y, w[name][0], x, rows, cols, _TYPES[w[name][1]])

    K.launch_copy(s["x"], s["hidden"], h)
    K.launch_rmsnorm(s["norm"], s["x"], w["attn_norm"][0], 1, h, _EPS)
    gemv(s["q"], "attn_q", s["norm"], nh * hd, h)
    gemv(s["k"], "attn_k", s["norm"], nkv * hd, h)
    gemv(s["v"], "attn_v", s["norm"], nkv * hd, h)
    K.launch_rope(s["q"], s["k"], s["pos"], 1, 1, nh, nkv, hd, 500000.0, 1.0, False)
    K.launch_copy_to_kv_cache(s["k_cache"], s["v_cache"], s["k"], s["v"], 1, nkv, hd, pos, s["k_cache"].shape[0])
    K.launch_attention_decode(s["attn"], s["q"], s["k_cache"], s["v_cache"], c["ctx"], nh, nkv, hd, s["k_cache"].shape[0], hd ** -0.5)
    gemv(s["proj"], "attn_output", s["attn"], h, nh * hd)
    K.launch_add_inplace(s["x"], s["proj"], h)
    K.launch_rmsnorm(s["norm"], s["x"], w["ffn_norm"][0], 1, h, _EPS)
    gemv(s["gate"], "ffn_gate", s["norm"], f, h)
    gemv(s["up"], "ffn_up", s["norm"], f, h)
    K.launch_silu_mul(s["gate"], s["gate"], s["up"], f)
    gemv(s["proj"], "ffn_down", s["gate"], h, f)
    K.launch_add_inplace(s["x"], s["proj"], h)
    return {"hidden": s["x"], "key": s["k_cache"][pos], "value": s["v_cache"][pos]}


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "model":
        return s["model"].forward(s["tokens"], c["start"])
    if kind == "family":
        return s["model"].forward_logits(s["tokens"], c["start"], [c["tokens"] - 1])
    if kind == "gemv":
        kernels.launch_gemv(s["y"], s["W"], s["x"], c["rows"], c["cols"], _TYPES[c["type"]])
        return s["y"]
    if kind == "layer":
        return _layer_pass(s)
    rows = s["k_cache"].shape[0]
    if kind == "decode":
        kernels.launch_attention_decode(s["out"], s["q"], s["k_cache"], s["v_cache"], c["ctx"], c["heads"], c["kv_heads"], c["dim"], rows, c["dim"] ** -0.5)
    else:
        kernels.launch_attention_prefill(s["out"], s["q"], s["k_cache"], s["v_cache"], c["tokens"], c["start"], c["heads"], c["kv_heads"], c["dim"], rows,
                                         c["dim"] ** -0.5)
    return s["out"]


# ---- what a pass cannot do without --------------------------------------------------------------------------------------------

def _bytes(t, rows, cols):
    return rows * cols // _BLOCK[t][0] * _BLOCK[t][1]


def work(case):
    c, kind = case, case["kind"]
    if kind == "gemv":
        return {"bytes": _bytes(c["type"], c["rows"], c["cols"]) + 4 * (c["rows"] + c["cols"]), "flops": 2 * c["rows"] * c["cols"]}
    n = c.get("tokens", 1)
    start = c.get("start", c.get("ctx", 1) - 1)
    pairs = n * start + n * (n + 1) // 2
    if kind in ("decode", "prompt"):
        return {"bytes": 4 * c["kv_heads"] * c["dim"] * (start + n) + 8 * n * c["heads"] * c["dim"], "flops": 4 * pairs * c["heads"] * c["dim"]}
    if kind == "family":
        pairs = sum(min(start + i + 1, c["window"] + 4) for i in range(n))
        q, k, v = c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["kv_heads"] * c["vdim"]
        params = c["layers"] * c["width"] * (q + k + v + c["heads"] * c["vdim"] + 3 * c["ff"])
        head = c["vocab"] * c["width"]
        return {"bytes": 2 * (params + head) + c["layers"] * 2 * (k + v) * min(start + n, c["window"] + 4 + n),
                "flops": 2 * n * params + 2 * head + c["layers"] * 2 * pairs * c["heads"] * (c["dim"] + c["vdim"])}
    layers = c.get("layers", 1)
    h, q, kv, f = c["hidden"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["inter"]
    total, flops = 0, 0
    for i in range(layers):
        for name, rows, cols in (("attn_q", q, h), ("attn_k", kv, h), ("attn_v", kv, h), ("attn_output", h, q), ("ffn_gate", f, h), ("ffn_up", f, h), ("ffn_down", h, f)):
            total += _bytes(_mix_type(c["mix"], name, i, layers if kind == "model" else 8), rows, cols)
            flops += 2 * n * rows * cols
        total += 8 * h + 4 * kv * (start + n)
        flops += 4 * pairs * q
    if kind == "model":
        total += _bytes(_mix_type(c["mix"], "output", 0, 1), c["vocab"], h) + n * _bytes(_mix_type(c["mix"], "token_embd", 0, 1), 1, h) + 4 * (c["vocab"] + h)
        flops += 2 * c["vocab"] * h
    return {"bytes": total, "flops": flops}


# About four times what was seen against 64 bits (1.1e-6, 4.6e-5, 1.2e-6, 3.9e-6, 6e-4, and 1.6e-5 for one token of a family, whose prompts split
# their activations into two BF16).  GEMV and attention work in 32 bits or splits as good; the rotation's angle carries the rounding of its 32-bit
# frequency times the position, which a model's layers carry on; a layer's key is rounded to the cache's 16 bits, now and then to the other side.
_TOLERANCE = {"gemv": 5e-6, "layer": 2e-4, "decode": 5e-6, "prompt": 2e-5, "model": 2e-3, "family": 1e-3}


def tolerance(case):
    return {"rel": _TOLERANCE[case["kind"]]}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------

def _dequant(w, t, rows, cols):
    """GGUF blocks -> float64 [rows, cols]."""
    if t == "F32":
        return w.double()
    if t == "F16":
        return w.view(torch.float16).reshape(rows, cols).double()
    n, size = _BLOCK[t]
    b = w.reshape(rows, cols // n, size)
    half = lambda i: b[:, :, i:i + 2].contiguous().view(torch.float16).double()   # noqa: E731
    if t == "Q8_0":
        return (half(0) * b[:, :, 2:].contiguous().view(torch.int8).double()).reshape(rows, cols)
    if t == "Q4_0":
        q = b[:, :, 2:]
        return (half(0) * (torch.cat([q & 15, q >> 4], 2).double() - 8)).reshape(rows, cols)
    if t == "Q6_K":
        ql, qh = b[:, :, :128].reshape(rows, -1, 2, 2, 32), b[:, :, 128:192].reshape(rows, -1, 2, 32)
        q = torch.stack([(ql[:, :, :, 0] & 15) | ((qh & 3) << 4), (ql[:, :, :, 1] & 15) | (((qh >> 2) & 3) << 4),
                         (ql[:, :, :, 0] >> 4) | (((qh >> 4) & 3) << 4), (ql[:, :, :, 1] >> 4) | ((qh >> 6) << 4)], 3)
        sc = b[:, :, 192:208].contiguous().view(torch.int8).double() * half(208)
        return ((q.reshape(rows, -1, 16, 16).double() - 32) * sc.unsqueeze(3)).reshape(rows, cols)
    s = b[:, :, 4:16]
    sc = torch.cat([s[:, :, 0:4] & 63, (s[:, :, 8:12] & 15) | ((s[:, :, 0:4] >> 6) << 4)], 2).double() * half(0)
    mn = torch.cat([s[:, :, 4:8] & 63, (s[:, :, 8:12] >> 4) | ((s[:, :, 4:8] >> 6) << 4)], 2).double() * half(2)
    qs = b[:, :, size - 128:].reshape(rows, -1, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], 3).reshape(rows, -1, 8, 32)
    if t == "Q5_K":
        bit = torch.arange(8, device=w.device, dtype=torch.uint8).reshape(1, 1, 8, 1)
        q = q | (((b[:, :, 16:48].unsqueeze(2) >> bit) & 1) << 4)
    return (q.double() * sc.unsqueeze(3) - mn.unsqueeze(3)).reshape(rows, cols)


def _product(x, w, t, cols):
    """x [n, cols] times the matrix's rows, a slice of them at a time."""
    rows = w.shape[0]
    step = max(1, (1 << 26) // cols)
    return torch.cat([x @ _dequant(w[r:r + step], t, min(step, rows - r), cols).T for r in range(0, rows, step)], 1)


def _rms(x, g):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + _EPS) * g.double()


def _attention(q, k, v, start, scale, window=0, keep=0, cap=0.0):
    """q [n, heads, dim], k and v [keys, kv_heads, .]; query i sees the keys up to start + i."""
    n, heads, group = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    i = torch.arange(n, device=q.device).unsqueeze(1) + start
    j = torch.arange(k.shape[0], device=q.device).unsqueeze(0)
    hidden = j > i
    if window:
        hidden |= (i - j >= window) & (j >= keep)
    out = []
    for h in range(heads):
        s = q[:, h] @ k[:, h // group].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        out.append(torch.softmax(s.masked_fill(hidden, -math.inf), 1) @ v[:, h // group])
    return torch.stack(out, 1)


def _rotate(x, pos):
    half = x.shape[2] // 2
    a = pos.double().reshape(-1, 1, 1) * 500000.0 ** (-torch.arange(half, device=x.device, dtype=torch.float64) * 2 / x.shape[2])
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], 2)


def _layer64(x, w, c, start, cache=None):
    """One decoder layer for the tokens at start ...; `cache`: the keys and values before them, else x holds the sequence from its start."""
    n, h, nh, nkv, hd, f = x.shape[0], c["hidden"], c["heads"], c["kv_heads"], c["dim"], c["inter"]
    pos = torch.arange(start, start + n, device=x.device)
    u = _rms(x, w["attn_norm"][0])
    q = _rotate(_product(u, *w["attn_q"], h).reshape(n, nh, hd), pos)
    k = _rotate(_product(u, *w["attn_k"], h).reshape(n, nkv, hd), pos).half()      # the cache holds F16
    v = _product(u, *w["attn_v"], h).reshape(n, nkv, hd).half()
    ks, vs = (torch.cat([p.double(), t.double()]) for p, t in zip(cache, (k, v))) if cache else (k.double(), v.double())
    a = _attention(q, ks, vs, start, hd ** -0.5).reshape(n, nh * hd)
    x = x + _product(a, *w["attn_output"], nh * hd)
    u = _rms(x, w["ffn_norm"][0])
    g = _product(u, *w["ffn_gate"], h)
    return x + _product(g * torch.sigmoid(g) * _product(u, *w["ffn_up"], h), *w["ffn_down"], f), k, v


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "model":
        w, before, now = _model_weights(c, seed)
        x = _dequant(w["token_embd"][0][torch.tensor(before + now, device="cuda")], w["token_embd"][1], c["start"] + c["tokens"], c["hidden"])
        for i in range(c["layers"]):
            x = _layer64(x, {n.split(".")[-1]: v for n, v in w.items() if n.startswith("blk.%d." % i)}, c, 0)[0]
        return _product(_rms(x[-1:], w["output_norm"][0]), *w["output"], c["hidden"])[0]
    if kind == "family":
        t, before, now = _family_weights(c, seed)
        x = t["embed"][torch.tensor(before + now, device="cuda")].double()
        n = x.shape[0]
        for i in range(c["layers"]):
            W = {k[len("l%d." % i):]: v.double() for k, v in t.items() if k.startswith("l%d." % i)}
            u = _rms(x, W["norm1"])
            q = _rms(u @ W["mix.q"].T, W["mix.q.norm"]).reshape(n, c["heads"], c["dim"])
            k = _rms(u @ W["mix.k"].T, W["mix.k.norm"]).bfloat16().double().reshape(n, c["kv_heads"], c["dim"])      # the cache holds BF16
            v = (u @ W["mix.v"].T).bfloat16().double().reshape(n, c["kv_heads"], c["vdim"])
            a = _attention(q, k, v, 0, c["dim"] ** -0.5, c["window"], 4, 30.0).reshape(n, -1)
            g = u @ W["mlp.gate"].T
            act = 0.5 * g * (1 + torch.tanh(math.sqrt(2 / math.pi) * (g + 0.044715 * g ** 3)))
            x = x + 0.5 * ((a @ W["mix.o"].T) * W["ls1"] + ((act * (u @ W["mlp.up"].T)) @ W["mlp.down"].T) * W["ls2"])
        return (_rms(x[-1:], t["final.norm"]) @ t["head"].double().T)
    s = prepare(case, seed)
    if kind == "gemv":
        return _product(s["x"].double().unsqueeze(0), s["W"], c["type"], c["cols"])[0]
    if kind == "layer":
        pos = c["ctx"] - 1
        x, k, v = _layer64(s["hidden"].double().unsqueeze(0), s["weights"], c, pos, (s["k_cache"][:pos], s["v_cache"][:pos]))
        return {"hidden": x[0], "key": k[0].double(), "value": v[0].double()}
    start = c.get("start", c.get("ctx", 1) - 1)
    n = c.get("tokens", 1)
    return _attention(s["q"].double(), s["k_cache"][:start + n].double(), s["v_cache"][:start + n].double(), start, c["dim"] ** -0.5)
