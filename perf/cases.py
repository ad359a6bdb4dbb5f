"""The work whose speed counts: calls of the operators and of the language models through their public entry points, over
the sizes that programs use. `listed()` names some, `draw()` gives more of the same ranges; `exact()` is the same
work in 64 bits by plain torch.

Kinds of case:
  elementwise  a bias added to activations, products, activations, casts, swiglu: one launch, latency at the small end
  rows         softmax, norms and reductions over any axes
  chain        rmsNorm + residual + softmax + cast in one pass
  matmul       products of matrices, batched or with a shared right operand, and linear layers (right operand transposed)
  attention    scaledDotProductAttention with its masks, grouped heads, chunks of queries behind older keys
  qwen3        a prompt and single-token steps of the Qwen3-0.6B shape (bf16 weights, fp32 activations)
  lm           the same of the Duzozen (dense, with experts) and Derupel (dense) models in bf16
"""
import math
import zlib

import numpy as np
import torch

from ytensor_b200 import api
from ytensor_b200.derupel import DECAYED, LATENT, DerupelConfig, DerupelForCausalLM, DerupelLayer
from ytensor_b200.duzozen import DuzozenConfig, DuzozenForCausalLM, DuzozenLayer
from ytensor_b200.native_lm import MLP_DENSE, MLP_MOE
from ytensor_b200.qwen3 import Qwen3Config, Qwen3ForCausalLM

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}


def listed():
    return [
        # the bias behind a linear layer of a few rows: what a small network's step is made of
        {"name": "bias_add_small", "kind": "elementwise", "op": "add", "rows": 7, "cols": 1024, "dtype": "f32"},
        # an image network's normalisation: statistics over every axis but the channel
        {"name": "batchnorm_image", "kind": "rows", "op": "batchNorm", "n": 16, "c": 96, "h": 56, "w": 56, "dtype": "f32"},
        # the fused row chain on activations of 4096 channels
        {"name": "chain_4096", "kind": "chain", "b": 8, "l": 2048, "h": 4096, "residual": "shared"},
        # batches of activations times one weight matrix
        {"name": "matmul_bf16_batched", "kind": "matmul", "batch": 8, "m": 2048, "n": 4096, "k": 4096, "dtype": "bf16",
         "form": "shared"},
        # the size of the reference's own benchmark, in its default number format
        {"name": "matmul_f32_1024", "kind": "matmul", "batch": 1, "m": 1024, "n": 1024, "k": 1024, "dtype": "f32",
         "form": "shared"},
        # a long prompt's causal attention with four query heads to a key head
        {"name": "attn_bf16_causal", "kind": "attention", "b": 2, "kv": 8, "groups": 4, "lq": 4096, "lk": 4096, "d": 128,
         "dtype": "bf16", "mask": "causal"},
        # the default number format, an odd length
        {"name": "attn_f32_causal", "kind": "attention", "b": 1, "kv": 8, "groups": 2, "lq": 1000, "lk": 1000, "d": 128,
         "dtype": "f32", "mask": "causal"},
        # reading a long prompt
        {"name": "qwen3_prefill", "kind": "qwen3", "batch": 1, "prompt": 2000, "steps": 0},
        # one user: a short prompt, then token by token
        {"name": "qwen3_decode_1", "kind": "qwen3", "batch": 1, "prompt": 100, "steps": 40},
        # many users
        {"name": "qwen3_decode_32", "kind": "qwen3", "batch": 32, "prompt": 60, "steps": 20},
        # a long prompt through windowed attention and a mixture of experts
        {"name": "duzozen_experts_prefill", "kind": "lm", "model": "duzozen", "width": 1024, "layers": 2, "experts": 64,
         "prompt": 4000, "steps": 0},
        # a prompt, then token by token, through linear and latent attention
        {"name": "derupel_dense_decode", "kind": "lm", "model": "derupel", "width": 1024, "layers": 12, "experts": 0,
         "prompt": 500, "steps": 40},
    ]


# ---------------------------------------------------------------------------------------------- drawn cases
def _log(rng, lo, hi, odd=0.4):
    """A whole number, even over the logarithm; often a multiple of 64 or 8, else as it falls."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() > odd:
        step = 64 if n >= 256 else 8 if n >= 32 else 1
        n = (n + step - 1) // step * step
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["elementwise", "rows", "rows", "chain", "matmul", "matmul", "attention", "attention", "qwen3",
                       "qwen3", "lm", "lm"])
    dtype = rng.choice(["f32", "f32", "bf16", "f16"])
    if kind == "elementwise":
        op = rng.choice(["add", "mul", "swish", "gelu", "cast", "swiglu"])
        return {"kind": kind, "op": op, "rows": _log(rng, 1, 4096), "cols": _log(rng, 64, 8192),
                "dtype": "f32" if op == "cast" else dtype}
    if kind == "rows":
        op = rng.choice(["batchNorm", "groupNorm", "layerNorm", "rmsNorm", "softmax", "sum", "mean", "max"])
        if op in ("batchNorm", "groupNorm"):
            side = _log(rng, 7, 112)
            return {"kind": kind, "op": op, "n": _log(rng, 1, 32), "c": 8 * rng.randint(1, 32), "h": side, "w": side,
                    "dtype": dtype}
        return {"kind": kind, "op": op, "n": 1, "c": 1, "h": _log(rng, 1, 4096), "w": _log(rng, 64, 8192),
                "axis": rng.choice([3, 3, 2]) if op != "rmsNorm" else 3, "dtype": dtype}
    if kind == "chain":
        return {"kind": kind, "b": _log(rng, 1, 8), "l": _log(rng, 1, 2048), "h": 4 * _log(rng, 64, 1024),
                "residual": rng.choice(["shared", "own"])}
    if kind == "matmul":
        form = rng.choice(["shared", "batched", "linear"])
        while True:
            c = {"kind": kind, "batch": rng.choice([1, 1, 2, 4, 8]), "m": _log(rng, 1, 4096), "n": _log(rng, 64, 8192),
                 "k": _log(rng, 64, 8192), "dtype": dtype, "form": form}
            if c["batch"] * c["m"] * c["n"] * c["k"] <= (2.7e11 if dtype != "f32" else 3.2e10):
                return c
    if kind == "attention":
        while True:
            lk = _log(rng, 16, 4096)
            c = {"kind": kind, "b": rng.choice([1, 1, 2, 4]), "kv": rng.choice([1, 4, 8, 12]),
                 "groups": rng.choice([1, 1, 2, 4]), "lq": rng.choice([lk, lk, _log(rng, 1, lk)]), "lk": lk,
                 "d": rng.choice([64, 64, 128, 128, 80]), "dtype": dtype,
                 "mask": rng.choice(["causal", "causal", "none", "bool", "bias"])}
            work = c["b"] * c["kv"] * c["groups"] * c["lq"] * lk * c["d"]
            if work <= (1.4e11 if dtype != "f32" and c["mask"] != "bias" and c["d"] != 80 else 8e9):
                return c
    if kind == "qwen3":
        batch = rng.choice([1, 1, 2, 4, 8, 16, 32])
        prompt = _log(rng, 1, 2048 // batch)
        steps = 0 if prompt > 700 else rng.randint(1, 40 if batch < 8 else 20)
        return {"kind": kind, "batch": batch, "prompt": prompt, "steps": steps}
    prompt, model = _log(rng, 1, 4096), rng.choice(["duzozen", "derupel"])
    experts = rng.choice([0, 64]) if model == "duzozen" else 0  # (deeper, near ties of the routers would add up)
    return {"kind": kind, "model": model, "width": rng.choice([512, 1024, 1024]),
            "layers": 2 if experts else rng.choice([4, 8, 12]), "experts": experts, "prompt": prompt,
            "steps": 0 if prompt > 1000 else rng.randint(1, 40)}


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, shape, dtype="f32", std=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * std).to(DTYPES[dtype])


def _operands(c, seed):
    """name -> tensor of an operator case."""
    g, dt = _gen(seed), c.get("dtype", "f32")
    if c["kind"] == "elementwise":
        s = {"x": _randn(g, (c["rows"], c["cols"] * (2 if c["op"] == "swiglu" else 1)), dt)}
        if c["op"] == "add":
            s["y"] = _randn(g, (c["cols"],), dt)
        elif c["op"] == "mul":
            s["y"] = _randn(g, (c["rows"], c["cols"]), dt)
        return s
    if c["kind"] == "rows":
        if c["op"] in ("batchNorm", "groupNorm"):
            s = {"x": _randn(g, (c["n"], c["c"], c["h"], c["w"]), dt) * 1.5 + 0.3}
            s["w"], s["b"] = 1 + 0.1 * _randn(g, (c["c"],), dt), 0.1 * _randn(g, (c["c"],), dt)
            return s
        s = {"x": _randn(g, (c["h"], c["w"]), dt, 2.0)}
        size = c["w"] if c["axis"] == 3 else c["h"]
        if c["op"] in ("rmsNorm", "layerNorm"):
            s["w"] = 1 + 0.1 * _randn(g, (size,), dt)
        if c["op"] == "layerNorm":
            s["b"] = 0.1 * _randn(g, (size,), dt)
        return s
    if c["kind"] == "chain":
        own = c["residual"] == "own"
        return {"x": _randn(g, (c["b"], c["l"], c["h"])), "w": 1 + 0.1 * _randn(g, (c["h"],)),
                "r": _randn(g, (c["b"] if own else 1, c["l"], c["h"]))}
    if c["kind"] == "matmul":
        lead = (c["batch"],) if c["batch"] > 1 else ()
        a = _randn(g, (*lead, c["m"], c["k"]), dt)
        std = c["k"] ** -0.5
        if c["form"] == "linear":
            return {"a": a, "b": _randn(g, (c["n"], c["k"]), dt, std)}
        return {"a": a, "b": _randn(g, (*(lead if c["form"] == "batched" else ()), c["k"], c["n"]), dt, std)}
    heads = c["kv"] * c["groups"]
    s = {"q": _randn(g, (c["b"], heads, c["lq"], c["d"]), dt), "k": _randn(g, (c["b"], c["kv"], c["lk"], c["d"]), dt),
         "v": _randn(g, (c["b"], c["kv"], c["lk"], c["d"]), dt)}
    if c["mask"] == "bool":  # every query keeps its own place and about two thirds of the others
        keep = torch.rand((c["lq"], c["lk"]), generator=g, device="cuda") < 0.66
        keep |= torch.eye(c["lq"], c["lk"], dtype=torch.bool, device="cuda")
        keep[:, 0] = True
        s["mask"] = keep
    elif c["mask"] == "bias":
        s["bias"] = _randn(g, (c["lq"], c["lk"]))
    return s


def _lm_config(c):
    """Layers of the proportions that the benchmark's models have, at the case's width and depth."""
    W, heads = c["width"], c["width"] // 64
    dense = dict(mlp=MLP_DENSE, ff=W * 9 // 2)
    if c["model"] == "duzozen":
        moe = dict(mlp=MLP_MOE, ff=W * 3 // 8, experts=c["experts"], identity=8, top=8, groups=8, keep=8)
        att = dict(heads=heads, kv_heads=heads // 2, dim=128, vdim=128, scale=128 ** -0.5, softcap=20.0, window=1024,
                   v_mix=True)
        return DuzozenConfig(width=W, vocab=32768, eps=1e-6, layers=[
            DuzozenLayer(**att, **(moe if c["experts"] and l else dense)) for l in range(c["layers"])])
    decay = [1 - 2.0 ** (-2 - 8.0 * h / heads) for h in range(heads)]
    mixers = (dict(mixer=LATENT, heads=heads, dim=64, vdim=128, rot_dim=64, rot_dims=64, kv_rank=512, q_rank=512,
                   scale=128 ** -0.5),
              dict(mixer=DECAYED, heads=heads, dim=128, vdim=128, decay=decay))
    return DerupelConfig(width=W, vocab=32768, eps=1e-6, embed_scale=W ** 0.5, layers=[
        DerupelLayer(**mixers[l % 4 != 3], **dense) for l in range(c["layers"])])


class _Weights:
    """name -> random bf16 tensor on the device, made when it is asked for."""

    def __init__(self, shapes, seed):
        self.shapes, self.seed = shapes, int(seed)

    def __getitem__(self, name):
        g, shape, leaf = _gen(self.seed * 1000003 + zlib.crc32(name.encode())), self.shapes[name], name.split(".")[-1]
        if leaf.startswith("norm"):
            return _randn(g, shape, "bf16", 0.1) + 1
        if leaf == "vmix":
            return torch.full(shape, 0.5, dtype=torch.bfloat16, device="cuda")
        if leaf == "correction":
            return _randn(g, shape, "bf16", 0.002)
        # a trained router is sure of its first choices: logits of 4 rms, so that the last of the chosen weighs little
        return _randn(g, shape, "bf16", 0.03 if leaf == "embed" else (4 if leaf == "router" else 1) * shape[-1] ** -0.5)


def _qwen3_config(c):
    return Qwen3Config(max_position_embeddings=max(256, c["prompt"] + c["steps"]))


def _qwen3_shapes(cfg):
    H, D, I = cfg.hidden_size, cfg.head_dim, cfg.intermediate_size
    s = {"embed": (cfg.vocab_size, H), "norm": (H,)}
    for l in range(cfg.num_hidden_layers):
        s[("qkv", l)] = ((cfg.num_attention_heads + 2 * cfg.num_key_value_heads) * D, H)
        s[("o", l)], s[("gate_up", l)], s[("down", l)] = (H, cfg.num_attention_heads * D), (2 * I, H), (H, I)
        s[("q_norm", l)] = s[("k_norm", l)] = (D,)
        s[("norm1", l)] = s[("norm2", l)] = (H,)
    return s


def _qwen3_weight(shape, key, seed):
    """A weight on the device; matrices bf16, as a checkpoint stores them, norm weights fp32."""
    g = _gen(int(seed) * 1000003 + zlib.crc32(repr(key).encode()))
    return 1 + 0.1 * _randn(g, shape) if len(shape) == 1 else _randn(g, shape, "bf16", 0.02)


def _ids(c, seed, vocab, batch):
    return torch.randint(0, vocab, (batch, c["prompt"] + c["steps"]), generator=_gen(seed + 7), device="cuda",
                         dtype=torch.int32)


def prepare(case, seed):
    if case["kind"] == "qwen3":
        cfg = _qwen3_config(case)
        host = {}
        for key, shape in _qwen3_shapes(cfg).items():
            w = _qwen3_weight(shape, key, seed)
            host[key] = w.view(torch.int16).cpu().numpy().view(np.uint16) if w.dtype == torch.bfloat16 else w.cpu().numpy()
        m = Qwen3ForCausalLM(cfg, batch=case["batch"])
        m.load_weights(host)
        return {"case": case, "model": m, "ids": _ids(case, seed, cfg.vocab_size, case["batch"])}
    if case["kind"] == "lm":
        cfg = _lm_config(case)
        make = DuzozenForCausalLM if case["model"] == "duzozen" else DerupelForCausalLM
        m = make(cfg, batch=1, max_tokens=case["prompt"] + case["steps"] + 1)
        m.load_weights(_Weights(cfg.tensor_shapes(), seed))
        return {"case": case, "model": m, "ids": _ids(case, seed, cfg.vocab, 1)}
    return {"case": case, **_operands(case, seed)}


# ---------------------------------------------------------------------------------------------- a pass
def _places(case):
    """Places of the prompt whose logits a replayed trace asks for: every 64th from the end."""
    return list(range((case["prompt"] - 1) % 64, case["prompt"], 64))


def _serve(s):
    """The prompt, then one token per sequence and step. The continuation is given, as a replayed trace gives it; the
    greedy choice is formed at every step."""
    c, m, ids = s["case"], s["model"], s["ids"]
    m.reset_kv_cache()
    first = ids[:, :c["prompt"]].contiguous()
    logits = m.forward_at(first, _places(c)) if c["kind"] == "lm" else m.forward(first)
    out, tokens = [logits], torch.empty(ids.shape[0], c["steps"] + 1, dtype=torch.int32, device=ids.device)
    for t in range(c["steps"] + 1):
        tok, _ = m.argmax(logits[-1:] if c["kind"] == "lm" else logits)
        tokens[:, t] = tok
        if t < c["steps"]:
            logits = m.forward(ids[:, c["prompt"] + t:c["prompt"] + t + 1].contiguous())
            out.append(logits)
    return {"logits": out, "tokens": tokens}


def run(state):
    c, s = state["case"], state
    kind, op = c["kind"], c.get("op")
    if kind in ("qwen3", "lm"):
        return _serve(s)
    if kind == "elementwise":
        if op in ("add", "mul"):
            return getattr(api, op)(s["x"], s["y"])
        return api.cast(s["x"], torch.bfloat16) if op == "cast" else getattr(api, op)(s["x"])
    if kind == "rows":
        if op == "batchNorm":
            return api.batchNorm(s["x"], s["w"], s["b"])
        if op == "groupNorm":
            return api.groupNorm(s["x"], 8, s["w"], s["b"])
        axis = c["axis"] - 2
        if op == "layerNorm":
            return api.layerNorm(s["x"], s["w"], s["b"], axis)
        if op == "rmsNorm":
            return api.rmsNorm(s["x"], s["w"], axis)
        return getattr(api, op)(s["x"], axis)
    if kind == "chain":
        return api.rmsnorm_add_softmax_cast(s["x"], s["w"], s["r"])
    if kind == "matmul":
        return api.linear(s["a"], s["b"]) if c["form"] == "linear" else api.matmul(s["a"], s["b"])
    return api.scaledDotProductAttention(s["q"], s["k"], s["v"], c["d"] ** -0.5, mask=s.get("mask"), bias=s.get("bias"),
                                         causal=c["mask"] == "causal")


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _attend(q, k, v, scale, seen=None, bias=None, cap=0.0):
    """q [..., T, D], k [..., S, D], v [..., S, Dv], one head at a time."""
    out = torch.empty(*q.shape[:-1], v.shape[-1], dtype=torch.float64, device=q.device)
    for i in np.ndindex(*q.shape[:-2]):
        p = q[i] @ k[i].T * scale
        if cap:
            p = cap * torch.tanh(p / cap)
        if bias is not None:
            p = p + bias
        if seen is not None:
            p = p.masked_fill(~seen, -math.inf)
        out[i] = torch.softmax(p, -1) @ v[i]
    return out


def _causal(n, s, window=0):
    d = torch.arange(s - n, s, device="cuda")[:, None] - torch.arange(s, device="cuda")[None]
    return (d >= 0) & (d < window) if window else d >= 0


def _heads(x, n):  # [T, n * d] -> [n, T, d]
    return x.reshape(x.shape[0], n, -1).transpose(0, 1)


def _joined(x):
    return x.transpose(0, 1).reshape(x.shape[1], -1)


def _exact_qwen3(c, seed):
    cfg = _qwen3_config(c)
    shapes = _qwen3_shapes(cfg)

    def get(name, layer=None):
        key = name if layer is None else (name, layer)
        return _qwen3_weight(shapes[key], key, seed).double()

    ids = _ids(c, seed, cfg.vocab_size, c["batch"]).long()
    B, T = ids.shape
    H, G, D = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    embed = get("embed")
    x = embed[ids].reshape(B * T, -1)
    angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * cfg.rope_theta ** (
        -2.0 * torch.arange(D // 2, device="cuda", dtype=torch.float64) / D)
    cos, sin, seen = angle.cos(), angle.sin(), _causal(T, T)

    def turned(h, w):  # [B, n, T, D]
        h = _rms(h, w, cfg.rms_norm_eps)
        a, b = h[..., :D // 2], h[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    for l in range(cfg.num_hidden_layers):
        y = _rms(x, get("norm1", l), cfg.rms_norm_eps) @ get("qkv", l).T
        y = y.reshape(B, T, H + 2 * G, D).transpose(1, 2)
        q, k = turned(y[:, :H], get("q_norm", l)), turned(y[:, H:H + G], get("k_norm", l))
        o = _attend(q, k.repeat_interleave(H // G, 1), y[:, H + G:].repeat_interleave(H // G, 1), D ** -0.5, seen)
        x = x + o.transpose(1, 2).reshape(B * T, -1) @ get("o", l).T
        gate, up = (_rms(x, get("norm2", l), cfg.rms_norm_eps) @ get("gate_up", l).T).chunk(2, -1)
        x = x + (torch.nn.functional.silu(gate) * up) @ get("down", l).T
    x = _rms(x.reshape(B, T, -1)[:, c["prompt"] - 1:], get("norm"), cfg.rms_norm_eps)
    return [x[:, t] @ embed.T for t in range(c["steps"] + 1)]


def _mixture(get, p, h, x):
    logits = h @ get(p + "router").T
    score = torch.softmax(logits, -1)
    choice = score + get(p + "correction")
    per = choice.reshape(h.shape[0], x.groups, -1)
    keep = torch.zeros_like(per[..., 0]).scatter(1, per.amax(-1).topk(x.keep, -1).indices, 1.0)
    choice = per.masked_fill(keep[..., None] == 0, -math.inf).reshape(choice.shape)
    chosen = torch.zeros_like(choice).scatter(1, choice.topk(x.top, -1).indices, 1.0)
    out = torch.zeros_like(h)
    for e in range(choice.shape[1]):
        t = chosen[:, e].nonzero()[:, 0]
        s, n = score[t, e][:, None], f"{p}e{e}."
        if len(t) and e >= x.experts:
            out[t] += s * h[t]
        elif len(t):
            gated = torch.nn.functional.silu(h[t] @ get(n + "gate").T) * (h[t] @ get(n + "up").T)
            out[t] += s * (gated @ get(n + "down").T)
    return out


def _duzozen_mixer(get, p, h, x, first):
    q, k, own = (_heads(h @ get(p + n).T, m) for n, m in (("q", x.heads), ("k", x.kv_heads), ("v", x.kv_heads)))
    v = own
    if first is not None:
        lam = get(p + "vmix")
        v = (1 - lam) * own + lam * first
    r = x.heads // x.kv_heads
    T = h.shape[0]
    o = _attend(q, k.repeat_interleave(r, 0), v.repeat_interleave(r, 0), x.scale, _causal(T, T, x.window), None, x.softcap)
    return _joined(o) @ get(p + "o").T, own if first is None else first


def _derupel_mixer(get, p, h, x, eps):
    T = h.shape[0]
    gate = torch.sigmoid(h @ get(p + "g").T)
    if x.mixer == DECAYED:
        q, k, v = (_heads(torch.nn.functional.silu(h @ get(p + n).T), x.heads) for n in "qkv")
        o = torch.empty_like(v)
        d = (torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]).double()
        for i in range(x.heads):
            o[i] = (q[i] @ k[i].T * torch.where(d >= 0, x.decay[i] ** d.clamp(min=0), 0.0)) @ v[i]
        return (_rms(_joined(o), get(p + "norm"), eps) * gate) @ get(p + "o").T
    angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * x.rot_base ** (
        -2.0 * torch.arange(x.rot_dims // 2, device="cuda", dtype=torch.float64) / x.rot_dims)
    cos, sin = angle.cos(), angle.sin()

    def turned(a):  # [n, T, rot_dim], neighbouring pairs
        u, v = a[..., 0::2], a[..., 1::2]
        return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).reshape(a.shape)

    q = _heads(_rms(h @ get(p + "dq").T, get(p + "dq.norm"), eps) @ get(p + "uq").T, x.heads)
    kv = h @ get(p + "dkv").T
    c = _rms(kv[:, :x.kv_rank], get(p + "dkv.norm"), eps)
    key = turned(kv[None, :, x.kv_rank:]).expand(x.heads, -1, -1)
    q = torch.cat([q[..., :x.dim], turned(q[..., x.dim:])], -1)
    k = torch.cat([_heads(c @ get(p + "uk").T, x.heads), key], -1)
    o = _attend(q, k, _heads(c @ get(p + "uv").T, x.heads), x.scale, _causal(T, T))
    return (_joined(o) * gate) @ get(p + "o").T


def _exact_lm(c, seed):
    cfg = _lm_config(c)
    w = _Weights(cfg.tensor_shapes(), seed)
    get, eps, first = (lambda name: w[name].double()), cfg.eps, None
    ids = _ids(c, seed, cfg.vocab, 1)[0].long()
    derupel = c["model"] == "derupel"
    x = get("embed")[ids] * (cfg.embed_scale if derupel else 1.0)
    for i, layer in enumerate(cfg.layers):
        p = f"l{i}."
        if derupel:
            x = x + _rms(_derupel_mixer(get, p + "mix.", x, layer, eps), get(p + "norm1"), eps)
            h, behind = x, "norm2"
        else:
            o, first = _duzozen_mixer(get, p + "mix.", _rms(x, get(p + "norm1"), eps), layer, first)
            x = x + _rms(o, get(p + "norm1b"), eps)
            h, behind = _rms(x, get(p + "norm2"), eps), "norm2b"
        if layer.mlp == MLP_MOE:
            y = _mixture(get, p + "mlp.", h, layer)
        else:
            y = h @ get(p + "mlp.up").T
            y = (y.clamp(min=0) ** 2 if derupel else torch.nn.functional.gelu(y)) @ get(p + "mlp.down").T
        x = x + _rms(y, get(p + behind), eps)
    x, head = _rms(x, get("final.norm"), eps), get("head")
    return [x[_places(c)] @ head.T] + [x[c["prompt"] + t][None] @ head.T for t in range(c["steps"])]


def exact(case, seed):
    c, kind, op = case, case["kind"], case.get("op")
    if kind in ("qwen3", "lm"):
        return {"logits": (_exact_qwen3 if kind == "qwen3" else _exact_lm)(c, seed), "tokens": None}
    s = {k: v if v.dtype == torch.bool else v.double() for k, v in _operands(c, seed).items()}
    if kind == "matmul":
        return s["a"] @ (s["b"].transpose(-1, -2) if c["form"] == "linear" else s["b"])
    if kind == "attention":
        k, v = (s[n].repeat_interleave(c["groups"], 1) for n in "kv")
        seen = _causal(c["lq"], c["lk"]) if c["mask"] == "causal" else s.get("mask")
        return _attend(s["q"], k, v, c["d"] ** -0.5, seen, s.get("bias"))
    x = s["x"]
    if kind == "chain":
        return torch.softmax(_rms(x, s["w"], 1e-6) + s["r"], -1)
    if kind == "elementwise":
        if op == "swiglu":
            gate, up = x.chunk(2, -1)
            return gate * torch.sigmoid(gate) * up
        return {"add": lambda: x + s["y"], "mul": lambda: x * s["y"], "swish": lambda: x * torch.sigmoid(x),
                "gelu": lambda: torch.nn.functional.gelu(x, approximate="tanh"), "cast": lambda: x}[op]()
    if op in ("batchNorm", "groupNorm"):
        y = x if op == "batchNorm" else x.reshape(c["n"], 8, -1)
        axes = (0, 2, 3) if op == "batchNorm" else (2,)
        y = (y - y.mean(axes, keepdim=True)) / torch.sqrt(y.var(axes, unbiased=False, keepdim=True) + 1e-5)
        return y.reshape(x.shape) * s["w"][:, None, None] + s["b"][:, None, None]
    axis = c["axis"] - 2
    if op == "rmsNorm":
        return _rms(x, s["w"], 1e-5)
    if op == "layerNorm":
        y = (x - x.mean(axis, keepdim=True)) / torch.sqrt(x.var(axis, unbiased=False, keepdim=True) + 1e-5)
        shape = (-1, 1) if axis == 0 else (1, -1)
        return y * s["w"].reshape(shape) + s["b"].reshape(shape)
    if op == "max":
        best, at = x.max(axis, keepdim=True)
        return best, at
    return torch.softmax(x, axis) if op == "softmax" else getattr(x, op)(axis, keepdim=True)


# ---------------------------------------------------------------------------------------------- work and tolerance
def _lm_macs(cfg, length):
    """Multiply-adds per token of the matrices that a token goes through, their bytes (every expert where `length` tokens
    choose among them), and the multiply-adds of the mixers over `length` tokens."""
    W, macs, nbytes, mix = cfg.width, 0, 0, 0.0
    for x in cfg.layers:
        m = 0
        if isinstance(x, DerupelLayer):
            m += 2 * W * x.heads * x.vdim
            if x.mixer == LATENT:
                m += W * (x.q_rank + x.kv_rank + x.rot_dim) + x.q_rank * x.heads * (x.dim + x.rot_dim)
                m += x.kv_rank * x.heads * (x.dim + x.vdim)
                mix += x.heads * (x.dim + x.rot_dim + x.vdim) * length * length / 2
            else:
                m += W * x.heads * (2 * x.dim + x.vdim)
                mix += 2 * length * x.heads * x.dim * x.vdim
        else:
            m += W * (x.heads + x.kv_heads) * (x.dim + x.vdim)
            span = min(length, x.window or length)
            mix += x.heads * (x.dim + x.vdim) * (length * span - span * span / 2)
        macs, nbytes = macs + m, nbytes + 2 * m
        if x.mlp == MLP_DENSE:
            macs, nbytes = macs + 2 * W * x.ff, nbytes + 4 * W * x.ff
        else:
            routes, each = x.experts + x.identity, 3 * W * x.ff
            macs += x.top * x.experts / routes * each + routes * W
            nbytes += 2 * (min(x.experts, length * x.top) * each + routes * W)
    return macs, nbytes, mix


def work(case):
    c, kind = case, case["kind"]
    n = SIZE[c.get("dtype", "f32")]
    if kind == "elementwise":
        e = c["rows"] * c["cols"]
        more = {"add": c["cols"] * n, "mul": e * n, "swiglu": e * n}.get(c["op"], 0)
        return {"bytes": e * (n + (2 if c["op"] == "cast" else n)) + more, "flops": e}
    if kind == "rows":
        e = c["n"] * c["c"] * c["h"] * c["w"]
        return {"bytes": e * n * (1 if c["op"] in ("sum", "mean", "max") else 2), "flops": e * 4}
    if kind == "chain":
        row = c["l"] * c["h"]
        return {"bytes": row * (6 * c["b"] + 4 * (c["b"] if c["residual"] == "own" else 1)), "flops": 10 * row * c["b"]}
    if kind == "matmul":
        b, m, k, j = c["batch"], c["m"], c["k"], c["n"]
        return {"bytes": n * (b * m * (k + j) + k * j * (b if c["form"] == "batched" else 1)), "flops": 2 * b * m * k * j}
    if kind == "attention":
        heads = c["b"] * c["kv"] * c["groups"]
        pairs = c["lq"] * c["lk"]
        nbytes = n * c["d"] * (2 * heads * c["lq"] + 2 * c["b"] * c["kv"] * c["lk"])
        nbytes += pairs * {"bool": 1, "bias": 4}.get(c["mask"], 0)
        if c["mask"] == "causal":
            pairs = c["lq"] * (c["lk"] - (c["lq"] - 1) / 2)
        return {"bytes": nbytes, "flops": 4 * heads * pairs * c["d"]}
    if kind == "qwen3":
        cfg, B, P, S = _qwen3_config(c), c["batch"], c["prompt"], c["steps"]
        layers, vocab = 28 * 15728640, cfg.vocab_size * cfg.hidden_size
        keys = 28 * 2 * cfg.num_key_value_heads * cfg.head_dim * 4
        flops = 2 * B * ((P + S) * layers + (1 + S) * vocab) + 28 * 4 * B * 16 * 128 * (P + S) ** 2 / 2
        nbytes = (1 + S) * 2 * (layers + vocab) + B * keys * (P + S + S * (P + S / 2)) + 4 * B * (1 + S) * cfg.vocab_size
        return {"bytes": nbytes, "flops": flops}
    cfg, P, S = _lm_config(c), c["prompt"], c["steps"]
    macs, once, mix = _lm_macs(cfg, P + S)
    _, step, _ = _lm_macs(cfg, 1)
    head = cfg.width * cfg.vocab
    return {"bytes": once + S * step + 2 * head * (1 + S) + 4 * cfg.vocab * (len(_places(c)) + S),
            "flops": 2 * ((P + S) * macs + mix + head * (len(_places(c)) + S))}


def tolerance(case):
    """About four times what the path was measured to be off `exact()`, or what its number format rounds to."""
    kind, op, dt = case["kind"], case.get("op"), case.get("dtype", "f32")
    if kind == "lm":  # bf16 activations; with experts a near tie of a router decides otherwise now and then
        return {"rel": 0.03, "max": 0.5, "differ": 0.01}
    if kind == "qwen3":  # activations enter the products as two bf16 numbers, 16 mantissa bits
        return {"rel": 5e-5, "max": 2e-3, "differ": 0.01}
    if op in ("add", "mul", "cast", "max"):
        return "exact"
    if kind == "chain" or dt == "bf16":
        return {"rel": 1e-2, "max": 4e-2}
    return {"rel": 5e-6, "max": 1e-4} if dt == "f32" else {"rel": 1e-3, "max": 1e-2}
