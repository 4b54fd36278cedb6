"""What the speed of this package is measured on.

Each case is one call of a public entry point as a program makes it: the matrix products of a decoder's linear layers
(a decode step's few rows, a batch of rows, a training-sized square), the integer product profiles with the activations
quantised in the call, the host-array call of `linalg`, one decoder block (prompt and decode step), and a whole greedy
continuation. The package's contract is bit identity, so every case's tolerance is "exact".

`listed()` are the fixed cases, `draw(rng)` gives others of the same ranges.
"""
import math

import numpy as np
import torch

from mojolearn_b200 import linalg, torch_ops
from mojolearn_b200.linalg import W_BF16, W_F32, W_INT8_EXP
from mojolearn_b200.models import CausalLM, CausalLMConfig
from mojolearn_b200.transformer import Linear, TransformerBlock

DEV = "cuda"
KINDS = {"float32": W_F32, "bfloat16": W_BF16, "int8": W_INT8_EXP}
BYTES = {"float32": 4, "bfloat16": 2, "int8": 1}


def listed():
    return [
        # one token through one MLP projection of a 7B-shaped decoder: the smallest call of a serving loop
        {"name": "row_int8", "path": "linear", "m": 1, "n": 11008, "k": 4096, "weight": "int8"},
        # a small decode batch on bfloat16 weights
        {"name": "rows8_bf16", "path": "linear", "m": 8, "n": 11008, "k": 4096, "weight": "bfloat16"},
        # a full decode batch on int8 weights
        {"name": "rows32_int8", "path": "linear", "m": 32, "n": 11008, "k": 4096, "weight": "int8"},
        # a short prompt's or a small training batch's rows through the same projection in float32
        {"name": "batch128_f32", "path": "matmul", "op": "NT", "m": 128, "n": 11008, "k": 4096},
        # a general product whose sides fit no tile
        {"name": "square1000_f32", "path": "matmul", "op": "NN", "m": 1000, "n": 1000, "k": 1000},
        # a large product: a long prompt or a training step's projection
        {"name": "square4096_f32", "path": "matmul", "op": "NT", "m": 4096, "n": 4096, "k": 4096},
        # the Gram matrix of a tall data set (covariance, normal equations): a million rows contracted
        {"name": "gram_f32", "path": "matmul", "op": "TN", "m": 32, "n": 32, "k": 1000000},
        # a linear layer in the integer profile: float32 activations quantised in the call, weight codes kept
        {"name": "int8_layer", "path": "int8_layer", "m": 4096, "n": 4096, "k": 4096},
        # host arrays in, host array out, as the numpy surface is called
        {"name": "host_f32", "path": "host", "m": 512, "n": 4096, "k": 4096},
        # a prompt through one block of the serving model, int8 weights
        {"name": "block_prompt", "path": "block", "batch": 4, "length": 1024, "cached": 0, "d": 2048, "heads": 16, "mlp": 8192,
         "weight": "int8"},
        # one decode step of that block at the serving batch and cache length
        {"name": "block_step", "path": "block", "batch": 32, "length": 1, "cached": 1100, "d": 2048, "heads": 16, "mlp": 8192,
         "weight": "int8"},
        # a prompt and its greedy continuation through a whole small model in float32
        {"name": "generate", "path": "generate", "batch": 8, "prompt": 512, "new": 128, "layers": 12, "d": 768, "heads": 12,
         "mlp": 3072, "vocab": 50304},
    ]


def _span(rng, lo, hi):
    """A size spread over the logarithm of its range; every second one is whatever comes, the others a multiple of 16."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return v if rng.random() < 0.5 else min(hi, max(lo, (v + 8) // 16 * 16))


def draw(rng):
    path = rng.choice(["linear", "linear", "linear", "matmul", "matmul", "gram", "int8_layer", "host", "block", "step",
                       "generate"])
    if path == "linear":
        return {"path": "linear", "m": _span(rng, 1, 48) if rng.random() < 0.7 else rng.choice([1, 1, 2, 4]),
                "n": _span(rng, 768, 50304), "k": 16 * rng.randint(48, 512) if rng.random() < 0.8 else rng.randint(768, 8192),
                "weight": rng.choice(["int8", "int8", "bfloat16", "float32"])}
    if path == "matmul":
        return {"path": "matmul", "op": rng.choice(["NN", "NT", "TN"]), "m": _span(rng, 48, 4096), "n": _span(rng, 128, 4096),
                "k": _span(rng, 128, 4096)}
    if path == "gram":
        side = _span(rng, 16, 96)
        return {"path": "matmul", "op": "TN", "m": side, "n": side, "k": _span(rng, 20000, 1000000)}
    if path == "int8_layer":
        return {"path": path, "m": _span(rng, 32, 4096), "n": _span(rng, 768, 8192),
                "k": 16 * rng.randint(48, 256) if rng.random() < 0.9 else rng.randint(64, 768)}
    if path == "host":
        return {"path": "host", "m": _span(rng, 16, 1024), "n": _span(rng, 128, 4096), "k": _span(rng, 128, 4096)}
    d, heads, mlp = rng.choice([(512, 8, 2048), (768, 12, 3072), (1024, 16, 2816), (2048, 16, 8192)])
    weight = rng.choice(["int8", "int8", "bfloat16", "float32"])
    if path == "block":
        return {"path": "block", "batch": rng.randint(1, 4), "length": _span(rng, 32, 1024), "cached": 0, "d": d, "heads": heads,
                "mlp": mlp, "weight": weight}
    if path == "step":
        return {"path": "block", "batch": _span(rng, 1, 32), "length": 1, "cached": _span(rng, 16, 1279), "d": d, "heads": heads,
                "mlp": mlp, "weight": weight}
    return {"path": "generate", "batch": rng.randint(1, 8), "prompt": _span(rng, 16, 512), "new": rng.randint(8, 96),
            "layers": rng.randint(2, 8), "d": 768, "heads": 12, "mlp": 3072, "vocab": rng.choice([8192, 32000, 50304])}


# ---- inputs --------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(gen, *shape, scale=1.0):
    return torch.randn(shape, generator=gen, device=DEV).mul_(scale)


def _weight(gen, n, k, kind):
    """(storage, exponents or None) of an [n, k] weight, entries of about 0.02."""
    if kind == "int8":
        codes = torch.randint(-127, 128, (n, k), generator=gen, device=DEV, dtype=torch.int8)
        return codes, torch.randint(-13, -10, (n,), generator=gen, device=DEV, dtype=torch.int32)
    w = _normal(gen, n, k, scale=0.02)
    return (w.to(torch.bfloat16).view(torch.uint16), None) if kind == "bfloat16" else (w, None)


def _block_inputs(c, seed):
    """The tensors of a block case: weights by name, the new tokens' rows, and the cached keys and values."""
    g, d, hd = _gen(seed), c["d"], c["d"] // c["heads"]
    w = {"input_layernorm.weight": 1 + _normal(g, d, scale=0.1), "post_attention_layernorm.weight": 1 + _normal(g, d, scale=0.1)}
    for name, n, k in (("q_proj", d, d), ("k_proj", d, d), ("v_proj", d, d), ("o_proj", d, d), ("gate_proj", c["mlp"], d),
                       ("up_proj", c["mlp"], d), ("down_proj", d, c["mlp"])):
        w[name + ".weight"] = _weight(g, n, k, c["weight"])
    x = _normal(g, c["batch"], c["length"], d)
    past = [_normal(g, c["batch"], c["heads"], c["cached"], hd) for _ in range(2)] if c["cached"] else None
    return w, x, past


def _lm_inputs(c, seed):
    g, d, it = _gen(seed), c["d"], c["mlp"]
    w = {"model.embed_tokens.weight": _normal(g, c["vocab"], d, scale=0.02), "model.norm.weight": 1 + _normal(g, d, scale=0.1),
         "lm_head.weight": _normal(g, c["vocab"], d, scale=0.02)}
    for i in range(c["layers"]):
        p = "model.layers.%d." % i
        for name in ("input_layernorm.weight", "post_attention_layernorm.weight"):
            w[p + name] = 1 + _normal(g, d, scale=0.1)
        for name, n, k in (("self_attn.q_proj", d, d), ("self_attn.k_proj", d, d), ("self_attn.v_proj", d, d),
                           ("self_attn.o_proj", d, d), ("mlp.up_proj", it, d), ("mlp.down_proj", d, it)):
            w[p + name + ".weight"] = _normal(g, n, k, scale=0.02)
    ids = torch.randint(0, c["vocab"], (c["batch"], c["prompt"]), generator=g, device=DEV, dtype=torch.int32)
    return w, ids


def _product_inputs(c, seed):
    g, m, n, k = _gen(seed), c["m"], c["n"], c["k"]
    if c["path"] == "linear":
        return _normal(g, m, k), _weight(g, n, k, c["weight"])
    op = c.get("op", "NT")
    return _normal(g, *((k, m) if op == "TN" else (m, k))), _normal(g, *((n, k) if op == "NT" else (k, n)))


def prepare(c, seed):
    path = c["path"]
    if path == "block":
        w, x, past = _block_inputs(c, seed)
        w = {name: Linear.from_device(t[0], t[1], KINDS[c["weight"]]) if isinstance(t, tuple) else t for name, t in w.items()}
        block = TransformerBlock(w, n_heads=c["heads"])
        cache = block.allocate_state(c["batch"], c["cached"] + c["length"])
        if past is not None:
            cache.k[:, :, :c["cached"]] = past[0]
            cache.v[:, :, :c["cached"]] = past[1]
        return {"case": c, "block": block, "x": x, "cache": cache}
    if path == "generate":
        w, ids = _lm_inputs(c, seed)
        cfg = CausalLMConfig(vocab=c["vocab"], d_model=c["d"], n_layers=c["layers"], n_heads=c["heads"], intermediate=c["mlp"],
                             mlp="gelu", max_positions=2048)
        return {"case": c, "lm": CausalLM(cfg, w), "ids": ids}
    a, b = _product_inputs(c, seed)
    if path == "host":
        return {"case": c, "a": a.cpu().numpy(), "b": b.cpu().numpy()}
    if path == "int8_layer":
        b = torch_ops.quantize_int8(b)
    return {"case": c, "a": a, "b": b}


def run(s):
    c = s["case"]
    path = c["path"]
    if path == "linear":
        w, e = s["b"]
        if c["weight"] == "int8":
            return torch_ops.linear_int8w(s["a"], w, e)
        if c["weight"] == "bfloat16":
            return torch_ops.matmul_bf16(s["a"], w, transpose_b=True)
        return torch_ops.matmul(s["a"], w, transpose_b=True)
    if path == "matmul":
        return torch_ops.matmul(s["a"], s["b"], transpose_a=c["op"] == "TN", transpose_b=c["op"] == "NT")
    if path == "int8_layer":
        qa, ea = torch_ops.quantize_int8(s["a"])
        return torch_ops.matmul_int8(qa, ea, *s["b"])
    if path == "host":
        return linalg.matmul(s["a"], s["b"], transpose_b=True)
    if path == "block":
        cache = s["cache"]
        cache.cached_tokens = c["cached"]  # the same call again: the new tokens' slots are written anew
        y = s["block"].step(s["x"], cache) if c["length"] == 1 and c["cached"] else s["block"].forward(s["x"], cache)
        return {"y": y, "k": cache.k, "v": cache.v}
    ids, logits = s["lm"].generate(s["ids"], c["new"], return_logits=True)
    return {"ids": ids, "logits": logits}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def work(c):
    path = c["path"]
    if path == "block":
        d, mlp, b, l, used = c["d"], c["mlp"], c["batch"], c["length"], c["cached"] + c["length"]
        weights = 4 * d * d + 3 * d * mlp
        pairs = b * sum(c["cached"] + i + 1 for i in range(l))  # (query, visible key) pairs of one head
        return {"bytes": weights * BYTES[c["weight"]] + 4 * (2 * b * l * d) + 4 * 2 * b * used * d,
                "flops": 2 * b * l * weights + 4 * pairs * d}
    if path == "generate":
        d, b = c["d"], c["batch"]
        layer = 4 * d * d + 2 * d * c["mlp"]
        weights = c["layers"] * layer + c["vocab"] * d
        rows = b * (c["prompt"] + c["new"] - 1)
        pairs = b * sum(i + 1 for i in range(c["prompt"] + c["new"] - 1))
        kv = 4 * 2 * b * d * c["layers"] * sum(c["prompt"] + i for i in range(c["new"]))
        return {"bytes": 4 * weights * c["new"] + kv + 4 * b * c["new"] * c["vocab"],
                "flops": 2 * rows * c["layers"] * layer + 2 * b * c["new"] * c["vocab"] * d + 4 * pairs * d * c["layers"]}
    m, n, k = c["m"], c["n"], c["k"]
    wbytes = {"linear": BYTES.get(c.get("weight"), 4), "int8_layer": 1}.get(path, 4)
    extra = 4 * n if path == "int8_layer" or c.get("weight") == "int8" else 0
    return {"bytes": m * k * 4 + n * k * wbytes + extra + 4 * m * n, "flops": 2 * m * n * k}


def tolerance(c):
    """Every output is pinned to the bit by the package's numerical contract."""
    return "exact"


# ---- the same in 64 bits, in plain torch ---------------------------------------------------------------------------

def _pow2(e):
    """2 ** e of whole numbers, exact (a power function may be an ulp off, which would break ties)."""
    return ((e.long() + 1023) << 52).view(torch.float64)


def _wide(t):
    """A weight's value in 64 bits."""
    w, e = t if isinstance(t, tuple) else (t, None)
    if w.dtype == torch.uint16:
        w = w.view(torch.bfloat16)
    return w.double() * _pow2(e)[:, None] if e is not None else w.double()


def _codes(x):
    """Rows as seven-bit codes times a power of two."""
    x = x.double()
    _, ex = torch.frexp(x.abs().amax(dim=1, keepdim=True))
    step = _pow2(ex - 7)
    return torch.clamp(torch.round(x / step), -127, 127) * step


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w


def _rotate(x, positions):
    half = x.shape[-1] // 2
    inv = 10000.0 ** (-torch.arange(half, device=DEV, dtype=torch.float64) / half)
    ang = positions.double()[:, None] * inv
    cos, sin = ang.cos(), ang.sin()
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _attend(q, k, v, first):
    """Causal attention of [B, H, L, hd] queries at positions first.. over all keys, a sequence at a time."""
    out = []
    qpos = first + torch.arange(q.shape[2], device=DEV)
    hidden = torch.arange(k.shape[2], device=DEV)[None, :] > qpos[:, None]
    for i in range(q.shape[0]):
        s = (q[i] @ k[i].transpose(-1, -2)) / math.sqrt(q.shape[-1])
        out.append(torch.softmax(s.masked_fill(hidden, float("-inf")), dim=-1) @ v[i])
    return torch.stack(out)


def _decoder(x, w, heads, past, gated):
    """One block in 64 bits: (y, keys, values), keys and values of all positions."""
    b, l, d = x.shape
    hd = d // heads
    first = past[0].shape[2] if past is not None else 0
    split = lambda t: t.reshape(b, l, heads, hd).transpose(1, 2)  # noqa: E731
    h = _rms(x, w["input_layernorm.weight"].double())
    q, k, v = (split(h @ _wide(w[n + "_proj.weight"]).T) for n in "qkv")
    pos = first + torch.arange(l, device=DEV)
    q, k = _rotate(q, pos), _rotate(k, pos)
    if past is not None:
        k, v = torch.cat([past[0].double(), k], dim=2), torch.cat([past[1].double(), v], dim=2)
    ctx = _attend(q, k, v, first).transpose(1, 2).reshape(b, l, d)
    r = x + ctx @ _wide(w["o_proj.weight"]).T
    h = _rms(r, w["post_attention_layernorm.weight"].double())
    up = h @ _wide(w["up_proj.weight"]).T
    act = torch.nn.functional.silu(h @ _wide(w["gate_proj.weight"]).T) * up if gated else torch.nn.functional.gelu(up)
    return r + act @ _wide(w["down_proj.weight"]).T, k, v


def exact(c, seed):
    path = c["path"]
    if path == "block":
        w, x, past = _block_inputs(c, seed)
        y, k, v = _decoder(x.double(), w, c["heads"], past, True)
        return {"y": y, "k": k, "v": v}
    if path == "generate":
        w, ids = _lm_inputs(c, seed)
        layers = [{n.split(".")[-2] + ".weight": t for n, t in w.items() if n.startswith("model.layers.%d." % i)}
                  for i in range(c["layers"])]
        logits, past = [], [None] * c["layers"]
        new = ids.long()
        for _ in range(c["new"]):
            h = w["model.embed_tokens.weight"][new].double()
            for i, lw in enumerate(layers):
                h, k, v = _decoder(h, lw, c["heads"], past[i], False)
                past[i] = (k, v)
            logits.append(_rms(h[:, -1], w["model.norm.weight"].double()) @ w["lm_head.weight"].double().T)
            new = logits[-1].argmax(dim=-1, keepdim=True)
        return {"ids": None, "logits": torch.stack(logits, dim=1)}
    a, b = _product_inputs(c, seed)
    if path == "linear":
        return a.double() @ _wide(b).T
    if path == "int8_layer":
        return _codes(a) @ _codes(b).T
    op = c.get("op", "NT")
    out = (a.double().T if op == "TN" else a.double()) @ (b.double().T if op == "NT" else b.double())
    return out.cpu().numpy() if path == "host" else out
