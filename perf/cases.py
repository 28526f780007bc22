"""The work that programs built on this package have it do, as cases that can be timed.

Every case goes through a public entry point (the kernel classes, `triton_attn_func` /
`flash_attn_func`, the int8 functions, `Int8DecoderLayer`) with the tensors such a program has
in hand. `listed()` are the fixed cases, `draw()` gives others of the same ranges, `exact()` is
the same arithmetic as plain torch has it in 64 bits, without this package.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import trinix_b200 as T
from trinix_b200.decoder import Int8DecoderLayer
from trinix_b200.functional import flash_attn_func

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}
EPS = 1e-6

# The largest listed memory-bound case moves about 1.8 GB; a drawn one stays below it.
MOST_BYTES = 1_500_000_000
# The largest listed attention case has 2.2e12 operations.
MOST_FLOPS = 2_000_000_000_000


def listed():
    return [
        # A norm of a small model on a short batch: nothing but call and launch latency.
        norm_case("rmsnorm", 512, 768, "f32", False, name="rmsnorm_small"),
        # Training a 4096-wide model: one LayerNorm, forward and backward, on 32768 tokens.
        norm_case("layernorm", 32768, 4096, "bf16", True, name="layernorm_train"),
        # Training with a fused residual norm at a width that is no power of two, ragged rows.
        norm_case("residual_rmsnorm", 2999, 3000, "f16", True, name="residual_rmsnorm_train"),
        # Storing and loading activations or weights as per-row int8.
        {"name": "int8_roundtrip", "op": "int8", "rows": 8192, "cols": 4096, "dtype": "bf16"},
        # The norm in front of an int8 GEMM on 32768 tokens.
        {"name": "rmsnorm_int8", "op": "norm_int8", "rows": 32768, "cols": 4096, "dtype": "bf16"},
        # Rotary embedding of the queries and grouped keys of a prefill.
        {"name": "rope_prefill", "op": "rope", "batch": 8, "seq": 2048, "heads": 32, "kv_heads": 8,
         "dim": 128, "dtype": "bf16"},
        # The gated activation of an MLP in training, forward and backward.
        glu_case("swiglu", 16384, 11008, "bf16", True, name="swiglu_train"),
        # The prefill of a grouped-query model: the largest call.
        attn_case("causal", 16, 4096, 4096, 32, 8, 128, "bf16", name="attn_prefill"),
        # Sliding-window prefill of a ragged length.
        attn_case("window", 4, 3001, 3001, 32, 8, 128, "bf16", window=1024, name="attn_window"),
        # An encoder over a padded batch: no causal order, an additive mask, head dim 64.
        attn_case("full", 8, 509, 509, 16, 16, 64, "f16", mask=True, name="attn_encoder_masked"),
        # One decoding step against a KV cache.
        attn_case("decode", 16, 1, 4093, 32, 8, 128, "bf16", name="attn_decode"),
        # A whole decoder layer with int8 weights on four sequences.
        {"name": "decoder_layer", "op": "layer", "batch": 4, "seq": 2048, "embed": 4096,
         "heads": 32, "kv_heads": 8, "ffn": 11008},
    ]


# ------------------------------------------------------------------------------ kinds of case
NORMS = ("rmsnorm", "layernorm", "residual_rmsnorm", "residual_layernorm", "rmsnorm_mish")
GLUS = ("swiglu", "geglu", "reglu")


def norm_case(kind, rows, cols, dtype, train, **more):
    return {"op": "norm", "kind": kind, "rows": rows, "cols": cols, "dtype": dtype, "train": train,
            **more}


def glu_case(kind, rows, hidden, dtype, train, **more):
    return {"op": "glu", "kind": kind, "rows": rows, "hidden": hidden, "dtype": dtype,
            "train": train, **more}


def attn_case(kind, batch, seq_q, seq_k, heads, kv_heads, dim, dtype, **more):
    """kind: "causal", "alibi" (causal with slopes), "window" (the last `window` keys), "full",
    "decode" (the last seq_q rows of a causal order over seq_k keys)."""
    return {"op": "attn", "kind": kind, "batch": batch, "seq_q": seq_q, "seq_k": seq_k,
            "heads": heads, "kv_heads": kv_heads, "dim": dim, "dtype": dtype, **more}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A feature width: mostly a multiple of 128, often of 8, now and then an odd one."""
    n = _log(rng, lo, hi)
    r = rng.random()
    step = 128 if r < 0.55 else 8 if r < 0.9 else 1
    return max(step, n // step * step)


def _rows(rng, row_bytes):
    """Token counts from one sequence's last token to a large batch."""
    return _log(rng, 1, max(2, min(65536, MOST_BYTES // row_bytes)))


def draw(rng):
    op = rng.choice(["norm", "norm", "int8", "norm_int8", "rope", "glu", "attn", "attn", "attn",
                     "decode", "layer"])
    if op == "norm":
        dtype, cols, train = rng.choice(["bf16", "bf16", "f16", "f32"]), _width(rng, 256, 12288), \
            rng.random() < 0.5
        return norm_case(rng.choice(NORMS), _rows(rng, 7 * cols * SIZE[dtype]), cols, dtype, train)
    if op in ("int8", "norm_int8"):
        dtype, cols = rng.choice(["bf16", "bf16", "f16", "f32"]), _width(rng, 256, 12288)
        return {"op": op, "rows": _rows(rng, 5 * cols * SIZE[dtype]), "cols": cols, "dtype": dtype}
    if op == "glu":
        dtype, hidden, train = rng.choice(["bf16", "bf16", "f16", "f32"]), \
            _width(rng, 512, 16384), rng.random() < 0.5
        return glu_case(rng.choice(GLUS), _rows(rng, 8 * hidden * SIZE[dtype]), hidden, dtype,
                        train)
    if op == "rope":
        heads, dim = rng.choice([8, 12, 16, 32, 40]), rng.choice([64, 80, 128, 128])
        kv_heads = rng.choice([h for h in (1, 2, 4, 8, heads) if heads % h == 0])
        dtype, batch = rng.choice(["bf16", "f16", "f32"]), rng.choice([1, 2, 4, 8])
        row = 2 * batch * (heads + kv_heads) * dim * SIZE[dtype]
        return {"op": op, "batch": batch, "seq": _log(rng, 1, min(16384, MOST_BYTES // row)),
                "heads": heads, "kv_heads": kv_heads, "dim": dim, "dtype": dtype}
    if op == "layer":
        embed = rng.choice([2048, 3072, 4096])
        heads = embed // 128
        return {"op": op, "batch": rng.choice([1, 2, 4]), "seq": _log(rng, 64, 2048),
                "embed": embed, "heads": heads,
                "kv_heads": rng.choice([4, 8]),
                "ffn": embed * 11 // 4 // 128 * 128}
    heads, dim = rng.choice([8, 12, 16, 32]), rng.choice([64, 128, 128])
    kv_heads = rng.choice([h for h in (1, 2, 4, 8, heads) if heads % h == 0])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    if op == "decode":
        batch, seq_q = _log(rng, 1, 64), rng.choice([1, 1, 1, 2, 5, 16])
        longest = min(32768, MOST_BYTES // (4 * batch * kv_heads * dim))
        return attn_case("decode", batch, seq_q, _log(rng, 64, longest), heads, kv_heads, dim,
                         dtype)
    kind = rng.choice(["causal", "causal", "alibi", "window", "full", "full"])
    batch = rng.choice([1, 2, 4, 8, 16])
    seq = _log(rng, 64, min(8192, math.isqrt(MOST_FLOPS // (4 * batch * heads * dim))))
    more = {}
    if kind == "window":
        more["window"] = max(16, _log(rng, 16, max(17, seq // 2)))
    if kind == "full" and seq <= 2048:
        more["mask"] = rng.random() < 0.5
    return attn_case(kind, batch, seq, seq, heads, kv_heads, dim, dtype, **more)


# --------------------------------------------------------------------------------- the inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _randn(g, *shape, dtype=torch.float32, std=1.0, mean=0.0):
    t = torch.randn(*shape, generator=g, device=DEV)
    if std != 1.0 or mean != 0.0:
        t.mul_(std).add_(mean)
    return t.to(dtype)


def _with_outliers(g, x):
    """0.1 % of the entries twenty times as large, as activations in front of an int8 GEMM are."""
    hit = torch.rand(x.shape, generator=g, device=DEV) < 1e-3
    return torch.where(hit, x * 20, x)


def _rope_tables(seq, dim):
    inv = 1.0 / 10000.0 ** (torch.arange(0, dim, 2, device=DEV, dtype=torch.float32) / dim)
    a = torch.outer(torch.arange(seq, device=DEV, dtype=torch.float32), inv)
    a = torch.cat((a, a), dim=-1)
    return a.cos(), a.sin()


def _padding_mask(c):
    """An additive (B, 1, Sq, Sk) mask: sequence b keeps between half and all of its keys."""
    b, sk = c["batch"], c["seq_k"]
    keep = sk - (torch.arange(b, device=DEV) * 37) % max(1, sk // 2)
    hidden = torch.arange(sk, device=DEV)[None] >= keep[:, None]
    m = torch.zeros(b, 1, c["seq_q"], sk, device=DEV)
    return m.masked_fill_(hidden[:, None, None, :], float("-inf"))


def _inputs(c, seed):
    """The tensors of a case, by name: the same for `prepare` and `exact`."""
    g = _gen(seed)
    if c["op"] == "norm":
        dt, shape = DTYPES[c["dtype"]], (c["rows"], c["cols"])
        d = {"x": _randn(g, *shape, dtype=dt),
             "w": _randn(g, c["cols"], dtype=dt, std=0.02, mean=1.0)}
        if "residual" in c["kind"]:
            d["r"] = _randn(g, *shape, dtype=dt)
        if "layernorm" in c["kind"]:
            d["b"] = _randn(g, c["cols"], dtype=dt, std=0.02)
        if c["train"]:
            d["dy"] = _randn(g, *shape, dtype=dt)
        return d
    if c["op"] in ("int8", "norm_int8"):
        dt = DTYPES[c["dtype"]]
        x = _randn(g, c["rows"], c["cols"])
        if c["op"] == "int8":
            return {"x": _with_outliers(g, x).to(dt)}
        return {"x": x.to(dt), "w": _randn(g, c["cols"], dtype=dt, std=0.02, mean=1.0)}
    if c["op"] == "rope":
        dt, lead = DTYPES[c["dtype"]], (c["batch"], c["seq"])
        cos, sin = _rope_tables(c["seq"], c["dim"])
        return {"q": _randn(g, *lead, c["heads"], c["dim"], dtype=dt),
                "k": _randn(g, *lead, c["kv_heads"], c["dim"], dtype=dt), "cos": cos, "sin": sin}
    if c["op"] == "glu":
        dt = DTYPES[c["dtype"]]
        d = {"x": _randn(g, c["rows"], 2 * c["hidden"], dtype=dt)}
        if c["train"]:
            d["dy"] = _randn(g, c["rows"], c["hidden"], dtype=dt)
        return d
    if c["op"] == "attn":
        dt, b, dim = DTYPES[c["dtype"]], c["batch"], c["dim"]
        d = {"q": _randn(g, b, c["seq_q"], c["heads"], dim, dtype=dt),
             "k": _randn(g, b, c["seq_k"], c["kv_heads"], dim, dtype=dt),
             "v": _randn(g, b, c["seq_k"], c["kv_heads"], dim, dtype=dt)}
        if c["kind"] == "alibi":
            d["slopes"] = 2.0 ** (-8.0 * torch.arange(1, c["heads"] + 1, device=DEV) / c["heads"])
        if c.get("mask"):
            d["mask"] = _padding_mask(c)
        return d
    e, f, kv = c["embed"], c["ffn"], c["kv_heads"] * (c["embed"] // c["heads"])
    shapes = {"wq": (e, e), "wk": (kv, e), "wv": (kv, e), "wo": (e, e), "w_up": (f, e),
              "w_gate": (f, e), "w_down": (e, f)}
    return {"x": _randn(g, c["batch"], c["seq"], e, dtype=torch.bfloat16),
            "weights": {n: _randn(g, *s, dtype=torch.bfloat16, std=0.02)
                        for n, s in shapes.items()}}


def prepare(case, seed):
    s = _inputs(case, seed)
    if case["op"] == "layer":
        s["layer"] = Int8DecoderLayer(case["embed"], case["heads"], case["kv_heads"], case["ffn"],
                                      s.pop("weights"), max_seq_len=max(2048, case["seq"]))
    if case.get("train"):
        for n in ("x", "r", "w", "b"):
            if n in s:
                s[n].requires_grad_()
    return {"case": dict(case), **s}


# --------------------------------------------------------------------------------- the passes
GLU_KERNELS = {"swiglu": T.TritonSwiGLUKernel, "geglu": T.TritonGeGLUKernel,
               "reglu": T.TritonReGLUKernel}


def _norm_forward(c, s):
    if c["kind"] == "rmsnorm":
        return T.TritonRMSNormKernel.apply(s["x"], s["w"], EPS)
    if c["kind"] == "layernorm":
        return T.TritonLayerNormKernel.apply(s["x"], s["w"], s["b"], EPS)
    if c["kind"] == "residual_rmsnorm":
        return T.TritonFusedResidualRMSNormKernel.apply(s["x"], s["r"], s["w"], EPS)
    if c["kind"] == "residual_layernorm":
        return T.TritonFusedResidualLayerNormKernel.apply(s["x"], s["r"], s["w"], s["b"], EPS)
    return T.TritonFusedRMSNormActivationKernel.apply(s["x"], s["w"], EPS, "mish")


def _with_grads(y, s):
    """y and the gradients of the inputs, as a training step has them."""
    names = [n for n in ("x", "r", "w", "b") if n in s]
    grads = torch.autograd.grad(y, [s[n] for n in names], s["dy"])
    return {"y": y, **{"d" + n: g for n, g in zip(names, grads)}}


def run(state):
    c, s = state["case"], state
    if c["op"] == "norm":
        y = _norm_forward(c, s)
        return _with_grads(y, s) if c["train"] else {"y": y}
    if c["op"] == "int8":
        codes, scales = T.quantize_rowwise(s["x"])
        return {"codes": codes, "scales": scales,
                "back": T.dequantize_rowwise(codes, scales, s["x"].dtype)}
    if c["op"] == "norm_int8":
        codes, scales = T.rmsnorm_quantize(s["x"], s["w"], EPS)
        return {"codes": codes, "scales": scales}
    if c["op"] == "rope":
        q, k = T.TritonRoPEKernel.apply(s["q"], s["k"], s["cos"], s["sin"])
        return {"q": q, "k": k}
    if c["op"] == "glu":
        y = GLU_KERNELS[c["kind"]].apply(s["x"])
        return _with_grads(y, s) if c["train"] else {"y": y}
    if c["op"] == "attn":
        if c["kind"] == "decode":
            return {"out": flash_attn_func(s["q"], s["k"], s["v"], causal=True)}
        return {"out": T.triton_attn_func(
            s["q"], s["k"], s["v"], attn_mask=s.get("mask"),
            causal=c["kind"] in ("causal", "alibi"),
            window_size=(c["window"], 0) if c["kind"] == "window" else None,
            alibi_slopes=s.get("slopes"))}
    return {"y": s["layer"].forward_fused(s["x"])}


# ------------------------------------------------------------------- what a pass cannot avoid
def _visible(c):
    """Query-key pairs of one head."""
    n, m = c["seq_q"], c["seq_k"]
    if c["kind"] in ("causal", "alibi"):
        return n * (n + 1) // 2
    if c["kind"] == "window":
        w = min(c["window"], n - 1)
        return (w + 1) * (w + 2) // 2 + (n - w - 1) * (w + 1)
    if c["kind"] == "decode":
        q = min(n, m)
        return q * (q + 1) // 2 + (m - q) * q
    return n * m


def work(case):
    c = case
    if c["op"] == "norm":
        n, s = c["rows"] * c["cols"], SIZE[c["dtype"]]
        ins = 2 if "residual" in c["kind"] else 1
        # forward: the inputs and y; backward: the inputs and dy again, one dx for both of them
        tensors = ins + 1 + (ins + 2 if c["train"] else 0)
        return {"bytes": tensors * n * s, "flops": 8 * n * (3 if c["train"] else 1)}
    if c["op"] == "int8":
        n, s = c["rows"] * c["cols"], SIZE[c["dtype"]]
        return {"bytes": 2 * (n * (s + 1) + 4 * c["rows"]), "flops": 6 * n}
    if c["op"] == "norm_int8":
        n, s = c["rows"] * c["cols"], SIZE[c["dtype"]]
        return {"bytes": n * (s + 1) + 4 * c["rows"], "flops": 10 * n}
    if c["op"] == "rope":
        n = c["batch"] * c["seq"] * (c["heads"] + c["kv_heads"]) * c["dim"]
        return {"bytes": 2 * n * SIZE[c["dtype"]] + 4 * c["seq"] * c["dim"], "flops": 3 * n}
    if c["op"] == "glu":
        n = c["rows"] * c["hidden"]
        return {"bytes": (8 if c["train"] else 3) * n * SIZE[c["dtype"]],
                "flops": (25 if c["train"] else 8) * n}
    if c["op"] == "attn":
        kv = c["batch"] * c["seq_k"] * c["kv_heads"] * c["dim"]
        q = c["batch"] * c["seq_q"] * c["heads"] * c["dim"]
        mask = 4 * c["batch"] * c["seq_q"] * c["seq_k"] if c.get("mask") else 0
        return {"bytes": 2 * (2 * q + 2 * kv) + mask,
                "flops": 4 * c["batch"] * c["heads"] * c["dim"] * _visible(c)}
    e, f, d = c["embed"], c["ffn"], c["embed"] // c["heads"]
    weights = 2 * e * e + 2 * c["kv_heads"] * d * e + 3 * e * f
    tokens = c["batch"] * c["seq"]
    pairs = c["batch"] * c["heads"] * c["seq"] * (c["seq"] + 1) // 2
    return {"bytes": weights + 4 * tokens * e, "flops": 2 * tokens * weights + 4 * d * pairs}


def tolerance(case):
    """About four times what the outputs are off from `exact`: the storage type's rounding, and in
    32 bits the order of the sums."""
    c = case
    if c["op"] == "int8":
        return "exact"  # codes and scales are defined bit for bit
    if c["op"] == "norm_int8":
        # The order of a row's sum of squares turns a rounding now and then.
        return {"rel": 1e-4, "max": 1e-2, "differ": 1e-5}
    if c["op"] == "layer":
        return {"rel": 1.5e-2}
    if c["op"] == "attn":
        return {"rel": 1e-2 if c["dtype"] == "bf16" else 1.2e-3}
    return {"rel": {"f32": 1e-6, "f16": 1e-3, "bf16": 7e-3}[c["dtype"]]}


# --------------------------------------------------------------------------------- in 64 bits
def _norm64(c, s):
    x = s["x"] + s["r"] if "r" in s else s["x"]
    if "layernorm" in c["kind"]:
        return F.layer_norm(x, x.shape[-1:], s["w"], s["b"], EPS)
    n = s["w"] * (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS))
    return F.mish(n) if c["kind"] == "rmsnorm_mish" else n


def _glu64(c, x):
    up, gate = x.chunk(2, dim=-1)
    act = {"swiglu": F.silu, "geglu": lambda t: F.gelu(t, approximate="tanh"),
           "reglu": F.relu}[c["kind"]]
    return up * act(gate)


def _by_rows(c, s, fn, rows=4096):
    """fn over blocks of rows, in 64 bits; gradients of the parameters summed over the blocks."""
    params = {n: s[n].double().requires_grad_(c["train"]) for n in ("w", "b") if n in s}
    outs, sums = {}, {}
    for at in range(0, c["rows"], rows):
        part = {n: s[n][at:at + rows].double().requires_grad_(c["train"])
                for n in ("x", "r") if n in s}
        with torch.set_grad_enabled(c["train"]):
            y = fn(c, {**part, **params})
        outs.setdefault("y", []).append(y.detach())
        if c["train"]:
            wanted = {**part, **params}
            grads = torch.autograd.grad(y, list(wanted.values()), s["dy"][at:at + rows].double())
            for n, g in zip(wanted, grads):
                if n in params:
                    sums["d" + n] = sums.get("d" + n, 0) + g
                else:
                    outs.setdefault("d" + n, []).append(g)
    return {**{n: torch.cat(v) for n, v in outs.items()}, **sums}


def _quantised64(x, rows=4096):
    scales = (x.abs().amax(-1).float() / 127.0)
    safe = torch.where(scales > 0, scales, torch.ones_like(scales)).double()
    codes = torch.cat([torch.round(x[i:i + rows].double() / safe[i:i + rows, None])
                       for i in range(0, x.shape[0], rows)])
    return codes.clamp_(-127, 127).to(torch.int8), scales.double()


def _attention64(q, k, v, c, s):
    """One kv head's query heads at a time, 1024 query rows at a time."""
    batch, n, heads, dim = q.shape
    m, group = k.shape[1], heads // k.shape[2]
    out = torch.empty(batch, n, heads, dim, dtype=torch.float64, device=q.device)
    j = torch.arange(m, device=q.device)
    for b in range(batch):
        for h in range(heads):
            kk, vv = k[b, :, h // group].double(), v[b, :, h // group].double()
            for at in range(0, n, 1024):
                i = torch.arange(at, min(n, at + 1024), device=q.device)[:, None]
                w = (q[b, at:at + 1024, h].double() @ kk.t()) * dim ** -0.5
                if c["kind"] in ("causal", "alibi", "window"):
                    hide = j > i
                    if c["kind"] == "window":
                        hide = hide | (j < i - c["window"])
                    w.masked_fill_(hide, float("-inf"))
                if c["kind"] == "decode":
                    w.masked_fill_(j > i + (m - n), float("-inf"))
                if "slopes" in s:
                    w -= s["slopes"][h].double() * (i - j).abs()
                if "mask" in s:
                    w += s["mask"][b, 0, at:at + 1024].double()
                out[b, at:at + 1024, h] = torch.softmax(w, dim=-1) @ vv
    return out


def _rotated64(t, cos, sin):
    half = t.shape[-1] // 2
    t = t.double()
    turned = torch.cat((-t[..., half:], t[..., :half]), dim=-1)
    return t * cos.double()[None, :, None] + turned * sin.double()[None, :, None]


def _layer64(c, s):
    w = {}
    for n, t in s["weights"].items():
        codes, scales = _quantised64(t)
        # the layer multiplies with the dequantised weights as bf16 holds them
        w[n] = (codes.double() * scales[:, None]).to(torch.bfloat16).double()
    heads, kv, d = c["heads"], c["kv_heads"], c["embed"] // c["heads"]
    cos, sin = _rope_tables(c["seq"], d)
    cos, sin = cos.to(torch.bfloat16), sin.to(torch.bfloat16)  # the module's tables
    norm = lambda t: t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + EPS)  # noqa: E731
    outs = []
    for b in range(c["batch"]):
        x = s["x"][b:b + 1].double()
        n = norm(x)
        q = _rotated64((n @ w["wq"].t()).view(1, -1, heads, d), cos, sin)
        k = _rotated64((n @ w["wk"].t()).view(1, -1, kv, d), cos, sin)
        v = (n @ w["wv"].t()).view(1, -1, kv, d)
        a = _attention64(q, k, v, {"kind": "causal"}, {}).reshape(1, -1, c["embed"])
        h = x + a @ w["wo"].t()
        n = norm(h)
        outs.append(h + ((n @ w["w_up"].t()) * F.silu(n @ w["w_gate"].t())) @ w["w_down"].t())
    return torch.cat(outs)


def exact(case, seed):
    c, s = case, _inputs(case, seed)
    if c["op"] == "norm":
        return _by_rows(c, s, _norm64)
    if c["op"] == "glu":
        return _by_rows(c, s, lambda c, p: _glu64(c, p["x"]), rows=2048)
    if c["op"] == "int8":
        codes, scales = _quantised64(s["x"])
        return {"codes": codes, "scales": scales, "back": codes.double().mul_(scales[:, None])}
    if c["op"] == "norm_int8":
        # The codes are those of the norm as the activation type holds it.
        y = _by_rows({**c, "kind": "rmsnorm", "train": False}, s, _norm64)["y"]
        codes, scales = _quantised64(y.to(DTYPES[c["dtype"]]))
        return {"codes": codes, "scales": scales}
    if c["op"] == "rope":
        return {n: _rotated64(s[n], s["cos"], s["sin"]) for n in ("q", "k")}
    if c["op"] == "attn":
        return {"out": _attention64(s["q"], s["k"], s["v"], c, s)}
    return {"y": _layer64(c, s)}
