"""What the single-GPU performance of this framework is measured on.

A rank of a tensor-parallel group runs these kernels between its collectives: plain GEMMs from one token to a whole
prefill chunk, the gate/up projection with its SwiGLU, the QKV projection with rotation and cache write, grouped-query
decode attention over a static cache, residual add + RMSNorm, and whole steps of the model runner.  The shapes are the
shards of the 70B configuration at TP = 8 (`LlamaConfig.shard`), the headline GEMM of `bench.py` (N = K = 8192, fp16),
the 8B configuration, and ragged sizes in between.  Collectives need several GPUs and are not measured here.
"""
from __future__ import annotations

import math

import torch

from ooverlap_b200.models import llama
from ooverlap_b200.ops import attn_decode, gemm, gemm_rope_kv_write, gemm_swiglu, rmsnorm, rope_tables

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
LARGEST_FLOPS = 2.0 * 8192 ** 3
LARGEST_BYTES = 1.0e9
EPS = 1e-5
HEAD = 128


def listed():
    return [
        # Residual add + RMSNorm of a decode batch: the smallest call, its launch is what it costs.
        dict(name="norm_decode", op="norm", rows=16, hidden=8192, dtype="bf16"),
        # The same on a prefill chunk of 16384 tokens: a stream over memory.
        dict(name="norm_prefill", op="norm", rows=16384, hidden=8192, dtype="bf16"),
        # Gate/up projection of one decode step at a small batch: time to read the weights once.
        dict(name="gemm_decode", op="gemm", m=16, n=7168, k=8192, dtype="bf16"),
        # A mixed batch (decode tokens beside a short prompt) on the down projection.
        dict(name="gemm_mixed", op="gemm", m=250, n=8192, k=3584, dtype="bf16"),
        # Headline GEMM of bench.py, its smallest row count.
        dict(name="gemm_512", op="gemm", m=512, n=8192, k=8192, dtype="fp16"),
        # Headline GEMM of bench.py, its largest row count.
        dict(name="gemm_8192", op="gemm", m=8192, n=8192, k=8192, dtype="fp16"),
        # Ragged everything: no size is a multiple of a tile.
        dict(name="gemm_ragged", op="gemm", m=1037, n=4104, k=2056, dtype="bf16"),
        # Gate/up projection + SwiGLU in one call, decode batch of 64.
        dict(name="swiglu_decode", op="swiglu", m=64, f=3584, k=8192, dtype="bf16"),
        # Decode attention of a large batch, one KV head per rank, cache nearly full.
        dict(name="attn_batch", op="attn", b=256, h=8, kv=1, ctx=1900, max_len=2048, dtype="bf16"),
        # Decode attention of two long contexts with all heads of the 8B configuration on one GPU.
        dict(name="attn_long", op="attn", b=2, h=32, kv=8, ctx=30000, max_len=32768, dtype="fp16"),
        # One decode step of four layers and the vocabulary projection, replayed from a CUDA graph as generate() does.
        dict(name="decode_step", op="decode", b=32, layers=4, ctx=1088, max_len=2048, dtype="bf16"),
        # One layer over a prefill chunk of two prompts, and the logits of their last tokens.
        dict(name="prefill_step", op="prefill", b=2, t=2048, layers=1, max_len=2048, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["norm", "gemm", "gemm", "gemm", "swiglu", "qkv", "attn", "attn", "decode"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if op == "norm":
        hidden = rng.choice([1024, 2048, 4096, 5120, 8192]) if rng.random() < 0.6 else 8 * rng.randint(64, 1024)
        return dict(op=op, rows=_log(rng, 1, 16384), hidden=hidden, dtype=dtype)
    if op in ("gemm", "swiglu"):
        while True:
            m, k = _log(rng, 1, 8192), 8 * _log(rng, 64, 1024)
            n = 8 * _log(rng, 64, 1024)
            if op == "gemm" and rng.random() < 0.15:
                n += rng.randint(1, 7)
            wide = 2 if op == "swiglu" else 1
            if 2.0 * m * n * wide * k <= LARGEST_FLOPS:
                return dict(op=op, m=m, k=k, dtype=dtype, **({"f": n} if op == "swiglu" else {"n": n}))
    if op == "qkv":
        b, t = (_log(rng, 1, 256), 1) if rng.random() < 0.6 else (rng.randint(1, 4), rng.randint(17, 1024))
        return dict(op=op, b=b, t=t, h=8, kv=rng.choice([1, 2]), k=rng.choice([4096, 8192]), pos=rng.randint(0, 900),
                    max_len=2048, dtype=dtype)
    if op == "attn":
        while True:
            h, kv = rng.choice([(8, 1), (8, 2), (32, 8), (16, 1), (64, 8)])
            b, ctx = _log(rng, 1, 256), _log(rng, 16, 32768)
            max_len = ctx + _log(rng, 1, 2048)
            if 512.0 * b * kv * max_len <= LARGEST_BYTES:
                return dict(op=op, b=b, h=h, kv=kv, ctx=ctx, max_len=max_len, dtype=dtype)
    ctx = rng.randint(16, 2000)
    return dict(op=op, b=_log(rng, 1, 64), layers=rng.choice([1, 2, 3]), ctx=ctx, max_len=2048, dtype="bf16")


class _Inputs:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, dtype, scale=1.0):
        return torch.randn(*shape, device="cuda", generator=self.g, dtype=torch.float32).mul_(scale).to(dtype)


def _model(case, seed):
    cfg = llama.LLAMA3_70B.shard(8, layers=case["layers"])
    return llama.LlamaTP(cfg, None, dtype=DTYPES[case["dtype"]], max_batch=case["b"], max_len=case["max_len"], seed=int(seed))


def prepare(case, seed):
    op, dt, rnd = case["op"], DTYPES[case["dtype"]], _Inputs(seed)
    s = dict(op=op, case=dict(case))
    if op == "norm":
        rows, hidden = case["rows"], case["hidden"]
        s["x"], s["res"] = rnd.normal(rows, hidden, dtype=dt), rnd.normal(rows, hidden, dtype=dt)
        s["w"] = (1 + rnd.normal(hidden, dtype=torch.float32, scale=0.02)).to(dt)
    elif op in ("gemm", "swiglu"):
        n = case["n"] if op == "gemm" else 2 * case["f"]
        s["a"] = rnd.normal(case["m"], case["k"], dtype=dt)
        s["b"] = rnd.normal(n, case["k"], dtype=dt, scale=case["k"] ** -0.5)
    elif op == "qkv":
        b, t, h, kv, k = case["b"], case["t"], case["h"], case["kv"], case["k"]
        s["a"] = rnd.normal(b * t, k, dtype=dt)
        s["b"] = rnd.normal((h + 2 * kv) * HEAD, k, dtype=dt, scale=k ** -0.5)
        s["kc"] = torch.zeros(b, kv, case["max_len"], HEAD, device="cuda", dtype=dt)
        s["vc"] = torch.zeros_like(s["kc"])
        s["cos"], s["sin"] = rope_tables(case["max_len"], HEAD, 500000.0, "cuda")
        s["pos"] = torch.full((1,), case["pos"], dtype=torch.long, device="cuda")
    elif op == "attn":
        b, h, kv = case["b"], case["h"], case["kv"]
        s["q"] = rnd.normal(b, h, HEAD, dtype=dt)
        s["kc"] = rnd.normal(b, kv, case["max_len"], HEAD, dtype=dt)
        s["vc"] = rnd.normal(b, kv, case["max_len"], HEAD, dtype=dt)
        s["pos"] = torch.full((1,), case["ctx"] - 1, dtype=torch.long, device="cuda")
    else:
        model = s["model"] = _model(case, seed)
        b, t = case["b"], case.get("t", 1)
        s["tokens"] = torch.randint(0, model.cfg.vocab, (b, t), device="cuda", generator=rnd.g)
        if op == "decode":
            ctx = case["ctx"]
            model.k_cache[:, :, :, :ctx] = rnd.normal(*model.k_cache[:, :, :, :ctx].shape, dtype=dt)
            model.v_cache[:, :, :, :ctx] = rnd.normal(*model.v_cache[:, :, :, :ctx].shape, dtype=dt)
            s["pos"] = torch.full((1,), ctx, dtype=torch.long, device="cuda")
            _decode(s)  # the eager step that generate() takes before it captures
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["logits"] = _decode(s)
    return s


def _decode(s):
    m = s["model"]
    with torch.no_grad():
        return gemm(m.forward(s["tokens"], s["pos"]), m.lm_head)


def run(s):
    op = s["op"]
    if op == "norm":
        return rmsnorm(s["x"], s["w"], EPS, s["res"])
    if op == "gemm":
        return gemm(s["a"], s["b"])
    if op == "swiglu":
        return gemm_swiglu(s["a"], s["b"])
    if op == "qkv":
        c = s["case"]
        q = gemm_rope_kv_write(s["a"], s["b"], c["b"], c["t"], c["h"], c["kv"], s["kc"], s["vc"], s["cos"], s["sin"], s["pos"])
        return q, s["kc"], s["vc"]
    if op == "attn":
        return attn_decode(s["q"], s["kc"], s["vc"], s["pos"])
    m = s["model"]
    if op == "decode":
        s["graph"].replay()
        return s["logits"], m.k_cache, m.v_cache
    b, t = s["tokens"].shape
    with torch.no_grad():
        hidden = m.forward(s["tokens"], 0)
        logits = gemm(hidden.view(b, t, -1)[:, -1].contiguous(), m.lm_head)
    return logits, hidden, m.k_cache, m.v_cache


# ------------------------------------------------------------------------------------------------------- what it needs
def work(case):
    op = case["op"]
    if op == "norm":
        n = case["rows"] * case["hidden"]
        return {"bytes": 2.0 * (4 * n + case["hidden"]), "flops": 5.0 * n}
    if op in ("gemm", "swiglu"):
        m, k = case["m"], case["k"]
        n, out = (case["n"], case["n"]) if op == "gemm" else (2 * case["f"], case["f"])
        return {"bytes": 2.0 * (m * k + n * k + m * out), "flops": 2.0 * m * n * k}
    if op == "qkv":
        m, n, k = case["b"] * case["t"], (case["h"] + 2 * case["kv"]) * HEAD, case["k"]
        return {"bytes": 2.0 * (m * k + n * k + m * n), "flops": 2.0 * m * n * k}
    if op == "attn":
        kv = case["b"] * case["kv"] * case["ctx"] * HEAD
        q = case["b"] * case["h"] * HEAD
        return {"bytes": 4.0 * kv + 4.0 * q, "flops": 4.0 * q * case["ctx"]}
    cfg = llama.LLAMA3_70B.shard(8, layers=case["layers"])
    b, t = case["b"], case.get("t", 1)
    m, hd = b * t, cfg.head_dim
    per_layer = ((cfg.heads + 2 * cfg.kv_heads) * hd + cfg.heads * hd + 3 * cfg.ffn) * cfg.hidden
    weights, head = per_layer * cfg.layers, cfg.vocab * cfg.hidden
    new_kv = 2 * m * cfg.kv_heads * hd * cfg.layers
    if op == "decode":
        old_kv = 2 * b * cfg.kv_heads * hd * case["ctx"] * cfg.layers
        pairs = b * case["ctx"]
    else:
        old_kv, pairs = 0, b * t * (t + 1) // 2
    attention = 4.0 * pairs * cfg.heads * hd * cfg.layers
    return {"bytes": 2.0 * (weights + head + old_kv + new_kv + 2 * m * cfg.hidden + b * cfg.vocab),
            "flops": 2.0 * m * weights + 2.0 * b * head + attention}


def tolerance(case):
    """About four times the distance from the exact result that one rounding to the output type (and, where the op has
    a 16-bit intermediate of its own, that rounding too) gives."""
    bf16 = case["dtype"] == "bf16"
    if case["op"] in ("decode", "prefill"):
        return {"rel": 0.03 if bf16 else 0.004, "max": 0.4}
    if case["op"] == "norm":
        return {"rel": 0.0095 if bf16 else 0.0012, "max": 0.06}
    if case["op"] in ("swiglu", "attn"):
        return {"rel": 0.0085 if bf16 else 0.0011, "max": 0.1}
    return {"rel": 0.007 if bf16 else 0.0009, "max": 0.05}


# ---------------------------------------------------------------------------------------------------- 64-bit results
def _rotate(x, cos, sin):
    """x: [..., T, heads, hd], cos / sin: [T, hd / 2]; pairs are (2i, 2i + 1)."""
    a, b, c, s = x[..., 0::2], x[..., 1::2], cos[:, None, :], sin[:, None, :]
    return torch.stack((a * c - b * s, a * s + b * c), dim=-1).flatten(-2)


def _norm(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _attention(q, k, v, causal):
    """q: [T, H, hd], k / v: [KV, L, hd], one sequence; returns [T, H * hd]."""
    T, H, hd = q.shape
    KV, L = k.shape[0], k.shape[1]
    q = q.view(T, KV, H // KV, hd).permute(1, 2, 0, 3).reshape(KV, -1, hd)
    sc = (torch.bmm(q, k.transpose(1, 2)) / math.sqrt(hd)).view(KV, H // KV, T, L)
    if causal:
        sc = sc.masked_fill(torch.ones(T, L, dtype=torch.bool, device=q.device).triu(1), float("-inf"))
    o = torch.bmm(sc.softmax(-1).view(KV, -1, L), v)
    return o.view(KV, H // KV, T, hd).permute(2, 0, 1, 3).reshape(T, H * hd)


def exact(case, seed):
    s, op = prepare(case, seed), case["op"]
    d = {k: v.double() for k, v in s.items() if isinstance(v, torch.Tensor) and v.is_floating_point()}
    if op == "norm":
        h = d["x"] + d["res"]
        return _norm(h, d["w"]), h
    if op == "gemm":
        return d["a"] @ d["b"].t()
    if op == "swiglu":
        gu = d["a"] @ d["b"].t()
        return torch.nn.functional.silu(gu[:, :case["f"]]) * gu[:, case["f"]:]
    if op == "qkv":
        b, t, h, kv, p = case["b"], case["t"], case["h"], case["kv"], case["pos"]
        x = (d["a"] @ d["b"].t()).view(b, t, h + 2 * kv, HEAD)
        cos, sin = d["cos"][p:p + t], d["sin"][p:p + t]
        kc, vc = torch.zeros_like(d["kc"]), torch.zeros_like(d["vc"])
        kc[:, :, p:p + t] = _rotate(x[:, :, h:h + kv], cos, sin).transpose(1, 2)
        vc[:, :, p:p + t] = x[:, :, h + kv:].transpose(1, 2)
        return _rotate(x[:, :, :h], cos, sin).reshape(b * t, h * HEAD), kc, vc
    if op == "attn":
        L = case["ctx"]
        return torch.stack([_attention(s["q"][i:i + 1].double(), s["kc"][i, :, :L].double(), s["vc"][i, :, :L].double(), False)[0]
                            for i in range(case["b"])])
    return _exact_model(case, s)


def _exact_model(case, s):
    m = s["model"]
    cfg, hd, (b, t) = m.cfg, m.cfg.head_dim, s["tokens"].shape
    pos = case["ctx"] if case["op"] == "decode" else 0
    cos, sin = m.rope_cos32[pos:pos + t].double(), m.rope_sin32[pos:pos + t].double()
    h = m.embed[s["tokens"].reshape(-1)].double()
    kc, vc = m.k_cache.double(), m.v_cache.double()
    for i, layer in enumerate(m.layers):
        w = {k: v.double() for k, v in layer.items()}
        x = (_norm(h, w["norm1"]) @ w["wqkv"].t()).view(b, t, -1, hd)
        q = _rotate(x[:, :, :cfg.heads], cos, sin)
        kc[i, :b, :, pos:pos + t] = _rotate(x[:, :, cfg.heads:cfg.heads + cfg.kv_heads], cos, sin).transpose(1, 2)
        vc[i, :b, :, pos:pos + t] = x[:, :, cfg.heads + cfg.kv_heads:].transpose(1, 2)
        att = torch.cat([_attention(q[j], kc[i, j, :, :pos + t], vc[i, j, :, :pos + t], t > 1) for j in range(b)])
        h = h + att @ w["wo"].t()
        gu = _norm(h, w["norm2"]) @ w["wgu"].t()
        h = h + (torch.nn.functional.silu(gu[:, :cfg.ffn]) * gu[:, cfg.ffn:]) @ w["wd"].t()
    x = _norm(h, m.final_norm.double())
    logits = x.view(b, t, -1)[:, -1] @ m.lm_head.double().t()
    return (logits, kc, vc) if case["op"] == "decode" else (logits, x, kc, vc)
