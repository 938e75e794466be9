"""Timed cases: the framework's single-GPU work through its public entry points.

Every case is a dict of plain values with a ``kind``; the kinds and what they stand for:

    norm      RMSNorm forward and backward (``ops.norm.rmsnorm``): two of them in every block of every model
    linear    a projection, forward and backward (``ops.gemm.linear``): attention projections and heads of a trainer
    ffn       the gated feed-forward layer, forward and backward (``ops.gemm.glu_ffn``): the headline layer
    attn      attention, forward and backward (``ops.attention.attention``): training
    prefill   attention forward from one fused qkv matrix (``ops.attention.flash_attention``): prompt processing
    qgemm     a projection with group-quantised weights for many tokens (``ops.gemm.gemm_q``): prompt processing
    ce        cross-entropy over bf16 logits, forward and backward (``parallel.vocab_ce``): the loss of a trainer
    moe       a routed mixture-of-experts layer, forward and backward (``parallel.moe.EPMoE``)
    block     a whole decoder block, forward and backward (``models.hybrid.Block``)
    decode    one token of the decoder, embedding to argmax, for every sequence of a batch (``models.e2b.E2BDecoder``)

``draw`` gives further cases of the same ranges, ragged and odd sizes among them.
"""
from __future__ import annotations

import math

import torch
import torch.distributed as dist

DEV = "cuda"
BF16 = torch.bfloat16


def listed():
    return [
        # The smallest call: the norm of a short sequence; launches and host time count.
        dict(name="norm_small", kind="norm", rows=512, cols=2048),
        # A projection over a ragged number of tokens (packed sequences of a fine-tuning batch).
        dict(name="linear_ragged", kind="linear", tokens=1000, n=3072, k=2048),
        # The tensor-parallel FFN benchmark's layer on one GPU: 4096 tokens, 4096 -> 14336 -> 4096.
        dict(name="ffn_headline", kind="ffn", tokens=4096, d=4096, f=14336, act="silu"),
        # Attention of the hybrid trainer: one sequence of 8192 tokens, 16 heads of 128.
        dict(name="attn_train_long", kind="attn", B=1, T=8192, H=16, Hkv=16, hd=128, causal=True, window=0, drop=0.0),
        # Grouped-query attention over a ragged sequence length, heads of 64, a batch of short sequences.
        dict(name="attn_train_gqa", kind="attn", B=3, T=1111, H=8, Hkv=2, hd=64, causal=True, window=0, drop=0.0),
        # Prompt attention of the decoder: heads of 256, sliding window, the full context of a batch of 8.
        dict(name="attn_prefill_window", kind="prefill", B=8, T=1024, H=8, Hkv=2, hd=256, window=512),
        # Prompt projection with 4-bit weights: 512 tokens through the down projection.
        dict(name="qgemm_prefill", kind="qgemm", tokens=512, n=2048, k=8192, bits=4),
        # The trainer's loss: 8192 tokens, vocabulary 50304.
        dict(name="ce_train", kind="ce", rows=8192, vocab=50304),
        # The routed MoE benchmark's layer on one GPU: 8192 tokens, 64 experts of 1408, top-6, skewed loads.
        dict(name="moe_train", kind="moe", tokens=8192, d=2048, f=1408, experts=64, k=6),
        # A block of the hybrid trainer (24 of them make the model): one sequence of 8192 tokens.
        dict(name="block_train", kind="block", T=8192, d=2048, heads=16, kv_heads=16, hd=128, f=8192),
        # Decoding, one period of the model's layers (four local, one global) with its head, so that a rounding in the
        # first layer does not outgrow the comparison: one sequence with bf16 weights (latency), eight with 4-bit
        # weights (serving).
        dict(name="decode_bf16_b1", kind="decode", B=1, quant="bf16", layers=5, vocab=262144, pos_lo=512, pos_hi=767),
        dict(name="decode_w4_b8", kind="decode", B=8, quant="w4", layers=5, vocab=65536, pos_lo=512, pos_hi=767),
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer of lo..hi, a multiple of ``step``, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["norm", "linear", "ffn", "attn", "attn", "prefill", "qgemm", "ce", "moe", "block", "decode", "decode"])
    if kind == "norm":
        return dict(kind=kind, rows=_log_int(rng, 1, 32768), cols=_log_int(rng, 256, 8192, 8))
    if kind == "linear":
        return dict(kind=kind, tokens=_log_int(rng, 64, 8192, 8), n=_log_int(rng, 256, 8192, 64), k=_log_int(rng, 256, 8192, 64))
    if kind == "ffn":
        return dict(kind=kind, tokens=_log_int(rng, 64, 4096, 8), d=_log_int(rng, 512, 4096, 64),
                    f=_log_int(rng, 1024, 14336, 64), act=rng.choice(["silu", "gelu_tanh"]))
    if kind == "attn":
        T = _log_int(rng, 48, 8192)
        Hkv = rng.choice([1, 2, 4, 8])
        H = Hkv * rng.choice([1, 2, 4])
        B = rng.randint(1, max(1, min(8, (16 * 8192 * 8192) // (2 * H * T * T))))
        causal = rng.random() < 0.8
        window = _log_int(rng, 64, T) if causal and T > 64 and rng.random() < 0.25 else 0
        return dict(kind=kind, B=B, T=T, H=H, Hkv=Hkv, hd=rng.choice([64, 128]), causal=causal, window=window,
                    drop=0.1 if rng.random() < 0.15 else 0.0)
    if kind == "prefill":
        return dict(kind=kind, B=rng.randint(1, 8), T=_log_int(rng, 32, 1024), H=8, Hkv=2, hd=rng.choice([128, 256]),
                    window=rng.choice([0, 512, 300]))
    if kind == "qgemm":
        n, k = rng.choice([(3072, 2048), (2048, 2048), (16384, 2048), (2048, 8192), (1536, 1024)])
        return dict(kind=kind, tokens=_log_int(rng, 9, 4096), n=n, k=k, bits=rng.choice([4, 8]))
    if kind == "ce":
        return dict(kind=kind, rows=_log_int(rng, 64, 8192), vocab=rng.choice([50304, 50257, 32000, 32064, 16128, 40001]))
    if kind == "moe":
        return dict(kind=kind, tokens=_log_int(rng, 512, 8192, 64), d=rng.choice([1024, 2048]), f=rng.choice([512, 768, 1408]),
                    experts=rng.choice([8, 16, 64]), k=rng.choice([2, 4, 6]))
    if kind == "block":
        heads = rng.choice([8, 16])
        return dict(kind=kind, T=_log_int(rng, 256, 8192, 8), d=128 * heads, heads=heads, kv_heads=rng.choice([heads, heads // 4]),
                    hd=128, f=rng.choice([2816, 4096, 8192]))
    lo = _log_int(rng, 16, 900)                     # positions already in the caches
    return dict(kind="decode", B=rng.randint(1, 8), quant=rng.choice(["bf16", "w4", "w8"]), layers=rng.choice([3, 5]),
                vocab=rng.choice([262144, 65536]), pos_lo=lo, pos_hi=min(1000, lo + 256))


# ------------------------------------------------------------------------------------------------------- inputs
def _randn(shape, g, std=1.0, dtype=BF16):
    return (torch.randn(shape, generator=g, device=DEV, dtype=torch.float32) * std).to(dtype)


def _inputs(c, seed):
    """The tensors of a case, from its seed alone (what ``prepare`` hands to the framework and ``exact`` works from)."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 40))
    k = c["kind"]
    if k == "norm":
        return dict(x=_randn((c["rows"], c["cols"]), g), w=1 + _randn((c["cols"],), g, 0.1), dy=_randn((c["rows"], c["cols"]), g))
    if k == "linear":
        return dict(x=_randn((c["tokens"], c["k"]), g), w=_randn((c["n"], c["k"]), g, 0.02), dy=_randn((c["tokens"], c["n"]), g))
    if k == "ffn":
        return dict(x=_randn((c["tokens"], c["d"]), g), wgu=_randn((2 * c["f"], c["d"]), g, 0.02),
                    wd=_randn((c["d"], c["f"]), g, 0.02), dy=_randn((c["tokens"], c["d"]), g))
    if k == "attn":
        B, T, H, Hkv, hd = (c[n] for n in ("B", "T", "H", "Hkv", "hd"))
        return dict(q=_randn((B, T, H, hd), g), k=_randn((B, T, Hkv, hd), g), v=_randn((B, T, Hkv, hd), g), do=_randn((B, T, H, hd), g))
    if k == "prefill":
        return dict(qkv=_randn((c["B"] * c["T"], (c["H"] + 2 * c["Hkv"]) * c["hd"]), g))
    if k == "qgemm":
        return dict(x=_randn((c["tokens"], c["k"]), g), w=_randn((c["n"], c["k"]), g, 0.02))
    if k == "ce":
        t = torch.randint(0, c["vocab"], (c["rows"],), generator=g, device=DEV)
        t[:: 17] = -100                                                   # padding tokens
        return dict(logits=_randn((c["rows"], c["vocab"]), g, 2.0), targets=t)
    if k == "moe":
        T, D, F, E = c["tokens"], c["d"], c["f"], c["experts"]
        return dict(x=_randn((T, D), g), wr=_randn((E, D), g, 0.02), w1=_randn((E * 2 * F, D), g, 0.02), w2=_randn((E * D, F), g, 0.02),
                    bias=torch.randn(E, generator=g, device=DEV), dy=_randn((T, D), g))
    if k == "block":
        d, hd = c["d"], c["hd"]
        return dict(x=_randn((c["T"], d), g), dy=_randn((c["T"], d), g), norm1=1 + _randn((d,), g, 0.1), norm2=1 + _randn((d,), g, 0.1),
                    w_qkv=_randn(((c["heads"] + 2 * c["kv_heads"]) * hd, d), g, 0.02), w_o=_randn((d, c["heads"] * hd), g, 0.02),
                    w_gate_up=_randn((2 * c["f"], d), g, 0.02), w_down=_randn((d, c["f"]), g, 0.02))
    cfg, B = _decode_shape(c), c["B"]
    pos = torch.randint(c["pos_lo"], c["pos_hi"] + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    tok = torch.randint(0, c["vocab"], (B,), generator=g, device=DEV, dtype=torch.int32)
    # a prompt's keys and values: projections of normalised activations (std 0.9 at this width and initialisation)
    cache = [_randn((2, B, cfg["kv_heads"], cfg["max_seq"], cfg["head_dim"]), g, 0.9) for _ in range(c["layers"])]
    return dict(pos=pos, tok=tok, cache=cache)


def _decode_shape(c):
    return dict(layers=c["layers"], d_model=2048, q_heads=8, kv_heads=2, head_dim=256, d_ff=8192, vocab=c["vocab"], window=512,
                local_per_global=4, theta=1e6, eps=1e-6, max_seq=1024, init_std=0.02)


def _decode_seed(seed):
    return int(seed) % 9973


class _Solo:
    """The context of a job of one process, with a symmetric heap of its own that is given back with the state."""

    def __init__(self, heap_bytes):
        from mesh_b200.config import MeshConfig, set_config
        from mesh_b200.distributed.context import MeshContext
        from mesh_b200.runtime.rendezvous import Rendezvous
        set_config(MeshConfig.from_env(heap_bytes=heap_bytes))
        self.ctx = MeshContext(0, 1, torch.device(DEV, 0), Rendezvous(dist.HashStore(), 0, 1), None)

    def __del__(self):
        if self.ctx._heap is not None:
            self.ctx._heap.close()


def prepare(c, seed):
    s = dict(c)
    k = c["kind"]
    s.update(i := _inputs(c, seed))
    if k in ("norm", "linear", "ffn"):
        for n in ("x", "w", "wgu", "wd"):
            if n in i:
                i[n].requires_grad_(True)
    elif k == "attn":
        for n in ("q", "k", "v"):
            i[n].requires_grad_(True)
        s["dropout"] = dict(p=c["drop"], seed=1234 + int(seed) % 1000) if c["drop"] else None
    elif k == "prefill":
        B, T, H, Hkv, hd = (c[n] for n in ("B", "T", "H", "Hkv", "hd"))
        q = i["qkv"]
        s["q"] = q[:, :H * hd].view(B, T, H, hd)
        s["k"] = q[:, H * hd:(H + Hkv) * hd].view(B, T, Hkv, hd)
        s["v"] = q[:, (H + Hkv) * hd:].view(B, T, Hkv, hd)
    elif k == "qgemm":
        from mesh_b200.ops.decode import quantize_w4, quantize_w8
        s["codes"], s["scales"] = (quantize_w4 if c["bits"] == 4 else quantize_w8)(i["w"])
        del s["w"]
    elif k == "ce":
        i["logits"].requires_grad_(True)
    elif k == "moe":
        from mesh_b200.parallel.moe import EPMoE
        T, D, F, E = c["tokens"], c["d"], c["f"], c["experts"]
        cap = 2 * T * c["k"] + 256 * E + 256
        s["solo"] = _Solo(4 * cap * D * 2 + (8 << 20))
        s["layer"] = EPMoE(s["solo"].ctx, T, D, F, E, c["k"])
    elif k == "block":
        from mesh_b200.models.hybrid import Block, HybridConfig
        from mesh_b200.parallel.topology import ParallelContext, ParallelDims
        cfg = HybridConfig(vocab=50304, d_model=c["d"], n_layers=24, n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["hd"],
                           d_ff=c["f"], seq_len=c["T"], striped=False)
        b = Block(cfg, ParallelContext(None, ParallelDims()), 0, BF16, torch.device(DEV, 0))
        s["params"] = [b.norm1, b.attn.w_qkv, b.attn.w_o, b.norm2, b.ffn.w_gate_up, b.ffn.w_down]
        with torch.no_grad():
            for p, n in zip(s["params"], ("norm1", "w_qkv", "w_o", "norm2", "w_gate_up", "w_down")):
                p.copy_(i[n])
                del s[n]
        s["block"], s["posn"] = b, torch.arange(c["T"], device=DEV)
        i["x"].requires_grad_(True)
    else:
        from mesh_b200.distributed.context import MeshContext
        from mesh_b200.models.e2b import E2BConfig, E2BDecoder
        ctx = MeshContext(0, 1, torch.device(DEV, 0), None, None)
        m = E2BDecoder(E2BConfig(**_decode_shape(c)), ctx, c["B"], c["quant"], seed=_decode_seed(seed))
        m.pos.copy_(i["pos"])
        m.tok.copy_(i["tok"])
        m.capture()
        for L, kv in zip(m.layers, i["cache"]):
            L["kc"].copy_(kv[0])
            L["vc"].copy_(kv[1])
        del s["cache"]
        s["model"], s["caches"] = m, [t for L in m.layers for t in (L["kc"], L["vc"])]
    return s


def run(s):
    k = s["kind"]
    if k == "norm":
        from mesh_b200.ops.norm import rmsnorm
        y = rmsnorm(s["x"], s["w"])
        return [y, *torch.autograd.grad(y, (s["x"], s["w"]), s["dy"])]
    if k == "linear":
        from mesh_b200.ops.gemm import linear
        y = linear(s["x"], s["w"])
        return [y, *torch.autograd.grad(y, (s["x"], s["w"]), s["dy"])]
    if k == "ffn":
        from mesh_b200.ops.gemm import glu_ffn
        y = glu_ffn(s["x"], s["wgu"], s["wd"], s["act"])
        return [y, *torch.autograd.grad(y, (s["x"], s["wgu"], s["wd"]), s["dy"])]
    if k == "attn":
        from mesh_b200.ops.attention import attention
        y = attention(s["q"], s["k"], s["v"], causal=s["causal"], window=s["window"], dropout=s["dropout"])
        return [y, *torch.autograd.grad(y, (s["q"], s["k"], s["v"]), s["do"])]
    if k == "prefill":
        from mesh_b200.ops.attention import flash_attention
        return flash_attention(s["q"], s["k"], s["v"], causal=True, window=s["window"])
    if k == "qgemm":
        from mesh_b200.ops.gemm import gemm_q
        return gemm_q(s["x"], s["codes"], s["scales"])
    if k == "ce":
        from mesh_b200.parallel.vocab_ce import vocab_parallel_cross_entropy
        loss = vocab_parallel_cross_entropy(s["logits"], s["targets"], 0)
        return [loss, *torch.autograd.grad(loss, s["logits"])]
    if k == "moe":
        y = s["layer"].forward(s["x"], s["wr"], s["w1"], s["w2"], s["bias"])
        return [y, *s["layer"].backward(s["dy"])]
    if k == "block":
        y = s["block"](s["x"], 1, s["posn"])
        return [y, *torch.autograd.grad(y, (s["x"], *s["params"]), s["dy"])]
    m = s["model"]
    m.pos.copy_(s["pos"])                      # every pass decodes the same token of the same sequences
    m.tok.copy_(s["tok"])
    m.decode(1, record=False)
    return [m.logits, m.tok, m.pos, *s["caches"]]


# ---------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(T, causal, window):
    """(query, key) pairs that the masks leave visible."""
    if not causal:
        return T * T
    w = min(window, T) if window else T
    return w * (w + 1) // 2 + (T - w) * w


def _weight_bytes(n, k, quant):
    return n * k * 2 if quant == "bf16" else n * k // 2 + n * k // 32 if quant == "w4" else n * k + n * k // 32


def work(c):
    k = c["kind"]
    if k == "norm":
        e = c["rows"] * c["cols"]
        return {"bytes": 2 * e * 4 + 6 * c["cols"], "flops": 12 * e}                # x, dy in; y, dx out
    if k == "linear":
        t, n, kk = c["tokens"], c["n"], c["k"]
        return {"bytes": 2 * (2 * t * kk + 2 * n * kk + 2 * t * n), "flops": 6 * t * n * kk}
    if k == "ffn":
        t, d, f = c["tokens"], c["d"], c["f"]
        return {"bytes": 2 * (4 * t * d + 6 * d * f), "flops": 18 * t * d * f}
    if k == "attn":
        q, kv = c["B"] * c["T"] * c["H"] * c["hd"], c["B"] * c["T"] * c["Hkv"] * c["hd"]
        p = c["B"] * c["H"] * _pairs(c["T"], c["causal"], c["window"])
        return {"bytes": 2 * (4 * q + 4 * kv), "flops": 14 * p * c["hd"]}
    if k == "prefill":
        p = c["B"] * c["H"] * _pairs(c["T"], True, c["window"])
        return {"bytes": 2 * c["B"] * c["T"] * (2 * c["H"] + 2 * c["Hkv"]) * c["hd"], "flops": 4 * p * c["hd"]}
    if k == "qgemm":
        t, n, kk = c["tokens"], c["n"], c["k"]
        return {"bytes": 2 * (t * kk + t * n) + _weight_bytes(n, kk, "w%d" % c["bits"]), "flops": 2 * t * n * kk}
    if k == "ce":
        e = c["rows"] * c["vocab"]
        return {"bytes": 4 * e, "flops": 6 * e}
    if k == "moe":
        t, d, f, e, kk = c["tokens"], c["d"], c["f"], c["experts"], c["k"]
        return {"bytes": 2 * (4 * t * d + 6 * e * d * f + 2 * e * d), "flops": 18 * t * kk * d * f + 6 * t * e * d}
    if k == "block":
        T, d, f, hd = c["T"], c["d"], c["f"], c["hd"]
        mats = (c["heads"] + 2 * c["kv_heads"]) * hd * d + d * c["heads"] * hd + 3 * d * f
        return {"bytes": 2 * (4 * T * d + 2 * mats), "flops": 6 * T * mats + 14 * c["heads"] * _pairs(T, True, 0) * hd}
    s = _decode_shape(c)
    d, hd, f = s["d_model"], s["head_dim"], s["d_ff"]
    shapes = [((s["q_heads"] + 2 * s["kv_heads"]) * hd, d), (d, s["q_heads"] * hd), (2 * f, d), (d, f)]
    b = sum(_weight_bytes(n, kk, c["quant"]) for n, kk in shapes) * c["layers"] + _weight_bytes(c["vocab"], d, c["quant"])
    keys = 0
    mean = (c["pos_lo"] + c["pos_hi"]) // 2 + 1
    for l in range(c["layers"]):
        keys += min(mean, s["window"]) if _local(s, l) else mean
    b += c["B"] * (keys * 2 * s["kv_heads"] * hd * 2 + c["vocab"] * 4)
    par = sum(n * kk for n, kk in shapes) * c["layers"] + c["vocab"] * d
    return {"bytes": b, "flops": 2 * par * c["B"] + 4 * c["B"] * keys * s["q_heads"] * hd}


def _local(s, l):
    return (l + 1) % (s["local_per_global"] + 1) != 0


def tolerance(c):
    """bf16 results of fp32 sums, about four times what the start differs by from the 64-bit statement; 8-bit mantissas
    round to 2**-9, and a chain of rounded intermediates adds up."""
    k = c["kind"]
    if k == "moe":
        # a token whose last two choices tie after rounding may take another expert: single rows differ wholly
        return {"rel": 0.025, "max": 0.99}
    if k == "decode":
        return {"rel": 0.03, "max": 0.5, "differ": 0.01}
    if k in ("block", "ffn", "attn"):
        return {"rel": 0.015, "max": 0.3}
    return {"rel": 0.01, "max": 0.2}


# ---------------------------------------------------------------------------------------------------- 64-bit statements
def _rms64(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _act64(t, name):
    return torch.nn.functional.silu(t) if name == "silu" else torch.nn.functional.gelu(t, approximate="tanh")


class _Attention64(torch.autograd.Function):
    """``q [T, H, hd]``, ``k, v [T, Hkv, hd]`` head by head, scores recomputed in the backward pass."""

    @staticmethod
    def _p(q, k, causal, window):
        T = q.shape[0]
        s = (q @ k.T) * q.shape[-1] ** -0.5
        if causal:
            i = torch.arange(T, device=q.device)
            hide = i[None, :] > i[:, None]
            if window:
                hide |= i[None, :] <= i[:, None] - window
            s.masked_fill_(hide, float("-inf"))
        return torch.softmax(s, -1)

    @staticmethod
    def forward(ctx, q, k, v, causal, window):
        ctx.save_for_backward(q, k, v)
        ctx.cfg = causal, window
        g = q.shape[1] // k.shape[1]
        return torch.stack([_Attention64._p(q[:, h], k[:, h // g], causal, window) @ v[:, h // g] for h in range(q.shape[1])], 1)

    @staticmethod
    def backward(ctx, do):
        q, k, v = ctx.saved_tensors
        g = q.shape[1] // k.shape[1]
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for h in range(q.shape[1]):
            j = h // g
            p = _Attention64._p(q[:, h], k[:, j], *ctx.cfg)
            dv[:, j] += p.T @ do[:, h]
            dp = do[:, h] @ v[:, j].T
            ds = p * (dp - (p * dp).sum(-1, keepdim=True)) * q.shape[-1] ** -0.5
            dq[:, h] = ds @ k[:, j]
            dk[:, j] += ds.T @ q[:, h]
        return dq, dk, dv, None, None


def _rope64(x, pos, theta):
    half = x.shape[-1] // 2
    inv = theta ** (-torch.arange(0, 2 * half, 2, device=x.device, dtype=torch.float64) / (2 * half))
    a = pos.double()[:, None] * inv[None]
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], -1)


def _quantised64(w, quant):
    """The values that group-quantised weights stand for: one fp16 scale per 64 inputs, codes around 8 or 128."""
    if quant == "bf16":
        return w.double()
    wf = w.float().view(w.shape[0], -1, 64)
    top, mid, lo, hi = (7.0, 8, 0, 15) if quant == "w4" else (127.0, 128, 1, 255)
    s = (wf.abs().amax(-1) / top).clamp_min(1e-8).to(torch.float16)
    code = torch.clamp(torch.round(wf / s.float()[..., None]) + mid, lo, hi)
    return ((code.double() - mid) * s.double()[..., None]).view(w.shape)


def _exact_decode(c, seed):
    i, s, B = _inputs(c, seed), _decode_shape(c), c["B"]
    hd, qh, kvh, d, f = s["head_dim"], s["q_heads"], s["kv_heads"], s["d_model"], s["d_ff"]

    def weight(n, kk, at):                     # the decoder draws its weights from its seed, matrix by matrix
        g = torch.Generator(device=DEV).manual_seed(at)
        return (torch.randn((n, kk), generator=g, device=DEV, dtype=torch.float32) * s["init_std"]).to(BF16)

    sd = _decode_seed(seed)
    emb = torch.cat([weight(c["vocab"] // 8, d, sd * 7919 + 500 + ch) for ch in range(8)])
    x = emb[i["tok"].long()].double()
    pos, caches = i["pos"].long(), []
    for l in range(c["layers"]):
        w = [_quantised64(weight(n, kk, sd * 1000003 + l * 101 + j), c["quant"]) for j, (n, kk) in
             enumerate([(qh * hd, d), (kvh * hd, d), (kvh * hd, d), (d, qh * hd), (f, d), (f, d), (d, f)], 1)]
        h = _rms64(x, 1.0)
        q = _rope64((h @ w[0].T).view(B, qh, hd), pos, s["theta"])
        kn = _rope64((h @ w[1].T).view(B, kvh, hd), pos, s["theta"])
        kc, vc = i["cache"][l][0].double(), i["cache"][l][1].double()
        for b in range(B):
            kc[b, :, pos[b]], vc[b, :, pos[b]] = kn[b], (h[b] @ w[2].T).view(kvh, hd)
        o = torch.empty((B, qh, hd), dtype=torch.float64, device=DEV)
        for b in range(B):
            p = int(pos[b])
            lo = max(0, p - s["window"] + 1) if _local(s, l) else 0
            kk, vv = (t[b, :, lo:p + 1].repeat_interleave(qh // kvh, 0) for t in (kc, vc))
            o[b] = (torch.softmax((q[b][:, None] @ kk.transpose(1, 2)) * hd ** -0.5, -1) @ vv)[:, 0]
        x = x + o.view(B, -1) @ w[3].T
        h = _rms64(x, 1.0)
        x = x + (_act64(h @ w[4].T, "gelu_tanh") * (h @ w[5].T)) @ w[6].T
        caches += [kc, vc]
    h = _rms64(x, 1.0)
    logits = torch.cat([h @ _quantised64(e, c["quant"]).T for e in emb.chunk(8)], 1)
    return [logits, None, None, *caches]


def _exact_moe(c, i):
    x, w1, w2, dy = i["x"].double(), i["w1"], i["w2"], i["dy"].double()
    T, D, F, E, k = c["tokens"], c["d"], c["f"], c["experts"], c["k"]
    wr = i["wr"].double()
    logits = (x @ wr.T).to(BF16).double()                       # the layer routes on bf16 logits
    p = torch.softmax(logits + i["bias"].double(), -1)
    top, idx = torch.topk(p, k, -1)
    total = top.sum(-1, keepdim=True)
    w = top / total
    out, dx = torch.zeros_like(x), torch.zeros_like(x)
    dw1, dw2 = torch.empty((E, 2 * F, D), dtype=torch.float64, device=DEV), torch.empty((E, D, F), dtype=torch.float64, device=DEV)
    dw = torch.zeros_like(w)
    for e in range(E):
        tok, j = (idx == e).nonzero(as_tuple=True)
        a, b = w1.view(E, 2 * F, D)[e].double(), w2.view(E, D, F)[e].double()
        xe, we = x[tok], w[tok, j][:, None]
        g, u = xe @ a[:F].T, xe @ a[F:].T
        sg = torch.sigmoid(g)
        h = g * sg * u
        y = h @ b.T
        out.index_add_(0, tok, y * we)
        dw[tok, j] = (y * dy[tok]).sum(-1)
        dye = dy[tok] * we
        dw2[e] = dye.T @ h
        dh = dye @ b
        dgu = torch.cat([dh * u * (sg + g * sg * (1 - sg)), dh * g * sg], 1)
        dw1[e] = dgu.T @ xe
        dx.index_add_(0, tok, dgu @ a)
    dtop = (dw - (dw * w).sum(-1, keepdim=True)) / total
    dp = torch.zeros_like(p).scatter_(1, idx, dtop)
    dl = p * (dp - (p * dp).sum(-1, keepdim=True))
    return [out, dx + dl @ wr, dl.T @ x, dw1.view(E * 2 * F, D), dw2.view(E * D, F)]


def exact(c, seed):
    k = c["kind"]
    if k == "decode":
        return _exact_decode(c, seed)
    if k == "attn" and c["drop"]:
        return None                                             # the mask is the framework's own generator
    i = _inputs(c, seed)
    if k == "moe":
        return _exact_moe(c, i)
    if k == "qgemm":
        return i["x"].double() @ _quantised64(i["w"], "w%d" % c["bits"]).T
    if k == "prefill":
        B, T, H, Hkv, hd = (c[n] for n in ("B", "T", "H", "Hkv", "hd"))
        t = i["qkv"].double().view(B, T, H + 2 * Hkv, hd)
        return torch.stack([_Attention64.apply(t[b, :, :H], t[b, :, H:H + Hkv], t[b, :, H + Hkv:], True, c["window"]) for b in range(B)])
    i = {n: t.double().requires_grad_(True) if t.is_floating_point() else t for n, t in i.items()}
    if k == "norm":
        y, leaves, dy = _rms64(i["x"], i["w"]), (i["x"], i["w"]), i["dy"]
    elif k == "linear":
        y, leaves, dy = i["x"] @ i["w"].T, (i["x"], i["w"]), i["dy"]
    elif k == "ffn":
        y = (_act64(i["x"] @ i["wgu"][:c["f"]].T, c["act"]) * (i["x"] @ i["wgu"][c["f"]:].T)) @ i["wd"].T
        leaves, dy = (i["x"], i["wgu"], i["wd"]), i["dy"]
    elif k == "attn":
        y = torch.stack([_Attention64.apply(i["q"][b], i["k"][b], i["v"][b], c["causal"], c["window"]) for b in range(c["B"])])
        leaves, dy = (i["q"], i["k"], i["v"]), i["do"]
    elif k == "ce":
        y = torch.nn.functional.cross_entropy(i["logits"], i["targets"], ignore_index=-100)
        leaves, dy = (i["logits"],), None
    else:
        x, H, Hkv, hd, f = i["x"], c["heads"], c["kv_heads"], c["hd"], c["f"]
        pos = torch.arange(c["T"], device=DEV)
        t = (_rms64(x, i["norm1"]) @ i["w_qkv"].T).view(-1, H + 2 * Hkv, hd)
        o = _Attention64.apply(_rope64(t[:, :H], pos, 10000.0), _rope64(t[:, H:H + Hkv], pos, 10000.0), t[:, H + Hkv:], True, 0)
        x1 = x + o.reshape(-1, H * hd) @ i["w_o"].T
        h = _rms64(x1, i["norm2"])
        y = x1 + (_act64(h @ i["w_gate_up"][:f].T, "silu") * (h @ i["w_gate_up"][f:].T)) @ i["w_down"].T
        leaves, dy = (x, i["norm1"], i["w_qkv"], i["w_o"], i["norm2"], i["w_gate_up"], i["w_down"]), i["dy"]
    return [y.detach(), *torch.autograd.grad(y, leaves, dy)]
