"""The work a user of this package has it do, as cases that can be timed.

A case is a dict: `op` (which public entry point), `qt` (format of the packed weights), `dtype` of
the activations, and the sizes.  The ranges:

* `mlp`     mlp_block: RMSNorm, gate / up, SiLU(gate) * up, down - the bulk of a decoder layer.
            hidden 1024 .. 8192, inter 2 .. 4 times that, 1 .. 8192 tokens
* `qkv`     qkv_rope: RMSNorm, the q / k / v projections and RoPE.  hidden 1024 .. 8192 with
            grouped-query heads of 64 or 128, 1 .. 512 tokens
* `linear`  q_gemm_dequant: o_proj, lm_head or any linear called by itself, with and without bias.
            K 1024 .. 16384, N 1000 .. 16384 (odd ones too), 1 .. 8192 tokens; blocks as a .gguf file
            stores them (Q4_K with eight scale pairs) for decode, 1 .. 64 tokens
* `pieces`  the primitives around the linears called one by one, as a host that keeps its own layer
            code does: rmsnorm_fused with a residual, rope_apply on q and k, swiglu

Tokens: 1 is interactive decode, 2 .. 64 is batched decode, above that prefill; a prompt's length is
any number.  hidden, inter and K are multiples of 256, the super-block of Q4_K and the granularity
of common decoder models.  Weights are N(0, 0.02) quantized to the format, activations N(0, 1).
"""
import math

import torch

import mlxr_b200 as mx

EPS = 1e-5
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}
QT = {"q4_0": mx.QuantType.Q4_0, "q8_0": mx.QuantType.Q8_0, "q4_k": mx.QuantType.Q4_K, "nf4": mx.QuantType.NF4,
      "gguf_q4_k": mx.QuantType.GGML_Q4_K}
BLOCK = {"q4_0": (32, 18), "q8_0": (32, 34), "q4_k": (256, 144), "nf4": (64, 34), "gguf_q4_k": (256, 144)}
MAX_POS = 8192
MAX_FLOPS = 2.0 * 3 * 8192 * 4096 * 14336     # no drawn case costs more than the largest listed one


def listed():
    return [
        # one token through the MLP block of a 1.1B-shaped model: the smallest call, launches and host time count
        dict(name="mlp_2048x5632_q4_0_m1", op="mlp", qt="q4_0", dtype="f16", M=1, hidden=2048, inter=5632),
        # interactive decode of an 8B-shaped model: the benchmark's workload
        dict(name="mlp_4096x14336_q4_k_m1", op="mlp", qt="q4_k", dtype="bf16", M=1, hidden=4096, inter=14336),
        # batched decode, 32 sequences
        dict(name="mlp_4096x14336_q4_k_m32", op="mlp", qt="q4_k", dtype="bf16", M=32, hidden=4096, inter=14336),
        # interactive decode of a 70B-shaped model: the largest weight stream
        dict(name="mlp_8192x28672_q4_k_m1", op="mlp", qt="q4_k", dtype="bf16", M=1, hidden=8192, inter=28672),
        # attention input of the 8B shape, one token
        dict(name="qkv_4096_q4_k_m1", op="qkv", qt="q4_k", dtype="bf16", M=1, hidden=4096, q_heads=32, kv_heads=8, head_dim=128),
        # the format sweep's linear: 8-bit weights at one token, 4-bit codebook weights at a batch of 16
        dict(name="linear_14336x4096_q8_0_m1", op="linear", qt="q8_0", dtype="bf16", M=1, N=14336, K=4096, bias=False),
        dict(name="linear_14336x4096_nf4_m16", op="linear", qt="nf4", dtype="bf16", M=16, N=14336, K=4096, bias=False),
        # blocks as a .gguf file stores them, a handful of sequences, a linear with bias
        dict(name="linear_4096x4096_gguf_q4_k_m5", op="linear", qt="gguf_q4_k", dtype="f16", M=5, N=4096, K=4096, bias=True),
        # prefill: one gate / up linear over 2048 tokens
        dict(name="linear_14336x4096_q4_k_m2048", op="linear", qt="q4_k", dtype="bf16", M=2048, N=14336, K=4096, bias=False),
        # a short prompt of odd length
        dict(name="mlp_4096x11008_q4_0_m333", op="mlp", qt="q4_0", dtype="f16", M=333, hidden=4096, inter=11008),
        # the primitives around the linears over a prompt of odd length
        dict(name="pieces_4096x14336_m1111", op="pieces", dtype="f16", M=1111, hidden=4096, inter=14336, q_heads=32, kv_heads=8, head_dim=128),
        # long-context prefill through the whole block: the largest
        dict(name="mlp_4096x14336_q4_k_m8192", op="mlp", qt="q4_k", dtype="bf16", M=8192, hidden=4096, inter=14336),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _flops(c):
    if c["op"] == "mlp":
        return 2.0 * c["M"] * 3 * c["hidden"] * c["inter"]
    if c["op"] == "qkv":
        return 2.0 * c["M"] * c["hidden"] * (c["q_heads"] + 2 * c["kv_heads"]) * c["head_dim"]
    if c["op"] == "linear":
        return 2.0 * c["M"] * c["N"] * c["K"]
    return 12.0 * c["M"] * (c["hidden"] + c["inter"])


def draw(rng):
    op = rng.choice(["mlp", "mlp", "mlp", "qkv", "linear", "linear", "linear", "pieces"])
    c = dict(op=op, dtype=rng.choice(["f16", "bf16"]))
    # decode, batched decode and prefill equally often
    kind = rng.choice(["one", "batch", "prefill"])
    c["M"] = rng.choice([1, 1, 1, 2]) if kind == "one" else _log(rng, 3, 64) if kind == "batch" else _log(rng, 65, 8192)
    if op != "pieces":
        c["qt"] = rng.choice(["q4_0", "q8_0", "q4_k", "q4_k", "nf4"] + (["gguf_q4_k"] if op == "linear" else []))
    if op in ("mlp", "pieces", "qkv"):
        c["hidden"] = 256 * _log(rng, 4, 32)
    if op in ("mlp", "pieces"):
        c["inter"] = 256 * round(c["hidden"] * rng.uniform(2.0, 4.0) / 256)
    if op in ("qkv", "pieces"):
        c["head_dim"] = rng.choice([64, 128])
        c["q_heads"] = c["hidden"] // c["head_dim"]
        # grouped-query attention: the query heads share the key / value heads in groups
        c["kv_heads"] = max(d for d in (1, 2, 4, 8) if c["q_heads"] % d == 0)
    if op == "qkv":
        c["M"] = min(c["M"], 512)
    if op == "linear":
        c["K"] = 256 * _log(rng, 4, 64)
        c["N"] = _log(rng, 1000, 16384)
        c["bias"] = rng.random() < 0.25
        if c["qt"] == "gguf_q4_k":
            c["M"] = min(c["M"], 64)
    while _flops(c) > MAX_FLOPS:
        c["M"] -= c["M"] // 4
    return c


# ---- weights: quantized on the device into the package's block layouts -----------------------------
def _f16_bytes(v):
    return v.to(torch.float16).contiguous().view(torch.uint8).reshape(*v.shape, 2)


def _nibbles(q):
    q = q.to(torch.uint8)
    return q[..., 0::2] | (q[..., 1::2] << 4)


def _safe_inv(d):
    return torch.where(d != 0, 1.0 / torch.where(d != 0, d, torch.ones_like(d)), torch.zeros_like(d))


def _q4_0(w):
    b = w.reshape(w.shape[0], -1, 32)
    big = b.gather(-1, b.abs().argmax(-1, keepdim=True))[..., 0]
    d = (big / -8.0).half().float()
    q = (torch.round(b * _safe_inv(d)[..., None]) + 8).clamp(0, 15)
    return torch.cat([_f16_bytes(d), _nibbles(q)], -1)


def _q8_0(w):
    b = w.reshape(w.shape[0], -1, 32)
    d = (b.abs().amax(-1) / 127.0).half().float()
    q = torch.round(b * _safe_inv(d)[..., None]).clamp(-127, 127).to(torch.int8)
    return torch.cat([_f16_bytes(d), q.view(torch.uint8)], -1)


def _nf4(w):
    from mlxr_b200.quantize import nf4_levels
    lv = torch.tensor(nf4_levels(), device=w.device)
    b = w.reshape(w.shape[0], -1, 64)
    a = b.abs().amax(-1).half().float()
    q = torch.bucketize(b * _safe_inv(a)[..., None], (lv[1:] + lv[:-1]) * 0.5)
    return torch.cat([_f16_bytes(a), _nibbles(q)], -1)


def _q4_k(w):
    """Four (scale, min) pairs per super-block, shared by sub-blocks {0,2,3}, {1}, {4,6,7}, {5};
    w ~ (q - 8) * sc * d + mn * dmin."""
    b = w.reshape(w.shape[0], -1, 8, 32)
    lo8, hi8 = b.amin(-1), b.amax(-1)
    groups = ((0, 2, 3), (1,), (4, 6, 7), (5,))
    lo = torch.stack([lo8[..., list(g)].amin(-1) for g in groups], -1)
    hi = torch.stack([hi8[..., list(g)].amax(-1) for g in groups], -1)
    ss = ((hi - lo) / 15.0).clamp_min(1e-12)
    sm = lo + 8.0 * ss
    d = (ss.amax(-1) / 63.0).half().float()
    sc = torch.round(ss * _safe_inv(d)[..., None]).clamp(1, 63)
    dmin = (sm.gather(-1, sm.abs().argmax(-1, keepdim=True))[..., 0] / 63.0).half().float()
    mn = torch.round(sm * _safe_inv(dmin)[..., None]).clamp(0, 63)
    pair = torch.tensor([0, 1, 0, 0, 2, 3, 2, 2], device=w.device)
    ss8, sm8 = (sc * d[..., None]).half().float()[..., pair], (mn * dmin[..., None]).half().float()[..., pair]
    q = (torch.round((b - sm8[..., None]) / ss8.clamp_min(1e-12)[..., None]) + 8).clamp(0, 15)
    s, m = sc.to(torch.int32), mn.to(torch.int32)
    head = []
    for g in (0, 2):
        head += [s[..., g] | ((m[..., g] & 3) << 6), (m[..., g] >> 2) | ((s[..., g + 1] & 15) << 4), (s[..., g + 1] >> 4) | (m[..., g + 1] << 2)]
    head = torch.stack(head + [torch.zeros_like(head[0])] * 6, -1).to(torch.uint8)
    return torch.cat([_f16_bytes(d), _f16_bytes(dmin), head, _nibbles(q.flatten(-2))], -1)


def _gguf_q4_k(w):
    """Eight (scale, min) pairs per super-block; w ~ q * sc * d - mn * dmin."""
    b = w.reshape(w.shape[0], -1, 8, 32)
    lo, hi = b.amin(-1).clamp_max(0.0), b.amax(-1)
    ss = ((hi - lo) / 15.0).clamp_min(1e-12)
    d, dmin = (ss.amax(-1) / 63.0).half().float(), (-lo.amin(-1) / 63.0).half().float()
    sc = torch.round(ss * _safe_inv(d)[..., None]).clamp(0, 63)
    mn = torch.round(-lo * _safe_inv(dmin)[..., None]).clamp(0, 63)
    q = torch.round((b + (mn * dmin[..., None])[..., None]) / (sc * d[..., None]).clamp_min(1e-12)[..., None]).clamp(0, 15).to(torch.uint8)
    s, m = sc.to(torch.int32), mn.to(torch.int32)
    head = torch.cat([s[..., :4] | ((s[..., 4:] >> 4) << 6), m[..., :4] | ((m[..., 4:] >> 4) << 6), (s[..., 4:] & 15) | ((m[..., 4:] & 15) << 4)], -1).to(torch.uint8)
    qs = q[..., 0::2, :] | (q[..., 1::2, :] << 4)      # 64-element chunks: low nibbles, then high nibbles
    return torch.cat([_f16_bytes(d), _f16_bytes(dmin), head, qs.flatten(-2)], -1)


_QUANTIZE = {"q4_0": _q4_0, "q8_0": _q8_0, "q4_k": _q4_k, "nf4": _nf4, "gguf_q4_k": _gguf_q4_k}


def _weights(N, K, qt, gen):
    w = torch.randn((N, K), device="cuda", generator=gen) * 0.02
    return _QUANTIZE[qt](w).contiguous().reshape(-1)


def _weight_bytes(N, K, qt):
    be, bb = BLOCK[qt]
    return N * (K // be) * bb


# ---- the interface ----------------------------------------------------------------------------------
def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dt = DTYPES[c["dtype"]]

    def acts(*shape):
        return torch.randn(shape, device="cuda", generator=gen).to(dt)

    def norm_weight(n):
        return (1.0 + 0.1 * torch.randn(n, device="cuda", generator=gen)).to(dt)

    s = dict(c)
    M = c["M"]
    if c["op"] in ("qkv", "pieces"):
        s["cos"], s["sin"] = mx.compute_rope_tables(MAX_POS, c["head_dim"], 500000.0, device=torch.device("cuda"))
        s["positions"] = torch.randint(0, MAX_POS, (M,), device="cuda", generator=gen, dtype=torch.int32)
    if c["op"] == "mlp":
        H, I = c["hidden"], c["inter"]
        s.update(x=acts(M, H), norm=norm_weight(H), gate=_weights(I, H, c["qt"], gen), up=_weights(I, H, c["qt"], gen), down=_weights(H, I, c["qt"], gen))
    elif c["op"] == "qkv":
        H, d = c["hidden"], c["head_dim"]
        s.update(x=acts(M, H), norm=norm_weight(H), wq=_weights(c["q_heads"] * d, H, c["qt"], gen),
                 wk=_weights(c["kv_heads"] * d, H, c["qt"], gen), wv=_weights(c["kv_heads"] * d, H, c["qt"], gen))
    elif c["op"] == "linear":
        s.update(x=acts(M, c["K"]), w=_weights(c["N"], c["K"], c["qt"], gen), b=acts(c["N"]) if c["bias"] else None)
    else:
        s.update(x=acts(M, c["hidden"]), residual=acts(M, c["hidden"]), norm=norm_weight(c["hidden"]), gate=acts(M, c["inter"]), up=acts(M, c["inter"]),
                 q=acts(M, c["q_heads"], c["head_dim"]), k=acts(M, c["kv_heads"], c["head_dim"]))
    return s


def run(state):
    s = state
    if s["op"] == "mlp":
        return mx.mlp_block(s["x"], s["norm"], s["gate"], s["up"], s["down"], s["inter"], QT[s["qt"]], EPS)
    if s["op"] == "qkv":
        return mx.qkv_rope(s["x"], s["norm"], s["wq"], s["wk"], s["wv"], s["cos"], s["sin"], s["positions"],
                           s["q_heads"], s["kv_heads"], s["head_dim"], QT[s["qt"]], EPS)
    if s["op"] == "linear":
        return mx.q_gemm_dequant(s["x"], s["w"], s["M"], s["N"], s["K"], QT[s["qt"]], BLOCK[s["qt"]][0], s["b"])
    return (mx.rmsnorm_fused(s["x"], s["norm"], EPS, s["residual"]), mx.rope_apply(s["q"], s["cos"], s["sin"], s["positions"]),
            mx.rope_apply(s["k"], s["cos"], s["sin"], s["positions"]), mx.swiglu(s["gate"], s["up"]))


def work(case):
    c = case
    M = c["M"]
    if c["op"] == "mlp":
        H, I = c["hidden"], c["inter"]
        n = 2 * _weight_bytes(I, H, c["qt"]) + _weight_bytes(H, I, c["qt"]) + 2 * (2 * M * H + H)
    elif c["op"] == "qkv":
        H, rows = c["hidden"], (c["q_heads"] + 2 * c["kv_heads"]) * c["head_dim"]
        n = _weight_bytes(rows, H, c["qt"]) + 2 * (M * H + H + M * rows) + M * (4 + 2 * c["head_dim"])
    elif c["op"] == "linear":
        n = _weight_bytes(c["N"], c["K"], c["qt"]) + 2 * (M * c["K"] + M * c["N"] + (c["N"] if c["bias"] else 0))
    else:
        heads = (c["q_heads"] + c["kv_heads"]) * c["head_dim"]
        n = 2 * M * (3 * c["hidden"] + 2 * heads + 3 * c["inter"]) + M * (4 + 2 * c["head_dim"]) + 2 * c["hidden"]
    return {"bytes": n, "flops": _flops(c)}


def tolerance(case):
    # pieces round once per output; a linear's weights and, in the block, n and h are rounded to the
    # activation dtype before the fp32-accumulated products
    if case["op"] == "pieces":
        return {"rel": 4e-3} if case["dtype"] == "bf16" else {"rel": 5e-4}
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 2e-3}
