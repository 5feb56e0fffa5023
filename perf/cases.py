"""The work that users of this library have it do, as cases that can be timed and compared.

Every case goes through the public entry points on one GPU, where each fused op runs as its local
product. The sizes are those of the benchmark (hidden 8192, FFN 28672, un-sharded or one rank's
share of 2, 4 or 8), of the shape files under ``tiling/shapes`` and of the attention benchmarks;
:func:`draw` spreads over the ranges that these stand for. Inputs are made on the GPU from the seed.

Families (``case["kind"]``):

``linear``     one tensor-parallel linear: matmul_allreduce, matmul_reduce_scatter or allgather_matmul
``mlp``        the tensor-parallel MLP block (up projection + activation, down projection)
``quant``      int8 linear with the dequantisation in the epilogue
``mx``         block-scaled fp8 linear on a 16-bit activation: quantise, pack the scales, multiply
``moe``        expert products over ragged token groups, 16-bit or int8
``moe_grad``   the experts' weight gradients (groups along K)
``attention``  flash attention, prefill and decode over a cache
``mla``        latent-attention decode over a paged cache
"""
import math

import torch

import mm_rs_with_catlass_b200 as catcoc
from mm_rs_with_catlass_b200.models.tp_mlp import TPMLP, TPMLPConfig

DEVICE = torch.device("cuda", 0)
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
HIDDEN, FFN = 8192, 28672
LARGEST_FLOPS = 4.0 * 8192 * HIDDEN * FFN          # the largest listed case
LARGEST_BYTES = 2.0 * 1024 ** 3                    # operands of a drawn case


def listed():
    return [
        # the golden configuration: a call so small that only its latency counts
        dict(name="small_fp16", kind="linear", op="allreduce", m=256, n=256, k=512, dtype="fp16", trans_b=False),
        # row-parallel linear of a decode batch: 128 rows against a weight that has to be streamed once
        dict(name="linear_m128", kind="linear", op="allreduce", m=128, n=HIDDEN, k=FFN, dtype="bf16", trans_b=False),
        # column-parallel linear whose K no 16-byte pitch fits
        dict(name="linear_ragged_k", kind="linear", op="allgather", m=1024, n=5120, k=6148, dtype="fp16", trans_b=False),
        # mid-size linear with ragged rows and columns, weight stored [N, K]
        dict(name="linear_trans_b", kind="linear", op="reduce_scatter", m=8144, n=1696, k=5120, dtype="bf16", trans_b=True),
        # training / prefill step of the MLP block at the benchmark's size
        dict(name="mlp_m8192", kind="mlp", m=8192, hidden=HIDDEN, ffn=FFN, activation="gelu"),
        # int8 serving: 1024 tokens
        dict(name="quant_m1024", kind="quant", m=1024, n=HIDDEN, k=FFN, bias=True, trans_b=False, out="bf16"),
        # fp8 serving: 4096 tokens against one rank's share of four
        dict(name="mx_m4096", kind="mx", m=4096, n=HIDDEN, k=FFN // 4, fmt="e4m3"),
        # mixture of experts, forward: 32 experts, ragged groups
        dict(name="moe_experts", kind="moe", groups=32, tokens=14080, n=4096, k=2048, dtype="bf16", trans_b=True),
        # ... and backward: the experts' weight gradients
        dict(name="moe_weight_grad", kind="moe_grad", groups=32, tokens=14080, m=2048, n=4096, dtype="bf16"),
        # causal prefill with grouped-query heads
        dict(name="attn_prefill", kind="attention", b=2, hq=32, hk=8, sq=8192, sk=8192, d=128, causal=True, dtype="bf16"),
        # one decode step over a cache
        dict(name="attn_decode", kind="attention", b=16, hq=32, hk=8, sq=1, sk=4096, d=128, causal=True, dtype="bf16"),
        # latent-attention decode step, sequences of mixed length
        dict(name="mla_decode", kind="mla", b=32, h=16, s=4096, q_len=1, causal=False, dtype="bf16"),
    ]


# ------------------------------------------------------------------------------------------
# drawn cases
# ------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, x, step):
    """``x``, or in a third of the draws a size near it that is only a multiple of ``step``."""
    return x if rng.random() < 0.67 else max(step, (x - rng.randrange(1, max(2, x // 8))) // step * step)


def _draw_once(rng):
    kind = rng.choice(["linear", "linear", "linear", "mlp", "quant", "mx", "moe", "moe", "moe_grad", "attention",
                       "attention", "attention", "mla", "mla"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    world = rng.choice([1, 2, 4, 8])
    if kind == "linear":
        op = rng.choice(["allreduce", "reduce_scatter", "allgather"])
        n, k = (FFN // world, HIDDEN) if op == "allgather" else (HIDDEN, FFN // world)
        if rng.random() < 0.4:
            n, k = _log(rng, 128, 16384), _log(rng, 128, 16384)
        return dict(kind=kind, op=op, m=_log(rng, 1, 16384), n=_ragged(rng, n, rng.choice([1, 8])),
                    k=_ragged(rng, k, rng.choice([1, 2, 8])), dtype=dtype, trans_b=rng.random() < 0.4)
    if kind == "mlp":
        return dict(kind=kind, m=_log(rng, 1, 8192), hidden=rng.choice([4096, HIDDEN]), ffn=FFN // world,
                    activation=rng.choice(["gelu", "silu"]))
    if kind == "quant":
        return dict(kind=kind, m=_log(rng, 1, 16384), n=_ragged(rng, HIDDEN, 16), k=_ragged(rng, FFN // world, 16),
                    bias=rng.random() < 0.5, trans_b=rng.random() < 0.4, out=rng.choice(["bf16", "fp16"]))
    if kind == "mx":
        return dict(kind=kind, m=_log(rng, 16, 8192), n=_ragged(rng, HIDDEN, 8), k=_ragged(rng, FFN // world, 32),
                    fmt=rng.choice(["e4m3", "e4m3", "e5m2"]))
    if kind == "moe":
        return dict(kind=kind, groups=rng.choice([8, 16, 32, 64]), tokens=_log(rng, 64, 32768),
                    n=rng.choice([1408, 2048, 4096]), k=rng.choice([1024, 2048, 4096]),
                    dtype=rng.choice(["bf16", "fp16", "int8"]), trans_b=rng.random() < 0.5)
    if kind == "moe_grad":
        return dict(kind=kind, groups=rng.choice([8, 16, 32]), tokens=_log(rng, 512, 32768), m=rng.choice([1024, 2048]),
                    n=rng.choice([1408, 2048, 4096]), dtype=dtype)
    if kind == "attention":
        d = rng.choice([64, 128, 128])
        hk = rng.choice([4, 8, 32])
        hq = 32
        b = _log(rng, 1, 16)
        if rng.random() < 0.4:        # decode: one to a few new tokens over a cache
            sk = _log(rng, 256, 16384)
            return dict(kind=kind, b=b, hq=hq, hk=hk, sq=rng.choice([1, 1, 2, 4]), sk=sk, d=d, causal=True, dtype=dtype)
        sq = _log(rng, 64, 16384)
        sk = sq if rng.random() < 0.7 else sq + _log(rng, 64, 4096)
        return dict(kind=kind, b=b, hq=hq, hk=hk, sq=sq, sk=sk, d=d, causal=rng.random() < 0.7, dtype=dtype)
    q_len = rng.choice([1, 1, 2, 4])
    return dict(kind="mla", b=_log(rng, 1, 128), h=rng.choice([16, 32, 64, 128]), s=_log(rng, 256, 16384), q_len=q_len,
                causal=q_len > 1, dtype=dtype)


def draw(rng):
    while True:
        case = _draw_once(rng)
        w = work(case)
        if w["flops"] <= 0.25 * LARGEST_FLOPS and w["bytes"] <= LARGEST_BYTES:
            return case


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _normal(g, *shape, dtype, std=1.0):
    return (torch.randn(*shape, device=DEVICE, dtype=torch.float32, generator=g) * std).to(dtype)


def _int8(g, *shape):
    return torch.randint(-127, 128, shape, device=DEVICE, dtype=torch.int8, generator=g)


def _uniform(g, n, lo, hi):
    return torch.rand(n, device=DEVICE, generator=g) * (hi - lo) + lo


def _group_sizes(tokens, groups, seed):
    """Token counts of the experts: from a quarter of the mean to seven quarters, in an order of the seed."""
    w = [0.25 + 1.5 * (i + 0.5) / groups for i in range(groups)]
    bounds, acc, begin = [], 0.0, 0
    for x in w:
        acc += x
        bounds.append(min(tokens, int(round(tokens * acc / groups))))
    bounds[-1] = tokens
    sizes = []
    for e in bounds:
        sizes.append(e - begin)
        begin = e
    order = torch.randperm(groups, generator=torch.Generator().manual_seed(seed)).tolist()
    return [sizes[i] for i in order]


def _kv_lens(b, s, q_len):
    """Sequence lengths of a decode batch: half of the longest to the longest."""
    return [max(q_len, s - (s // 2) * i // max(1, b - 1)) if b > 1 else s for i in range(b)]


def prepare(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind in ("linear", "mlp", "quant", "mx"):
        st["ctx"] = catcoc.default_context()
    if kind == "linear":
        dt = DTYPES[case["dtype"]]
        m, n, k = case["m"], case["n"], case["k"]
        st["a"] = _normal(g, m, k, dtype=dt)
        st["b"] = _normal(g, *((n, k) if case["trans_b"] else (k, n)), dtype=dt, std=0.02)
    elif kind == "mlp":
        cfg = TPMLPConfig(hidden=case["hidden"], ffn=case["ffn"], activation=case["activation"])
        st["mlp"] = TPMLP(cfg, st["ctx"], DEVICE, seed=seed)
        st["x"] = _normal(g, case["m"], case["hidden"], dtype=torch.bfloat16)
    elif kind == "quant":
        m, n, k = case["m"], case["n"], case["k"]
        st["x1"] = _int8(g, m, k)
        st["x2"] = _int8(g, *((n, k) if case["trans_b"] else (k, n)))
        st["s1"], st["s2"] = _uniform(g, m, 0.001, 0.02), _uniform(g, n, 0.0, 0.01)
        st["bias"] = torch.randint(-1000, 1000, (n,), device=DEVICE, dtype=torch.int32, generator=g) if case["bias"] else None
    elif kind == "mx":
        # the weight is quantised once; the activation arrives in 16 bits and is quantised in every step
        st["x"] = _normal(g, case["m"], case["k"], dtype=torch.bfloat16)
        w = _normal(g, case["n"], case["k"], dtype=torch.bfloat16, std=0.02)
        st["wq"], ws = catcoc.quantize_mxf8(w, case["fmt"])
        st["ws"] = catcoc.pack_scales(ws)
    elif kind in ("moe", "moe_grad"):
        ends, total = [], 0
        for c in _group_sizes(case["tokens"], case["groups"], seed):
            total += c
            ends.append(total)
        gr, t, n = case["groups"], case["tokens"], case["n"]
        if kind == "moe_grad":
            dt = DTYPES[case["dtype"]]
            st["a"], st["b"] = _normal(g, t, case["m"], dtype=dt), _normal(g, t, n, dtype=dt, std=0.1)
            st["ends"] = ends                                                    # the ranges are on the host
        else:
            k = case["k"]
            wshape = (gr, n, k) if case["trans_b"] else (gr, k, n)
            st["ends"] = torch.tensor(ends, dtype=torch.int32, device=DEVICE)    # the router's result is on the device
            if case["dtype"] == "int8":
                st["a"], st["b"] = _int8(g, t, k), _int8(g, *wshape)
                st["s1"] = _uniform(g, t, 0.001, 0.02)
                st["s2"] = _uniform(g, gr * n, 0.0, 0.01).view(gr, n)
            else:
                dt = DTYPES[case["dtype"]]
                st["a"], st["b"] = _normal(g, t, k, dtype=dt), _normal(g, *wshape, dtype=dt, std=0.02)
    elif kind == "attention":
        dt = DTYPES[case["dtype"]]
        b, d = case["b"], case["d"]
        st["q"] = _normal(g, b, case["hq"], case["sq"], d, dtype=dt)
        st["k"], st["v"] = (_normal(g, b, case["hk"], case["sk"], d, dtype=dt) for _ in range(2))
    else:
        dt = DTYPES[case["dtype"]]
        b, h, s, q_len = case["b"], case["h"], case["s"], case["q_len"]
        pages = (s + 127) // 128
        st["qn"], st["qr"] = _normal(g, b * q_len, h, 512, dtype=dt), _normal(g, b * q_len, h, 64, dtype=dt)
        st["ckv"], st["kr"] = _normal(g, b * pages, 128, 512, dtype=dt), _normal(g, b * pages, 128, 64, dtype=dt)
        st["table"] = torch.randperm(b * pages, device=DEVICE, generator=g).view(b, pages).to(torch.int32)
        order = torch.randperm(b, generator=torch.Generator().manual_seed(seed))
        st["lens"] = torch.tensor(_kv_lens(b, s, q_len), dtype=torch.int32)[order].to(DEVICE)
    return st


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "linear":
        if c["op"] == "allreduce":
            return catcoc.matmul_allreduce(st["a"], st["b"], trans_b=c["trans_b"])
        if c["op"] == "reduce_scatter":
            return catcoc.matmul_reduce_scatter(st["a"], st["b"], trans_b=c["trans_b"])
        return catcoc.allgather_matmul(st["a"], st["b"], trans_b=c["trans_b"])[0]
    if kind == "mlp":
        return st["mlp"].forward(st["x"])
    if kind == "quant":
        return catcoc.quant_matmul_reduce_scatter(st["x1"], st["x2"], st["s1"], st["s2"], st["bias"],
                                                  trans_b=c["trans_b"], out_dtype=DTYPES[c["out"]])
    if kind == "mx":
        xq, xs = catcoc.quantize_mxf8(st["x"], c["fmt"])
        return catcoc.mxf8_matmul_reduce_scatter(xq, catcoc.pack_scales(xs), st["wq"], st["ws"])
    if kind == "moe":
        if c["dtype"] == "int8":
            return catcoc.grouped_quant_matmul(st["a"], st["b"], st["s1"], st["s2"], st["ends"], trans_b=c["trans_b"])
        return catcoc.grouped_matmul(st["a"], st["b"], st["ends"], trans_b=c["trans_b"])
    if kind == "moe_grad":
        return catcoc.grouped_matmul_slice_k(st["a"], st["b"], st["ends"])
    if kind == "attention":
        return catcoc.flash_attention(st["q"], st["k"], st["v"], causal=c["causal"])
    return catcoc.mla_decode(st["qn"], st["qr"], st["ckv"], st["kr"], st["table"], st["lens"], q_len=c["q_len"],
                             causal=c["causal"])


# ------------------------------------------------------------------------------------------
# what a pass cannot do without, and how close two correct results are
# ------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2.0 * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}
    if kind == "mlp":
        m, h, f = case["m"], case["hidden"], case["ffn"]
        return {"bytes": 2.0 * (2 * m * h + 2 * h * f), "flops": 4.0 * m * h * f}
    if kind == "quant":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": m * k + k * n + 2.0 * m * n + 4.0 * (m + n), "flops": 2.0 * m * n * k}
    if kind == "mx":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2.0 * m * k + n * k * (1 + 1 / 32) + 2.0 * m * n, "flops": 2.0 * m * n * k}
    if kind == "moe":
        gr, t, n, k = case["groups"], case["tokens"], case["n"], case["k"]
        e = 1 if case["dtype"] == "int8" else 2
        used = sum(1 for c in _group_sizes(t, gr, 0) if c > 0)
        return {"bytes": float(e * (t * k + used * n * k) + 2 * t * n), "flops": 2.0 * t * n * k}
    if kind == "moe_grad":
        gr, t, m, n = case["groups"], case["tokens"], case["m"], case["n"]
        return {"bytes": 2.0 * (t * m + t * n + gr * m * n), "flops": 2.0 * t * m * n}
    if kind == "attention":
        b, hq, hk, sq, sk, d = (case[x] for x in ("b", "hq", "hk", "sq", "sk", "d"))
        # (query, key) pairs: query i sees keys up to i + sk - sq
        pairs = sq * (sk - sq) + sq * (sq + 1) / 2 if case["causal"] else sq * sk
        return {"bytes": 2.0 * (2 * b * hq * sq * d + 2 * b * hk * sk * d), "flops": 4.0 * b * hq * pairs * d}
    b, h, s, q_len = case["b"], case["h"], case["s"], case["q_len"]
    keys = float(sum(_kv_lens(b, s, q_len)))
    return {"bytes": 2.0 * (keys * 576 + b * q_len * h * (576 + 512)), "flops": 2.0 * q_len * h * keys * (576 + 512)}


# Largest error seen against the same function in fp64 (2-norm, and largest element over the rms): products
# bf16 1.7e-3 / 3.9e-3, fp16 2.1e-4 / 5e-4 (one rounding of an fp32 sum); the MLP block 2.4e-3 / 1.1e-2 (its
# hidden activation is rounded too); attention bf16 2.4e-3 / 4.1e-2, fp16 2.9e-4 / 2.1e-3; latent attention bf16
# 2.0e-3 / 9.3e-3 (probabilities are rounded to the operand type). About four times that is allowed.
_TOLERANCE = {
    ("product", "bf16"): (7e-3, 1.6e-2), ("product", "fp16"): (9e-4, 2e-3),
    ("mlp", "bf16"): (1e-2, 4.2e-2),
    ("attention", "bf16"): (9.5e-3, 1.7e-1), ("attention", "fp16"): (1.2e-3, 2e-2),
    ("mla", "bf16"): (8e-3, 3.8e-2), ("mla", "fp16"): (1.2e-3, 1e-2),
}


def tolerance(case):
    kind = case["kind"] if case["kind"] in ("mlp", "attention", "mla") else "product"
    out = case.get("out", case.get("dtype", "bf16"))       # the mx linear and the MLP block work in bf16
    rel, most = _TOLERANCE[kind, "bf16" if out == "int8" else out]   # int8 experts are dequantised to bf16
    return {"rel": rel, "max": most}
