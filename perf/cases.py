"""Workloads of the quantized-inference operators, as a user's program runs them.

Twelve listed cases cover the framework's public entry points from a few microseconds to a few
milliseconds: quantising activations, gradients and the key/value cache, expanding 4-bit weights,
FP8 linear layers (one token, a prompt, the backward pass), the FP8 SwiGLU MLP, W4A16 linear layers
at three batch sizes, and FP8 attention.  draw() gives more cases of the same kinds with other
sizes, ragged ones among them.  Inputs are synthetic: activations ~ N(0, 1), weights ~ N(0, 0.02)
quantised per output channel, gradients ~ N(0, 1e-3), nibbles uniform.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "gaudi-pytorch-bridge_b200")  # the repository's root is the working folder
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import b200_hpu_ops  # noqa: E402
from b200_hpu_ops import tp_mlp  # noqa: E402

E4M3, E5M2, BF16, F32 = torch.float8_e4m3fn, torch.float8_e5m2, torch.bfloat16, torch.float32
FP8 = {"e4m3": E4M3, "e5m2": E5M2}
FLOAT = {"bf16": BF16, "f32": F32}
HEAD_DIM = 128


def listed():
    return [
        # one decode step of 16 sequences: the hidden state goes to e4m3, its amax to the scale history; pure latency
        {"name": "quantize_decode", "kind": "quantize", "rows": 16, "cols": 4096, "src": "bf16", "dst": "e4m3", "stochastic": False},
        # a training step's gradient of 8192 tokens, rounded stochastically to e5m2, with its amax
        {"name": "quantize_gradient", "kind": "quantize", "rows": 8192, "cols": 8192, "src": "bf16", "dst": "e5m2", "stochastic": True},
        # keys and values of a prompt of ragged length into an e4m3 cache, and the cache read back as bf16
        {"name": "kv_cache", "kind": "kv_cache", "batch": 3, "tokens": 2731, "heads": 8},
        # GPTQ weights of a layer expanded to bf16 once per use, as a program without a fused GEMM does
        {"name": "expand_int4", "kind": "expand_int4", "k": 8192, "n": 8192, "group": 128, "signed": False, "zero_points": True},
        # one token through an FP8 linear layer: activation cast, then the GEMM with per-channel scales and bias
        {"name": "linear_decode", "kind": "linear", "tokens": 1, "k": 4096, "n": 14336, "bias": True},
        # the same layer over a prompt of 4096 tokens
        {"name": "linear_prefill", "kind": "linear", "tokens": 4096, "k": 4096, "n": 14336, "bias": True},
        # backward of an FP8 linear layer: input gradient in bf16, weight gradient accumulated into fp32
        {"name": "linear_backward", "kind": "linear_backward", "tokens": 8000, "k": 4096, "n": 4096},
        # the SwiGLU MLP of a 70B-sized model over 8192 tokens
        {"name": "mlp_prefill", "kind": "mlp", "tokens": 8192, "d": 8192, "ffn": 28672},
        # weight-only 4-bit linear layer: a decode batch of 16 on a checkpoint in its AutoGPTQ layout
        {"name": "w4a16_decode", "kind": "w4a16", "tokens": 16, "k": 8192, "n": 8192, "group": 128, "k_packed": True},
        # the same with a larger, ragged decode batch, weights repacked once into the operator layout
        {"name": "w4a16_batch", "kind": "w4a16", "tokens": 77, "k": 8192, "n": 8192, "group": 128, "k_packed": False},
        # the same over a prompt
        {"name": "w4a16_prefill", "kind": "w4a16", "tokens": 2048, "k": 8192, "n": 8192, "group": 128, "k_packed": False},
        # causal self-attention over two prompts of 8192 tokens, eight query heads on one key/value head
        {"name": "attention_prefill", "kind": "attention", "batch": 2, "kv_heads": 1, "group_heads": 8, "tokens": 8192, "causal": True},
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(v) // multiple * multiple)


def draw(rng):
    kind = rng.choice([c["kind"] for c in listed()])  # as often as it is listed
    if kind == "quantize":
        # any row length: hidden sizes are multiples of 8, flattened parameter buffers are not
        cols = _log_int(rng, 512, 16384, rng.choice([1, 8, 64, 128]))
        rows = max(1, min(_log_int(rng, 1, 16384), (1 << 26) // cols))
        dst = rng.choice(["e4m3", "e5m2"])
        return {"kind": kind, "rows": rows, "cols": cols, "src": rng.choice(["bf16", "bf16", "f32"]), "dst": dst,
                "stochastic": dst == "e5m2" and rng.random() < 0.5}
    if kind == "kv_cache":
        return {"kind": kind, "batch": rng.randint(1, 4), "tokens": _log_int(rng, 16, 8192), "heads": rng.choice([1, 2, 4, 8])}
    if kind == "expand_int4":
        return {"kind": kind, "k": _log_int(rng, 1024, 8192, 128), "n": _log_int(rng, 1024, 8192, 64), "group": rng.choice([64, 128]),
                "signed": rng.random() < 0.3, "zero_points": rng.random() < 0.7}
    if kind == "linear":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096), "k": _log_int(rng, 1024, 8192, 16), "n": _log_int(rng, 1024, 14336, 8),
                "bias": rng.random() < 0.5}
    if kind == "linear_backward":
        return {"kind": kind, "tokens": _log_int(rng, 256, 8192), "k": _log_int(rng, 1024, 8192, 64), "n": _log_int(rng, 1024, 8192, 64)}
    if kind == "mlp":
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "d": rng.choice([4096, 5120, 8192]), "ffn": _log_int(rng, 3584, 28672, 128)}
    if kind == "w4a16":
        tokens = _log_int(rng, 1, 2048)
        return {"kind": kind, "tokens": tokens, "k": _log_int(rng, 1024, 8192, 128), "n": _log_int(rng, 1024, 14336, 64),
                "group": rng.choice([64, 128]), "k_packed": tokens <= 16 and rng.random() < 0.5}
    return {"kind": "attention", "batch": rng.randint(1, 2), "kv_heads": rng.choice([1, 2]), "group_heads": rng.choice([1, 4, 8]),
            "tokens": _log_int(rng, 256, 8192), "causal": rng.random() < 0.75}


# ----------------------------------------------------------------------------- inputs
def _randn(gen, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, device="cuda", generator=gen, dtype=F32) * std).to(dtype)


def _scalar(v):
    return torch.tensor(float(v), device="cuda", dtype=F32)


def _weight8(gen, n, k, std=0.02):
    """e4m3 [n, k] with one scale per output channel, and scale_inv [n].  In blocks of rows, so that the largest
    weights need no fp32 copy of themselves."""
    w8 = torch.empty(n, k, device="cuda", dtype=E4M3)
    inv = torch.empty(n, device="cuda", dtype=F32)
    for lo in range(0, n, 4096):
        w = torch.randn(min(4096, n - lo), k, device="cuda", generator=gen, dtype=F32) * std
        s = w.abs().amax(dim=1) / 448.0
        inv[lo:lo + 4096] = s
        w8[lo:lo + 4096] = (w / s[:, None]).to(E4M3)
    return w8, inv


def _int4_weight(gen, k, n, group, k_packed=False, zero_points=True):
    def words(*shape):
        return torch.randint(-2 ** 31, 2 ** 31 - 1, shape, device="cuda", dtype=torch.int32, generator=gen)

    qw = words(k // 8, n) if k_packed else words(k, n // 8)
    scales = (torch.rand(k // group, n, device="cuda", generator=gen) * 0.015 + 0.005).to(BF16)
    return qw, scales, words(k // group, n // 8) if zero_points else None


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    c, kind, s = case, case["kind"], {"case": case, "seed": int(seed)}
    if kind == "quantize":
        gradient = c["dst"] == "e5m2"
        s["x"] = _randn(gen, c["rows"], c["cols"], std=1e-3 if gradient else 1.0, dtype=FLOAT[c["src"]])
        s["scale"] = _scalar(2.0 ** 23 if gradient else 64.0)  # delayed scaling: the scale is known before the cast
    elif kind == "kv_cache":
        s["kv"] = _randn(gen, 2, c["batch"], c["tokens"], c["heads"], HEAD_DIM)
        s["scale"], s["scale_inv"] = _scalar(448.0 / 6.0), _scalar(6.0 / 448.0)
    elif kind == "expand_int4":
        s["qw"], s["scales"], s["zp"] = _int4_weight(gen, c["k"], c["n"], c["group"], zero_points=c["zero_points"])
    elif kind == "linear":
        s["x"] = _randn(gen, c["tokens"], c["k"])
        s["w8"], s["w_inv"] = _weight8(gen, c["n"], c["k"])
        s["scale"], s["scale_inv"] = _scalar(448.0 / 6.0), _scalar(6.0 / 448.0)
        s["bias"] = _randn(gen, c["n"], std=0.01) if c["bias"] else None
    elif kind == "linear_backward":
        s["dy8"] = _randn(gen, c["tokens"], c["n"], std=8192.0, dtype=E5M2)
        s["x8"] = _randn(gen, c["tokens"], c["k"], std=74.0, dtype=E4M3)
        s["w8"] = _randn(gen, c["n"], c["k"], std=100.0, dtype=E4M3)
        s["dy_inv"], s["x_inv"], s["w_inv"] = _scalar(2.0 ** -23), _scalar(1 / 74.0), _scalar(2e-4)
        s["main_grad"] = _randn(gen, c["n"], c["k"], std=1e-2, dtype=F32)
    elif kind == "mlp":
        gate_up, gate_up_inv = _weight8(gen, 2 * c["ffn"], c["d"])
        down, down_inv = _weight8(gen, c["d"], c["ffn"])
        # random weights: their rows are already in the interleaved gate/up order
        shard = tp_mlp.MlpShard(gate_up, gate_up_inv, down, down_inv, c["ffn"])
        s["mlp"] = tp_mlp.TpFp8Mlp(shard, 448.0 / 6.0, 448.0 / 16.0, fused_gate_up=True)
        s["x"] = _randn(gen, c["tokens"], c["d"])
    elif kind == "w4a16":
        s["x"] = _randn(gen, c["tokens"], c["k"])
        s["qw"], s["scales"], s["zp"] = _int4_weight(gen, c["k"], c["n"], c["group"], c["k_packed"])
    else:
        b, g, r, t = c["batch"], c["kv_heads"], c["group_heads"], c["tokens"]
        s["q"] = _randn(gen, b, g, r, t, HEAD_DIM, std=74.0, dtype=E4M3)
        s["k"] = _randn(gen, b, g, 1, t, HEAD_DIM, std=74.0, dtype=E4M3)
        s["v"] = _randn(gen, b, g, 1, t, HEAD_DIM, std=74.0, dtype=E4M3)
        s["inv"] = torch.full((1,), 1 / 74.0, device="cuda")
        s["p_scale"], s["p_inv"] = torch.full((1,), 256.0, device="cuda"), torch.full((1,), 1 / 256.0, device="cuda")
    return s


# ----------------------------------------------------------------------------- one pass
def run(state):
    s, c = state, state["case"]
    kind, hpu = c["kind"], torch.ops.hpu
    if kind == "quantize":
        if c["stochastic"]:
            b200_hpu_ops.set_sr_seed(s["seed"])  # a step that is repeated rounds alike
        return hpu.cast_to_fp8_v2(s["x"], s["scale"], c["stochastic"], True, FP8[c["dst"]])
    if kind == "kv_cache":
        cache, _ = hpu.cast_to_fp8_v2(s["kv"], s["scale"], False, False, E4M3)
        return cache, hpu.cast_from_fp8(cache, s["scale_inv"], BF16)
    if kind == "expand_int4":
        op = hpu.convert_from_int4 if c["signed"] else hpu.convert_from_uint4
        return op(s["qw"], s["scales"], s["zp"], BF16)
    if kind == "linear":
        x8, _ = hpu.cast_to_fp8_v2(s["x"], s["scale"], False, False, E4M3)
        return hpu.fp8_gemm_v2(x8, False, s["w8"], True, None, BF16, s["scale_inv"], s["w_inv"], s["bias"], False, [1, c["n"]])
    if kind == "linear_backward":
        dx = hpu.fp8_gemm_v2(s["dy8"], False, s["w8"], False, None, BF16, s["dy_inv"], s["w_inv"])
        dw = hpu.fp8_gemm_v2(s["dy8"], True, s["x8"], False, s["main_grad"], F32, s["dy_inv"], s["x_inv"], None, True)
        return dx, dw
    if kind == "mlp":
        return s["mlp"](s["x"])
    if kind == "w4a16":
        return torch.ops.b200q.w4a16_gemm(s["x"], s["qw"], s["scales"], s["zp"], c["group"], c["k_packed"], BF16)
    inv = s["inv"]
    return hpu.fp8_sdpa_recomp_fwd(s["q"], s["k"], s["v"], None, 0.0, 1.0 / math.sqrt(HEAD_DIM), c["causal"], False, "None", inv, inv, inv,
                                   s["p_scale"], None, s["p_inv"], False, False, None, "left")[0]


# ----------------------------------------------------------------------------- what a pass cannot do without
def _int4_bytes(c, zero_points=True):
    groups = c["k"] // c["group"]
    return c["k"] * c["n"] // 2 + 2 * groups * c["n"] + (groups * c["n"] // 2 if zero_points else 0)


def work(case):
    c, kind = case, case["kind"]
    if kind == "quantize":
        n = c["rows"] * c["cols"]
        return {"bytes": n * (3 if c["src"] == "bf16" else 5) + 8, "flops": 0}
    if kind == "kv_cache":
        return {"bytes": 5 * 2 * c["batch"] * c["tokens"] * c["heads"] * HEAD_DIM, "flops": 0}
    if kind == "expand_int4":
        return {"bytes": _int4_bytes(c, c["zero_points"]) + 2 * c["k"] * c["n"], "flops": 0}
    if kind == "linear":
        m, k, n = c["tokens"], c["k"], c["n"]
        return {"bytes": 2 * m * k + n * k + 6 * n + 2 * m * n, "flops": 2 * m * k * n}
    if kind == "linear_backward":
        m, k, n = c["tokens"], c["k"], c["n"]
        return {"bytes": m * n + m * k + n * k + 2 * m * k + 8 * n * k, "flops": 4 * m * k * n}
    if kind == "mlp":
        m, d, f = c["tokens"], c["d"], c["ffn"]
        return {"bytes": 4 * m * d + 3 * d * f + 4 * (2 * f + d), "flops": 6 * m * d * f}
    if kind == "w4a16":
        m, k, n = c["tokens"], c["k"], c["n"]
        return {"bytes": _int4_bytes(c) + 2 * m * k + 2 * m * n, "flops": 2 * m * k * n}
    heads, t = c["batch"] * c["kv_heads"] * c["group_heads"], c["tokens"]
    pairs = t * (t + 1) // 2 if c["causal"] else t * t
    return {"bytes": 3 * heads * t * HEAD_DIM + 2 * c["batch"] * c["kv_heads"] * t * HEAD_DIM, "flops": 4 * heads * pairs * HEAD_DIM}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "kv_cache", "expand_int4"):
        return "exact"  # rounding is defined bit by bit, stochastic rounding by its seed
    if kind in ("linear", "w4a16"):
        return {"rel": 4e-3, "max": 1.6e-2}  # fp32 sums in another order, then one rounding to bf16
    if kind == "linear_backward":
        return {"rel": 4e-3, "max": 1.6e-2}  # as above for the input gradient; the weight gradient stays in fp32
    return {"rel": 1e-2, "max": 0.2}  # an e4m3 intermediate (SwiGLU, probabilities) may round the other way
