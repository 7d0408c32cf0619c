"""The work a user of this framework has it do, as a list of measurable cases.

Three kinds of user calls: the drop-in operators of ``cinfer_ascendc`` (grouped GEMM for prefill-sized
batches, grouped soft GEMV for decode-sized ones, FP4 -> BF16 dequantisation), called with the tensors an
engine holds, and ``MoELayer.forward``, the whole expert FFN of one layer.  Sizes and value distributions
are those of the benchmark configurations (``ascend_kernel_b200/inputs.py``, ``bench.py``) and of the tests;
``draw`` gives further cases of the same ranges.
"""
import math

import torch

from ascend_kernel_b200 import cinfer_ascendc, fp4_layout, inputs
from ascend_kernel_b200.moe_layer import MoELayer

DEV = "cuda"

# ---- the cases ----------------------------------------------------------------------------------


def _gemm(name, fmt, experts, tokens, top_k, K, N, split="routed"):
    return dict(name=name, op="gemm", fmt=fmt, experts=experts, tokens=tokens, top_k=top_k, K=K, N=N, split=split)


def _gemv(name, fmt, experts, tokens, top_k, K, N):
    return dict(name=name, op="gemv", fmt=fmt, experts=experts, tokens=tokens, top_k=top_k, K=K, N=N, split="routed")


def _layer(name, fmt, experts, tokens, top_k, hidden, inter):
    return dict(name=name, op="layer", fmt=fmt, experts=experts, tokens=tokens, top_k=top_k, hidden=hidden, inter=inter)


def listed():
    return [
        # the smallest call: a few experts and rows of a small model; launches and latency are all there is
        _gemm("gemm_int8_small", "int8", 4, 128, 1, 256, 512),
        # gate/up projection of a full prefill batch, tokens spread over the experts by popularity: the four
        # weight formats an engine loads (per-channel int8, per-group int4, and the reference's own fp8 and fp4)
        _gemm("gemm_int8_prefill", "int8", 256, 8192, 8, 7168, 4096, "zipf"),
        _gemm("gemm_fp8_prefill", "fp8", 256, 8192, 8, 7168, 4096, "zipf"),
        _gemm("gemm_int4_prefill", "int4", 256, 8192, 8, 7168, 4096, "zipf"),
        # down projection of an odd-sized chunk of a chunked prefill, about 32 rows an expert, fp4 as stored
        _gemm("gemm_fp4_chunk", "fp4", 256, 1021, 8, 2048, 7168),
        # gate/up projection of a decode step of 32 sequences
        _gemv("gemv_int8_decode", "int8", 256, 32, 8, 7168, 4096),
        # one sequence being decoded: eight experts with one row each
        _gemv("gemv_fp8_one_token", "fp8", 256, 1, 8, 7168, 4096),
        # down projection of a decode step of an odd number of sequences, fp4 as stored
        _gemv("gemv_fp4_decode", "fp4", 256, 37, 8, 2048, 7168),
        # a layer's fp4 expert weights unpacked to bf16
        dict(name="fp4_dequant", op="dequant", rows=256 * 2048, cols=7168),
        # the whole expert FFN of a layer: prefill on int8 and on fp4-stored experts, and a decode step
        _layer("layer_int8_prefill", "int8", 256, 4096, 8, 7168, 2048),
        _layer("layer_fp4_prefill", "fp4", 256, 4096, 8, 7168, 2048),
        _layer("layer_int8_decode", "int8", 256, 32, 8, 7168, 2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mult(rng, lo, hi, m):
    """A multiple of ``m`` in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, m * int(round(_log_int(rng, lo, hi) / m))))


def draw(rng):
    op = rng.choice(["gemm", "gemm", "gemm", "gemv", "gemv", "layer", "layer", "dequant"])
    if op == "dequant":
        return dict(op="dequant", rows=_log_int(rng, 64, 256 * 2048), cols=_mult(rng, 256, 7168, 32))
    experts = rng.choice([8, 16, 32, 64, 128, 160, 256])
    top_k = rng.choice([k for k in (1, 2, 4, 6, 8) if k <= experts])
    if op == "layer":
        return dict(op="layer", fmt=rng.choice(["int8", "fp4"]), experts=experts, tokens=_log_int(rng, 1, 4096), top_k=top_k,
                    hidden=_mult(rng, 512, 7168, 256), inter=_mult(rng, 256, 2048, 128))
    fmt = rng.choice(["int8", "fp8", "int4", "fp4"] + (["bf16"] if op == "gemm" and experts <= 128 else []))
    K = _mult(rng, 256, 7168, 128)
    N = _mult(rng, 256, min(7168, 7168 * 4096 // K), 128 if fmt == "fp8" else 256)
    if op == "gemm":
        # small batches that still go through the GEMM, up to the prefill batch of the largest case
        tokens, split = _log_int(rng, 16, 8192), rng.choice(["routed", "zipf"])
    else:
        # decode: up to about four rows an expert
        tokens, split = _log_int(rng, 1, min(64, max(1, 4 * experts // top_k))), "routed"
    return dict(op=op, fmt=fmt, experts=experts, tokens=tokens, top_k=top_k, K=K, N=N, split=split)


# ---- inputs -------------------------------------------------------------------------------------


def _bytes(shape, gen):
    """Uniform bytes, eight to a drawn 64-bit integer (every shape here holds a multiple of eight)."""
    n = math.prod(shape)
    r = torch.randint(-(1 << 63), (1 << 63) - 1, (n // 8,), generator=gen, device=DEV, dtype=torch.int64)
    return r.view(torch.uint8).view(*shape)


def _uniform(shape, lo, hi, gen):
    return (torch.rand(shape, generator=gen, device=DEV) * (hi - lo) + lo).to(torch.bfloat16)


def _counts(case, seed, gen):
    """Rows of each expert: by popularity (some experts get none), or every token on top_k different experts."""
    E = case["experts"]
    if case["split"] == "zipf":
        return inputs.zipf_counts(E, case["tokens"] * case["top_k"], 1.2, seed, n_zero=E // 64).to(DEV)
    ids = torch.rand(case["tokens"], E, generator=gen, device=DEV).topk(case["top_k"], dim=1).indices
    return torch.bincount(ids.reshape(-1), minlength=E).to(torch.int64)


def _weights(fmt, G, K, N, gen):
    """(weight, scale, offset) of a format; int8 / int4 with offsets, fp8 / fp4 as the reference defines them."""
    if fmt == "int8":
        return _bytes((G, K, N), gen).view(torch.int8), _uniform((G, N), 0.001, 0.01, gen), _uniform((G, N), -4.0, 4.0, gen)
    if fmt == "int4":
        return (_bytes((G, K, N // 2), gen).view(torch.int8), _uniform((G, K // 128, N), 0.005, 0.05, gen),
                _uniform((G, K // 128, N), -2.0, 2.0, gen))
    if fmt == "fp8":
        return _bytes((G, K, N), gen), torch.randn(G, K // 128, N // 128, generator=gen, device=DEV), None
    if fmt == "fp4":
        return _bytes((G, K, N // 2), gen).view(torch.int8), _uniform((G, K // 16, N), 0.25, 3.25, gen), None
    w = torch.empty(G, K, N, dtype=torch.bfloat16, device=DEV)
    for g in range(G):
        w[g] = torch.randn(K, N, generator=gen, device=DEV) * (K ** -0.5)
    return w, None, None


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    if case["op"] == "dequant":
        R, C = case["rows"], case["cols"]
        out = torch.empty(R, C, dtype=torch.bfloat16, device=DEV)
        scale = torch.randint(119, 128, (R, C // 32), generator=gen, device=DEV, dtype=torch.uint8)
        return dict(op="dequant", args=(_bytes((R, C // 2), gen), scale, out), out=out)
    if case["op"] == "layer":
        E, T, H, I = case["experts"], case["tokens"], case["hidden"], case["inter"]
        if case["fmt"] == "int8":
            w13, s13, o13 = _weights("int8", E, H, 2 * I, gen)
            w2, s2, o2 = _weights("int8", E, I, H, gen)
            layer = MoELayer(w13, s13, o13, w2, s2, o2, E, case["top_k"])
        else:
            w13, w2 = _bytes((E, H, I), gen), _bytes((E, I, H // 2), gen)
            s13 = torch.randint(119, 128, (E, H, 2 * I // 32), generator=gen, device=DEV, dtype=torch.uint8)
            s2 = torch.randint(119, 128, (E, I, H // 32), generator=gen, device=DEV, dtype=torch.uint8)
            layer = MoELayer(w13, s13, None, w2, s2, None, E, case["top_k"], weight_format="fp4")
        x = torch.randn(T, H, generator=gen, device=DEV).to(torch.bfloat16)
        logits = torch.randn(T, E, generator=gen, device=DEV).to(torch.bfloat16)
        return dict(op="layer", layer=layer, x=x, logits=logits)
    G, K, N, fmt = case["experts"], case["K"], case["N"], case["fmt"]
    counts = _counts(case, seed, gen)
    M = case["tokens"] * case["top_k"]
    x = torch.randn(M, K, generator=gen, device=DEV).to(torch.bfloat16)
    w, scale, offset = _weights(fmt, G, K, N, gen)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    if fmt in ("fp8", "fp4"):  # the reference's formats come with its group list: cumulative row counts
        kw, gl = {}, counts.cumsum(0)
    else:
        kw, gl = dict(group_list_type=1), counts
    if fmt == "fp4":  # in the order the reference stores them, which the operators read in place
        w = fp4_layout(w, to_ascend=True)
    none = torch.empty(0, dtype=torch.bfloat16, device=DEV)
    if case["op"] == "gemm":
        args = (x, w, none if scale is None else scale, none if offset is None else offset, gl, fmt, out)
    else:
        args = (x, w, scale, gl, fmt, out)  # decode weights without offsets
    return dict(op=case["op"], args=args, kw=kw, out=out)


def run(state):
    op = state["op"]
    if op == "gemm":
        cinfer_ascendc.grouped_gemm(*state["args"], **state["kw"])
    elif op == "gemv":
        cinfer_ascendc.grouped_soft_gemv(*state["args"], **state["kw"])
    elif op == "dequant":
        cinfer_ascendc.fp4_dequant(*state["args"])
    else:
        return state["layer"].forward(state["x"], state["logits"])
    return state["out"]


# ---- what a pass cannot do without ----------------------------------------------------------------


def _weight_bytes(fmt, K, N):
    """Bytes of one expert's weights and scales."""
    return {"int8": K * N + 4 * N, "int4": K * N // 2 + 4 * (K // 128) * N, "fp8": K * N + 4 * (K // 128) * (N // 128),
            "fp4": K * N // 2 + 2 * (K // 16) * N, "bf16": 2 * K * N}[fmt]


def _active(case):
    """Experts that get at least one row (expected number)."""
    E, T, k = case["experts"], case["tokens"], case["top_k"]
    if case.get("split") == "zipf":
        return min(E - E // 64, T * k)
    return E * (1.0 - (1.0 - k / E) ** T)


def work(case):
    if case["op"] == "dequant":
        n = case["rows"] * case["cols"]
        return dict(bytes=n * (0.5 + 1 / 32 + 2), flops=0)
    act = _active(case)
    if case["op"] == "layer":
        E, T, k, H, I = case["experts"], case["tokens"], case["top_k"], case["hidden"], case["inter"]
        if case["fmt"] == "int8":
            w = _weight_bytes("int8", H, 2 * I) + _weight_bytes("int8", I, H)
        else:
            w = 3 * H * I * (0.5 + 1 / 32)
        return dict(bytes=act * w + 2 * T * (2 * H + E), flops=6 * T * k * H * I)
    K, N, M = case["K"], case["N"], case["tokens"] * case["top_k"]
    return dict(bytes=act * _weight_bytes(case["fmt"], K, N) + 2 * M * (K + N), flops=2 * M * K * N)


def tolerance(case):
    if case["op"] == "dequant":
        return "exact"  # every value is representable
    # Against sums in 64 bits (small cases of every format): the operators' one rounding to bf16 of an fp32 sum shows
    # rel 1.66e-3, max 3.9e-3 (half a bf16 step); the layer, which rounds gate, up, activation, expert result and
    # weighted sum, rel 3.7e-3, max 2.1e-2.  Four times that:
    if case["op"] == "layer":
        return {"rel": 1.4e-2, "max": 8e-2}
    return {"rel": 6.6e-3, "max": 1.6e-2}
