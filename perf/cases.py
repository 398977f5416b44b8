"""The work a user of this library has it do, as cases that can be timed and compared.

A case is one pass through the C ABI of include/limn_b200.h (by way of `limn_b200._lib`, the binding every host
here uses): either a "forward" (sdpa) or a "step" (sdpa, sdpa_bwd_q_fused, sdpa_bwd_kv: what a training step calls
per attention layer). `listed()` names the ordinary ones, `draw()` makes more of the same kinds over their ranges.
"""

from __future__ import annotations

import ctypes
import math

import torch

from limn_b200._lib import DTYPE_CODES, check, lib

TORCH = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
BTHD = 1  # LIMN_B200_BTHD


def _case(kind, dtype, batch, heads, t_q, t_k, hd, *, causal, layout="dense", shortest=1.0, mul=1.0):
    """`layout`: "dense" (batch, heads, t, hd) operands; "token_major" (batch, t, heads, hd) operands; "projection":
    q, k and v are slices of one (batch, t, 3, heads, hd) tensor, results token-major. `shortest` < 1: a padded
    batch under a key mask whose sequences are between shortest * t_k and t_k long. `mul` scales q and k."""
    return {"kind": kind, "dtype": dtype, "batch": batch, "heads": heads, "t_q": t_q, "t_k": t_k, "hd": hd,
            "causal": causal, "layout": layout, "shortest": shortest, "mul": mul}


def listed() -> list[dict]:
    named = {
        # the smallest training call: the shape the CPU devices are checked on (1, 2, 128, 32), limn's default dtype
        "first_step_f32": _case("step", "float32", 1, 2, 128, 128, 32, causal=True),
        # one layer of the byte-level GPT (6 layers, d_model 512) kept in limn's default dtype
        "gpt_layer_f32": _case("step", "float32", 32, 8, 256, 256, 64, causal=True),
        # limn's long-context training example: 8192 tokens, 6 heads of 32
        "long_context_f32": _case("step", "float32", 1, 6, 8192, 8192, 32, causal=True),
        # generation with a model in the dtype it was trained in: one new token against a cache with empty slots
        "decode_one_request_f32": _case("forward", "float32", 1, 8, 1, 1999, 64, causal=False, shortest=0.75),
        # the same GPT layer with 16-bit attention operands, read where the projection left them
        "gpt_layer_bf16": _case("step", "bfloat16", 32, 8, 256, 256, 64, causal=True, layout="projection"),
        # long-context prefill of a batch, the forward's headline workload
        "prefill_4k_bf16": _case("forward", "bfloat16", 8, 32, 4096, 4096, 128, causal=True, mul=0.5),
        # prefill of a single prompt of a length nobody chose: few problems, ragged last tile
        "prompt_1000_bf16": _case("forward", "bfloat16", 1, 32, 1000, 1000, 128, causal=True),
        # training an encoder at 2k tokens
        "encoder_2k_bf16": _case("step", "bfloat16", 16, 16, 2048, 2048, 64, causal=False),
        # a padded batch of sentences through an encoder in half precision, operands token-major, key mask
        "padded_batch_f16": _case("step", "float16", 16, 12, 500, 500, 64, causal=False, layout="token_major", shortest=0.5),
        # ragged long training sequence with a sharp softmax
        "ragged_3000_bf16": _case("step", "bfloat16", 4, 40, 3000, 3000, 128, causal=True, mul=2.0),
        # a decoder's cross attention over an encoder's output: rectangular, both directions
        "cross_attention_bf16": _case("step", "bfloat16", 4, 16, 100, 1500, 64, causal=False),
        # batched generation: one new token per sequence against 4096 cached ones
        "decode_batch_bf16": _case("forward", "bfloat16", 8, 32, 1, 4096, 128, causal=False),
    }
    return [{"name": name, **case} for name, case in named.items()]


def _flops(case) -> float:
    """Two products forward, five backward, on the keys a row sees."""
    seen = case["t_k"] * (1.0 + case["shortest"]) / 2.0
    if case["causal"]:
        seen = (case["t_q"] + 1) / 2.0
    products = 7 if case["kind"] == "step" else 2
    return products * 2.0 * case["batch"] * case["heads"] * case["t_q"] * seen * case["hd"]


_MOST = {"float32": 90e9, "float16": 1.2e12, "bfloat16": 1.2e12}  # flops of the largest listed case of the dtype
_MOST_BYTES = 1 << 30


def draw(rng) -> dict:
    """One more case of the ranges above: the kind first, then sizes over their logarithm, odd ones among them."""

    def between(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    while True:
        kind = rng.choice(["train_16", "train_16", "train_f32", "prefill", "decode", "cross"])
        half = rng.choice(["bfloat16", "bfloat16", "float16"])
        if kind == "train_16":
            t = between(64, 4096)
            padded = rng.random() < 0.3
            case = _case("step", half, between(1, 32), rng.choice([4, 6, 8, 12, 16, 32]), t, t, rng.choice([32, 64, 64, 80, 128]),
                         causal=not padded and rng.random() < 0.6,
                         layout=rng.choice(["dense", "token_major"]) if padded else rng.choice(["dense", "token_major", "projection"]),
                         shortest=0.5 if padded else 1.0, mul=rng.choice([0.5, 1.0, 2.0]))
        elif kind == "train_f32":
            t = between(32, 8192)
            padded = rng.random() < 0.25
            case = _case("step", "float32", between(1, 32), rng.choice([2, 4, 6, 8, 12]), t, t, rng.choice([16, 32, 64, 64, 100, 128]),
                         causal=not padded, shortest=0.5 if padded else 1.0, mul=rng.choice([0.5, 1.0]))
        elif kind == "prefill":
            t = between(100, 8192)
            case = _case("forward", rng.choice([half, half, "float32"]), between(1, 16), rng.choice([8, 16, 32]), t, t,
                         rng.choice([64, 96, 128]), causal=True, mul=rng.choice([0.5, 1.0]))
        elif kind == "decode":
            case = _case("forward", rng.choice([half, half, "float32"]), between(1, 32), rng.choice([8, 16, 32]), rng.choice([1, 1, 1, 2, 4]),
                         between(64, 8192), rng.choice([64, 128]), causal=False, shortest=rng.choice([0.75, 1.0]))
        else:
            case = _case("step", rng.choice([half, half, "float32"]), between(1, 16), rng.choice([8, 12, 16]), between(16, 512), between(64, 4096),
                         rng.choice([64, 64, 128]), causal=False, shortest=rng.choice([0.5, 1.0]))
        if _flops(case) <= _MOST[case["dtype"]] and work(case)["bytes"] <= _MOST_BYTES:
            return case


def prepare(case, seed):
    """Operands drawn from the seed, and the result buffers a host's pool hands out. A decode step's cache slots, a
    batch's padding and the scale of q and k are as `case` says."""
    device = torch.device("cuda")
    gen = torch.Generator(device=device).manual_seed(int(seed))
    dtype = TORCH[case["dtype"]]
    b, h, t_q, t_k, hd = (case[key] for key in ("batch", "heads", "t_q", "t_k", "hd"))

    def normal(*shape):
        return torch.randn(shape, generator=gen, device=device)

    def rows(t):
        return (b, h, t, hd) if case["layout"] == "dense" else (b, t, h, hd)

    state = {"case": case, "seed": seed}
    if case["layout"] == "projection":
        qkv = normal(b, t_q, 3, h, hd)
        qkv[:, :, :2] *= case["mul"]
        state["qkv"] = qkv.to(dtype)
        slices = [state["qkv"][:, :, i] for i in range(3)]
        state["q"], state["k"], state["v"] = slices
        view = (t_q * 3 * h * hd, hd, 3 * h * hd)
        major = (t_q * h * hd, hd, h * hd)

        def strides(*triples):
            flat = [x for triple in triples for x in triple]
            return (ctypes.c_longlong * len(flat))(*flat)

        state["strides"] = {"fwd": strides(view, view, view, major), "dq": strides(view, view, view, major, major, major),
                            "dkv": strides(view, view, view, major, major, major)}
    else:
        state["q"] = (normal(*rows(t_q)) * case["mul"]).to(dtype)
        state["k"] = (normal(*rows(t_k)) * case["mul"]).to(dtype)
        state["v"] = normal(*rows(t_k)).to(dtype)
    state["mask"] = None
    if case["shortest"] < 1.0:
        low = max(1, math.ceil(case["shortest"] * t_k))
        lengths = torch.randint(low, t_k + 1, (b, 1, 1), generator=gen, device=device)
        seen = torch.arange(t_k, device=device)[None, None, :] < lengths
        state["mask"] = seen.expand(b, h, t_k).to(dtype).contiguous()
    state["out"] = torch.empty(rows(t_q), dtype=dtype, device=device)
    state["lse"] = torch.empty((b, h, t_q), dtype=torch.float32, device=device)
    if case["kind"] == "step":
        state["do"] = normal(*rows(t_q)).to(dtype)
        state["delta"] = torch.empty((b, h, t_q), dtype=torch.float32, device=device)
        state["dq"] = torch.empty(rows(t_q), dtype=dtype, device=device)
        state["dk"], state["dv"] = (torch.empty(rows(t_k), dtype=dtype, device=device) for _ in range(2))
    return state


def run(state):
    """One pass on the current stream, as a host's plan makes it: one call for a forward, three for a step."""
    case, L = state["case"], lib()
    stream = torch.cuda.current_stream().cuda_stream
    b, h, t_q, t_k, hd = (case[key] for key in ("batch", "heads", "t_q", "t_k", "hd"))
    code, causal, scale = DTYPE_CODES[case["dtype"]], int(case["causal"]), hd**-0.5
    q, k, v, out, lse = (state[key].data_ptr() for key in ("q", "k", "v", "out", "lse"))
    mask = state["mask"].data_ptr() if state["mask"] is not None else None
    if case["layout"] == "dense":
        fwd, dq_pass, dkv_pass = L.limn_b200_sdpa_fwd, L.limn_b200_sdpa_bwd_q_fused, L.limn_b200_sdpa_bwd_kv
        tails = [(code, b * h, t_q, t_k, hd, hd, causal, scale, stream)] * 3
    elif case["layout"] == "token_major":
        fwd, dq_pass, dkv_pass = L.limn_b200_sdpa_fwd_layout, L.limn_b200_sdpa_bwd_q_fused_layout, L.limn_b200_sdpa_bwd_kv_layout
        tails = [(BTHD, code, b, h, t_q, t_k, hd, hd, causal, scale, stream)] * 3
    else:
        fwd, dq_pass, dkv_pass = L.limn_b200_sdpa_fwd_strided, L.limn_b200_sdpa_bwd_q_fused_strided, L.limn_b200_sdpa_bwd_kv_strided
        tails = [(state["strides"][key], code, b, h, t_q, t_k, hd, hd, causal, scale, stream) for key in ("fwd", "dq", "dkv")]
    check(fwd(q, k, v, mask, out, lse, *tails[0]), "sdpa")
    if case["kind"] == "forward":
        return {"out": state["out"], "lse": state["lse"]}
    do, delta, dq, dk, dv = (state[key].data_ptr() for key in ("do", "delta", "dq", "dk", "dv"))
    check(dq_pass(q, k, v, out, do, lse, mask, dq, delta, *tails[1]), "sdpa_bwd_q_fused")
    check(dkv_pass(q, k, v, do, lse, delta, mask, dk, dv, *tails[2]), "sdpa_bwd_kv")
    return {key: state[key] for key in ("out", "lse", "delta", "dq", "dk", "dv")}


def work(case) -> dict:
    """Every operand read and every result written once; the products over the keys a row sees."""
    problems, size = case["batch"] * case["heads"], TORCH[case["dtype"]].itemsize
    q_rows, k_rows, hd = problems * case["t_q"], problems * case["t_k"], case["hd"]
    nbytes = (2 * q_rows + 2 * k_rows) * hd * size + 4 * q_rows
    if case["shortest"] < 1.0:
        nbytes += k_rows * size
    if case["kind"] == "step":
        nbytes += (2 * q_rows + 2 * k_rows) * hd * size + 4 * q_rows
    return {"bytes": nbytes, "flops": _flops(case)}


def tolerance(case) -> dict:
    """About four times what the kernels show against a float64 evaluation of the same inputs: 2.1e-6 at worst in
    float32 (dK and dV of 8192 queries), 4.9e-4 in float16 and 3.9e-3 in bfloat16 (dQ under a sharp softmax)."""
    return {"rel": {"float32": 1e-5, "float16": 2e-3, "bfloat16": 1e-2}[case["dtype"]]}
