"""The workloads that this package's speed is judged by.

Each case is what a program that serves or converts a JANG model has the package do, through the public entry
points: quantized linears from one row to a prefill chunk, a whole decode step as a captured plan, the routed
experts in decode and in prefill, and the converter's quantizer with its dequantizer.  Weights are N(0, 0.02) and
activations N(0, 1), the distributions of the benchmark; sizes are those of the benchmark's model shapes and
sweeps, and ragged ones between them.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass; returns its outputs
    work(case)          bytes and operations one pass cannot do without
    tolerance(case)     how far another correct implementation may be
"""
from __future__ import annotations

import math

import torch

import jangq_b200 as jq
from jangq_b200 import moe
from jangq_b200.stacks import MoEDecodeStack

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # the smallest call: one projection of a small model, one row, eager -- launch and host latency
        {"name": "linear_1x2048x2048_4bit", "kind": "linear", "M": 1, "N": 2048, "K": 2048, "bits": 4, "gs": 64,
         "dtype": "bf16"},
        # one decoded token of a dense decoder at the 8/2/6-bit profile: eight of its layers and the output head as a
        # captured plan over 57 matrices (1 GB of weights, far beyond L2)
        {"name": "decode_step_dense", "kind": "plan", "m": 1, "layers": 8, "hidden": 4096, "inter": 11008,
         "vocab": 32000, "attn_bits": 8, "mlp_bits": 2, "head_bits": 6, "gs": 64},
        # a batch of eight requests in decode, through one wide projection
        {"name": "linear_8x14336x4096_4bit_gs128", "kind": "linear", "M": 8, "N": 14336, "K": 4096, "bits": 4, "gs": 128,
         "dtype": "bf16"},
        # a ragged batch between decode and prefill (speculative decoding, a short chunk)
        {"name": "linear_61x4096x4096_6bit", "kind": "linear", "M": 61, "N": 4096, "K": 4096, "bits": 6, "gs": 64,
         "dtype": "bf16"},
        # a short prompt of odd length, float16 activations, the 8-bit attention width
        {"name": "linear_333x4096x4096_8bit_f16", "kind": "linear", "M": 333, "N": 4096, "K": 4096, "bits": 8, "gs": 64,
         "dtype": "f16"},
        # the 512-token prompt of the dense decoder, one 2-bit MLP projection
        {"name": "linear_512x11008x4096_2bit", "kind": "linear", "M": 512, "N": 11008, "K": 4096, "bits": 2, "gs": 64,
         "dtype": "bf16"},
        # a long prefill chunk, the largest contraction
        {"name": "linear_4096x14336x4096_4bit", "kind": "linear", "M": 4096, "N": 14336, "K": 4096, "bits": 4, "gs": 64,
         "dtype": "bf16"},
        # one decoded token through routed layers (6-bit attention, top-8 of 128 2-bit experts), replayed from a graph
        {"name": "decode_step_moe", "kind": "moe_step", "T": 1, "layers": 8, "hidden": 2048, "experts": 128, "inter": 768,
         "topk": 8, "expert_bits": 2, "attn_bits": 6},
        # sixteen requests in decode through the large routed layer with its shared 8-bit expert, eager
        {"name": "moe_16x4096_512experts_shared", "kind": "moe", "T": 16, "hidden": 4096, "experts": 512, "inter": 1024,
         "topk": 10, "expert_bits": 2, "shared_bits": 8, "gs": 64},
        # a 2048-token prefill through one routed layer, router selection included
        {"name": "moe_2048x2048_128experts", "kind": "moe", "T": 2048, "hidden": 2048, "experts": 128, "inter": 768,
         "topk": 8, "expert_bits": 2, "shared_bits": 0, "gs": 64},
        # the converter: one float16 matrix quantized at 4 bits
        {"name": "quantize_4096x4096_4bit_f16", "kind": "quantize", "N": 4096, "K": 4096, "bits": 4, "gs": 64,
         "dtype": "f16", "mode": "affine"},
        # the loader's way back: packed codes to bfloat16
        {"name": "dequantize_11008x4096_4bit", "kind": "dequantize", "N": 11008, "K": 4096, "bits": 4, "gs": 64,
         "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, lo, hi):
    """A number of weight rows: a multiple of 64 as model dimensions are, or any number (a vocabulary, a shard)."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.4 else max(64, n // 64 * 64)


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["plan", "moe_step", "moe", "moe", "quantize", "dequantize"])
    # every hidden and intermediate size of the benchmark's models is a multiple of 128
    K = _log(rng, 8, 86) * 128
    if kind == "linear":
        N = _rows(rng, 512, 32000)
        most = min(4096, 4096 * 14336 * 4096 // (N * K))
        return {"kind": kind, "M": max(1, min(most, _log(rng, 1, 4096))), "N": N, "K": K,
                "bits": rng.choice([2, 3, 4, 6, 8]), "gs": rng.choice([64, 64, 128]),
                "dtype": rng.choice(["bf16", "bf16", "bf16", "f16"])}
    if kind == "plan":
        return {"kind": kind, "m": rng.choice([1, 1, 1, 2, 4, 8, 16]), "layers": rng.randint(1, 8),
                "hidden": _log(rng, 8, 32) * 128, "inter": _log(rng, 16, 86) * 128, "vocab": _rows(rng, 8000, 32000),
                "attn_bits": rng.choice([4, 6, 8]), "mlp_bits": rng.choice([2, 3, 4]), "head_bits": rng.choice([6, 8]),
                "gs": rng.choice([64, 64, 128])}
    if kind == "moe_step":
        return {"kind": kind, "T": rng.choice([1, 1, 2, 3, 4]), "layers": _log(rng, 2, 8), "hidden": 2048,
                "experts": rng.choice([64, 128]), "inter": _log(rng, 4, 12) * 128, "topk": rng.choice([4, 6, 8]),
                "expert_bits": rng.choice([2, 2, 3, 4]), "attn_bits": rng.choice([4, 6, 8])}
    if kind == "moe":
        return {"kind": kind, "T": _log(rng, 1, 4096), "hidden": _log(rng, 8, 32) * 128,
                "experts": rng.choice([32, 64, 128, 256]), "inter": _log(rng, 4, 8) * 128, "topk": rng.choice([2, 4, 8, 10]),
                "expert_bits": rng.choice([2, 2, 3, 4]), "shared_bits": rng.choice([0, 0, 8]), "gs": rng.choice([64, 64, 128])}
    return {"kind": kind, "N": _rows(rng, 256, 12288), "K": K, "bits": rng.choice([2, 3, 4, 6, 8]),
            "gs": rng.choice([64, 64, 128]), "dtype": rng.choice(["f16", "bf16"]),
            "mode": rng.choice(["affine", "affine", "rtn"]) if kind == "quantize" else "affine"}


# ---- inputs ------------------------------------------------------------------------------------------

def _normal(gen, shape, dtype, scale=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * scale).to(dtype)


def _linear(gen, n, k, bits, gs, dtype=torch.bfloat16):
    return jq.JANGLinear.from_float(_normal(gen, (n, k), dtype, 0.02), bits=bits, group_size=gs).freeze()


def _bank(gen, experts, n, k, bits, gs):
    parts = []
    step = max(1, (1 << 28) // (n * k))          # about a gigabyte of float32 at a time
    for e in range(0, experts, step):
        w = _normal(gen, (min(step, experts - e), n, k), torch.bfloat16, 0.02)
        parts.append(jq.quantize(w, gs, bits))
    wq, s, b = (torch.cat(p) for p in zip(*parts))
    return jq.ExpertBank(wq, s, b, bits, gs)


def _plan_shapes(c):
    """(N, K, bits) of the plan's matrices and the groups that read the same activations."""
    mats, groups = [], []
    h, i = c["hidden"], c["inter"]
    for _ in range(c["layers"]):
        b = len(mats)
        mats += [(h, h, c["attn_bits"])] * 4 + [(i, h, c["mlp_bits"])] * 2 + [(h, i, c["mlp_bits"])]
        groups += [[b, b + 1, b + 2], [b + 3], [b + 4, b + 5], [b + 6]]
    mats.append((c["vocab"], h, c["head_bits"]))
    groups.append([len(mats) - 1])
    return mats, groups


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = c["kind"]
    if kind == "linear":
        dt = DTYPES[c["dtype"]]
        return {"kind": kind, "module": _linear(gen, c["N"], c["K"], c["bits"], c["gs"], dt),
                "x": _normal(gen, (c["M"], c["K"]), dt)}
    if kind == "plan":
        mats, groups = _plan_shapes(c)
        plan = jq.GemvPlan([_linear(gen, n, k, b, c["gs"]) for n, k, b in mats], m=c["m"], groups=groups)
        for x in {x.data_ptr(): x for x in plan.x}.values():        # linears of one width share their input
            x.copy_(_normal(gen, x.shape, x.dtype))
        return {"kind": kind, "plan": plan.capture()}
    if kind == "moe_step":
        stack = MoEDecodeStack(layers=c["layers"], hidden=c["hidden"], experts=c["experts"], inter=c["inter"],
                               topk=c["topk"], expert_bits=c["expert_bits"], attn_bits=c["attn_bits"], seed=seed)
        x = _normal(gen, (c["T"], c["hidden"]), torch.bfloat16)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            stack.step(x)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = stack.step(x)
        return {"kind": kind, "stack": stack, "x": x, "graph": graph, "out": out}
    if kind == "moe":
        h, i, e = c["hidden"], c["inter"], c["experts"]
        st = {"kind": kind, "k": c["topk"], "x": _normal(gen, (c["T"], h), torch.bfloat16),
              "logits": _normal(gen, (c["T"], e), torch.bfloat16),
              "gate": _bank(gen, e, i, h, c["expert_bits"], c["gs"]), "up": _bank(gen, e, i, h, c["expert_bits"], c["gs"]),
              "down": _bank(gen, e, h, i, c["expert_bits"], c["gs"]), "shared": None}
        if c["shared_bits"]:
            st["shared"] = (_linear(gen, i, h, c["shared_bits"], c["gs"]), _linear(gen, i, h, c["shared_bits"], c["gs"]),
                            _linear(gen, h, i, c["shared_bits"], c["gs"]))
        return st
    dt = DTYPES[c["dtype"]]
    w = _normal(gen, (c["N"], c["K"]), dt, 0.02)
    if kind == "quantize":
        return {"kind": kind, "w": w, "bits": c["bits"], "gs": c["gs"], "mode": c["mode"]}
    return {"kind": kind, "packed": jq.quantize(w, c["gs"], c["bits"]), "bits": c["bits"], "gs": c["gs"]}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["module"](state["x"])
    if kind == "plan":
        return state["plan"].run()
    if kind == "moe_step":
        state["graph"].replay()
        return state["out"]
    if kind == "moe":
        idx, w = moe.route_softmax_topk(state["logits"], state["k"])
        return jq.moe_layer(state["x"], idx, w, state["gate"], state["up"], state["down"], shared=state["shared"],
                            static_weights=True)
    if kind == "quantize":
        return jq.quantize(state["w"], state["gs"], state["bits"], mode=state["mode"])
    wq, s, b = state["packed"]
    return jq.dequantize(wq, s, b, state["gs"], state["bits"])


# ---- what a pass cannot do without --------------------------------------------------------------------

def _weight_bytes(n, k, bits, gs):
    return n * k * bits // 8 + n * (k // gs) * 4


def _experts_hit(tokens, experts, topk):
    """Expected number of distinct experts that `tokens` independent top-k choices name."""
    return experts * (1.0 - (1.0 - topk / experts) ** tokens)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "linear":
        m, n, k = c["M"], c["N"], c["K"]
        return {"bytes": _weight_bytes(n, k, c["bits"], c["gs"]) + 2 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "plan":
        mats, _ = _plan_shapes(c)
        return {"bytes": sum(_weight_bytes(n, k, b, c["gs"]) + 2 * c["m"] * (n + k) for n, k, b in mats),
                "flops": sum(2 * c["m"] * n * k for n, k, _ in mats)}
    if kind in ("moe_step", "moe"):
        t, h, i, e, k = c["T"], c["hidden"], c["inter"], c["experts"], c["topk"]
        gs = c.get("gs", 64)
        hit = _experts_hit(t, e, k)
        nbytes = hit * (2 * _weight_bytes(i, h, c["expert_bits"], gs) + _weight_bytes(h, i, c["expert_bits"], gs))
        flops = 2 * t * k * 3 * h * i
        if kind == "moe_step":
            attn = ((4096, h), (512, h), (512, h), (h, 4096))
            nbytes += sum(_weight_bytes(n, kk, c["attn_bits"], gs) for n, kk in attn) + 2 * e * h
            flops += sum(2 * t * n * kk for n, kk in attn) + 2 * t * e * h
            return {"bytes": int(c["layers"] * nbytes) + 4 * t * h, "flops": c["layers"] * flops}
        if c["shared_bits"]:
            nbytes += 2 * _weight_bytes(i, h, c["shared_bits"], gs) + _weight_bytes(h, i, c["shared_bits"], gs)
            flops += 2 * t * 3 * h * i
        return {"bytes": int(nbytes) + 2 * t * (2 * h + e), "flops": flops}
    n, k = c["N"], c["K"]
    return {"bytes": _weight_bytes(n, k, c["bits"], c["gs"]) + 2 * n * k, "flops": 2 * n * k}


def tolerance(case):
    """Codes, scales and dequantized weights are bit-exact.  The other figures are about four times what the present
    code shows against float64 sums: a product of 16-bit activations is rounded to 16 bits on the way out, and above
    sixteen rows its weights are rounded to 16 bits too."""
    kind = case["kind"]
    if kind in ("quantize", "dequantize"):
        return "exact"
    if kind == "linear":          # bf16: 1.7e-3 (output rounding) to 2.3e-3 (weights rounded as well); f16: 2.9e-4
        return {"rel": 9e-3} if case["dtype"] == "bf16" else {"rel": 1.2e-3}
    if kind == "plan":            # independent products, 1.7e-3 each
        return {"rel": 7e-3}
    if kind == "moe":             # three products and the SwiGLU between them: 3.9e-3 to 4.6e-3
        return {"rel": 1.8e-2}
    # a chain of bf16 layers: two kernels of this package differ by 1.0e-2 after eight layers, and by 4.2e-2 where a
    # near tie of two router logits sends the token to another expert in one of them (one seed of six)
    return {"rel": 6e-2}
