"""Performance cases: what a user of the package has it do, through its public entry points, over the sizes it is
used at.  Every case is one pass of one path:

    moe        a fused FP8 MoE layer: routing, then DlblasTritonFusedMoEBlockedF8Impl.forward (prefill and small batches)
    decode     one decode step of the masked-layout layer: routing, then FusedMoELowLatency.forward
    linear     a block-scaled FP8 linear layer: per_token_group_quant_fp8 of the activations, then fp8_gemm
    gating     dlblas_b200.topk_gating, forward, and forward + backward
    permute    the training permutation: permute, unpermute and the gradients of both
    m_grouped  the 16-bit grouped GEMM over ragged row groups (forward of a grouped linear layer)
    k_grouped  its weight gradient
    moe16      the vLLM-style unquantised fused_moe
    route      grouped top-k routing and the block-aligned token layout built from its ids

Sizes are those of the package's own configurations, tests and benchmark (the DeepSeek-V3- and Mixtral-shaped layers,
the dense FP8 sweep, the routing, gating and grouped-GEMM shapes), and generic ones between and beside them.
"""
import math

import numpy as np
import torch

import dlblas_b200
from dlblas_b200 import ops
from dlblas_b200.kernels.fp8 import per_token_group_quant_fp8
from dlblas_b200.kernels.fp8_gemm import fp8_gemm
from dlblas_b200.kernels.fused_moe_v2 import fused_moe
from dlblas_b200.kernels.grouped_gemm.BF16 import k_grouped_gemm, m_grouped_gemm
from dlblas_b200.kernels.moe import biased_grouped_topk
from dlblas_b200.kernels.moe_align_block_size import moe_align_block_size
from dlblas_b200.kernels.permute import permute, unpermute
from dlblas_b200.layers.moe.ep_moe import DlblasTritonFusedMoEBlockedF8Impl, FusedMoELowLatency

# fp8_gemm returns torch's default dtype: a serving process sets it once, at start-up
torch.set_default_dtype(torch.bfloat16)

DEV = "cuda"
FP8 = torch.float8_e4m3fn
ZIPF = 1.2      # skew of the experts' popularity in a decode step
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # a handful of requests through a small expert layer: launches and host work are what it costs
        {"name": "moe small", "kind": "moe", "tokens": 64, "hidden": 512, "inter": 1024, "experts": 8, "top_k": 2,
         "routing": "softmax", "dtype": "bf16"},
        # prefill of a Mixtral-8x7B-shaped layer: few large experts, long row segments
        {"name": "moe mixtral prefill", "kind": "moe", "tokens": 4096, "hidden": 4096, "inter": 14336, "experts": 8,
         "top_k": 2, "routing": "softmax", "dtype": "bf16"},
        # prefill of a DeepSeek-V3-shaped layer: many experts, ragged segments of about 256 rows
        {"name": "moe deepseek prefill", "kind": "moe", "tokens": 8192, "hidden": 7168, "inter": 2048, "experts": 256,
         "top_k": 8, "routing": "grouped", "dtype": "bf16"},
        # one decode step of the same layer, expert popularity skewed like Zipf(1.2)
        {"name": "decode deepseek", "kind": "decode", "tokens": 128, "hidden": 7168, "inter": 2048, "experts": 256,
         "top_k": 8},
        # a linear layer in decode (batch not a multiple of anything) ...
        {"name": "linear decode", "kind": "linear", "tokens": 100, "n": 7168, "k": 2048, "dtype": "bf16"},
        # ... and in prefill
        {"name": "linear prefill", "kind": "linear", "tokens": 8192, "n": 4096, "k": 7168, "dtype": "bf16"},
        # capacity-limited gating of a training step, with the gradients of the auxiliary loss and of the weights
        {"name": "gating train", "kind": "gating", "tokens": 4096, "experts": 64, "top_k": 8, "capacity": 1.0,
         "dtype": "fp32", "train": True},
        # token permutation of a training step, both directions, forward and backward; some slots are dropped
        {"name": "permute train", "kind": "permute", "tokens": 8192, "hidden": 4096, "experts": 64, "top_k": 8,
         "dropped": 0.05, "dtype": "bf16"},
        # grouped linear layer in training: forward over ragged groups, weights as [groups, k, n] ...
        {"name": "grouped forward", "kind": "m_grouped", "rows": 16384, "groups": 16, "n": 4096, "k": 3072,
         "trans_b": False, "dtype": "bf16"},
        # ... and its weight gradient
        {"name": "grouped weight gradient", "kind": "k_grouped", "rows": 40001, "groups": 32, "m": 1536, "n": 2048,
         "dtype": "bf16"},
        # unquantised expert layer of a small model, a mid-sized batch
        {"name": "moe 16-bit", "kind": "moe16", "tokens": 500, "hidden": 2048, "inter": 1024, "experts": 64, "top_k": 6,
         "dtype": "fp16"},
        # grouped routing of a large batch and the block-aligned layout made from its ids
        {"name": "route and align", "kind": "route", "tokens": 20000, "experts": 256, "groups": 8, "topk_group": 4,
         "top_k": 8, "block": 64, "dtype": "fp32"},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, evenly spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi, step=128):
    """A matrix dimension: a multiple of `step`, spread over its logarithm."""
    return max(lo, min(hi, _log(rng, lo, hi) // step * step))


KINDS = ("moe", "decode", "linear", "gating", "permute", "m_grouped", "k_grouped", "moe16", "route")


def draw(rng):
    kind = rng.choice(KINDS)
    while True:
        case = _draw(rng, kind)
        if _seconds(case) <= 1.75e-3:                    # no more than the largest listed one
            return case


def _draw(rng, kind):
    half = rng.choice(("bf16", "bf16", "fp16"))
    if kind == "moe":
        experts = rng.choice((8, 16, 32, 64, 128, 256))
        return {"kind": kind, "tokens": _log(rng, 1, 8192), "hidden": _width(rng, 512, 7168),
                "inter": _width(rng, 512, 14336), "experts": experts, "top_k": rng.choice((1, 2, 4, 6, 8)),
                "routing": "grouped" if experts >= 64 and rng.random() < 0.5 else "softmax", "dtype": half}
    if kind == "decode":
        return {"kind": kind, "tokens": _log(rng, 1, 128), "hidden": _width(rng, 1024, 7168),
                "inter": _width(rng, 512, 2048), "experts": rng.choice((32, 64, 128, 256)),
                "top_k": rng.choice((2, 4, 6, 8))}
    if kind == "linear":
        return {"kind": kind, "tokens": _log(rng, 1, 8192), "n": _width(rng, 512, 24576, 64),
                "k": _width(rng, 512, 7168), "dtype": half}
    if kind == "gating":
        experts = rng.choice((8, 16, 32, 64, 128, 256))
        top_k = rng.choice((1, 2, 4, 8))
        return {"kind": kind, "tokens": _log(rng, 64, 16384), "experts": experts, "top_k": top_k,
                "capacity": 1.0 if top_k * 1.5 > experts else rng.choice((1.0, 1.25, 1.5)),
                "dtype": rng.choice(("fp32", "fp16")), "train": rng.random() < 0.7}
    if kind == "permute":
        return {"kind": kind, "tokens": _log(rng, 64, 16384), "hidden": _width(rng, 512, 7168),
                "experts": rng.choice((8, 16, 64, 128, 256)), "top_k": rng.choice((1, 2, 4, 6, 8)),
                "dropped": rng.choice((0.0, 0.05, 0.3)), "dtype": rng.choice(("bf16", "bf16", "fp16", "fp32"))}
    if kind == "m_grouped":
        return {"kind": kind, "rows": _log(rng, 128, 65536), "groups": _log(rng, 2, 128),
                "n": _width(rng, 512, 7168, 64), "k": _width(rng, 512, 7168, 64), "trans_b": rng.random() < 0.5,
                "dtype": half}
    if kind == "k_grouped":
        return {"kind": kind, "rows": _log(rng, 256, 65536), "groups": _log(rng, 2, 128),
                "m": _width(rng, 512, 4096, 64), "n": _width(rng, 512, 4096, 64), "dtype": half}
    if kind == "moe16":
        experts = rng.choice((8, 16, 32, 64, 128))
        return {"kind": kind, "tokens": _log(rng, 1, 8192), "hidden": _width(rng, 512, 4096, 64),
                "inter": _width(rng, 256, 4096, 64), "experts": experts, "top_k": rng.choice((1, 2, 4, 6, 8)),
                "dtype": half}
    experts, groups = rng.choice(((64, 8), (128, 8), (160, 8), (256, 8), (256, 16)))
    return {"kind": "route", "tokens": _log(rng, 16, 40000), "experts": experts, "groups": groups,
            "topk_group": groups // 2, "top_k": rng.choice((4, 6, 8)), "block": rng.choice((16, 32, 64, 128)),
            "dtype": rng.choice(("fp32", "bf16"))}


# ---- inputs ------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    t = torch.randn(*shape, generator=g, device=DEV, dtype=dtype)
    return t.mul_(scale) if scale != 1.0 else t


def _fp8_weights(g, experts, n, k):
    """[experts, n, k] weights ~ N(0, 0.02^2) as e4m3 with one fp32 scale per 128 x 128 block (the last block of n may
    be partial)."""
    q = torch.empty(experts, n, k, dtype=FP8, device=DEV)
    s = torch.empty(experts, (n + 127) // 128, k // 128, dtype=torch.float32, device=DEV)
    step = max(1, 2 ** 28 // (n * k))
    for e0 in range(0, experts, step):
        c = min(step, experts - e0)
        w = _randn(g, c, n, k, dtype=torch.bfloat16, scale=0.02)
        if n % 128:
            w = torch.cat([w, w.new_zeros(c, 128 - n % 128, k)], dim=1)
        blk = w.view(c, -1, 128, k // 128, 128)
        amax = blk.abs().amax(dim=(2, 4), keepdim=True).float()
        s[e0:e0 + c] = (amax / 448.0).view(c, -1, k // 128)
        q[e0:e0 + c] = (blk * (448.0 / amax).to(torch.bfloat16)).clamp_(-448.0, 448.0).view(c, -1, k)[:, :n].to(FP8)
    return q, s


def _group_sizes(g, rows, groups):
    """Ragged sizes that add up to `rows`: shares of log-normal popularity."""
    share = torch.softmax(_randn(g, groups, scale=0.7), 0).double()
    ends = (torch.cumsum(share, 0) * rows).round().long().clamp_(max=rows)
    ends[-1] = rows
    return torch.diff(ends, prepend=ends.new_zeros(1))


def prepare(case, seed):
    g = _gen(seed)
    c = dict(case)
    st = {"case": c, "kind": c["kind"]}
    kind = c["kind"]
    dt = DTYPES[c.get("dtype", "bf16")]
    if kind in ("moe", "decode"):
        st["w13"] = _fp8_weights(g, c["experts"], 2 * c["inter"], c["hidden"])
        st["w2"] = _fp8_weights(g, c["experts"], c["hidden"], c["inter"])
        st["x"] = _randn(g, c["tokens"], c["hidden"], dtype=dt)
        st["logits"] = _randn(g, c["tokens"], c["experts"])
        if kind == "decode":
            rank = torch.randperm(c["experts"], generator=g, device=DEV).float() + 1.0
            st["logits"] -= ZIPF * torch.log(rank)
            st["layer"] = FusedMoELowLatency(1, None, c["experts"], c["hidden"], 0, out_dtype=dt)
        else:
            st["bias"] = _randn(g, c["experts"], scale=0.01)
            st["layer"] = DlblasTritonFusedMoEBlockedF8Impl(top_k=c["top_k"], num_experts=c["experts"],
                                                            renormalize=c["routing"] == "softmax", out_dtype=dt)
    elif kind == "linear":
        w, s = _fp8_weights(g, 1, c["n"], c["k"])
        st["w"], st["ws"] = w[0], s[0]
        st["x"] = _randn(g, c["tokens"], c["k"], dtype=dt)
    elif kind == "gating":
        st["logits"] = _randn(g, c["tokens"], c["experts"], dtype=dt)
        if c["train"]:
            st["logits"].requires_grad_(True)
            st["grads"] = (torch.full((), 0.01, dtype=dt, device=DEV),
                           _randn(g, c["top_k"] * c["tokens"], dtype=dt))
    elif kind == "permute":
        # distinct experts per token; a share of the slots is routed to no expert here (-1)
        ids = torch.randn(c["tokens"], c["experts"], generator=g, device=DEV, dtype=torch.float32)
        ids = ids.topk(c["top_k"], dim=1).indices
        if c["dropped"]:
            gone = torch.randperm(ids.numel(), generator=g, device=DEV)[:round(c["dropped"] * ids.numel())]
            ids.view(-1)[gone] = -1
        st["ids"] = ids.to(torch.int32)
        st["x"] = _randn(g, c["tokens"], c["hidden"], dtype=dt).requires_grad_(True)
        probs = torch.softmax(_randn(g, c["tokens"], c["top_k"]), dim=1)
        st["probs"] = probs.requires_grad_(True)
        st["grad"] = _randn(g, c["tokens"], c["hidden"], dtype=dt)
    elif kind == "m_grouped":
        st["sizes"] = _group_sizes(g, c["rows"], c["groups"])
        st["a"] = _randn(g, c["rows"], c["k"], dtype=dt)
        shape = (c["n"], c["k"]) if c["trans_b"] else (c["k"], c["n"])
        st["b"] = _randn(g, c["groups"], *shape, dtype=dt, scale=0.02)
    elif kind == "k_grouped":
        st["sizes"] = _group_sizes(g, c["rows"], c["groups"])
        st["a"] = _randn(g, c["rows"], c["m"], dtype=dt)
        st["b"] = _randn(g, c["rows"], c["n"], dtype=dt, scale=0.05)
    elif kind == "moe16":
        st["w1"] = _randn(g, c["experts"], 2 * c["inter"], c["hidden"], dtype=dt, scale=0.02)
        st["w2"] = _randn(g, c["experts"], c["hidden"], c["inter"], dtype=dt, scale=0.02)
        st["x"] = _randn(g, c["tokens"], c["hidden"], dtype=dt)
        st["logits"] = _randn(g, c["tokens"], c["experts"])
    elif kind == "route":
        st["x"] = _randn(g, c["tokens"], 16, dtype=torch.bfloat16)     # only its row count is looked at
        st["logits"] = _randn(g, c["tokens"], c["experts"], dtype=dt)
        st["bias"] = _randn(g, c["experts"], scale=0.01)
    else:
        raise ValueError(kind)
    return st


# ---- one pass ----------------------------------------------------------------------------------------------------
def run(state):
    c, kind = state["case"], state["kind"]
    if kind == "moe":
        if c["routing"] == "grouped":
            w, ids = biased_grouped_topk(state["x"], state["logits"], state["bias"], c["top_k"], True, 8, 4)
        else:
            w, ids = ops.route_softmax_topk(state["logits"], c["top_k"])
        return state["layer"].forward(state["x"], w, ids, *state["w13"], *state["w2"])
    if kind == "decode":
        w, ids = ops.route_softmax_topk(state["logits"], c["top_k"], True)
        return state["layer"].forward(state["x"], w, ids, *state["w13"], *state["w2"])
    if kind == "linear":
        xq, xs = per_token_group_quant_fp8(state["x"], 128)
        return fp8_gemm(xq, state["w"], xs, state["ws"])
    if kind == "gating":
        l_aux, ec_idx, weights, select = dlblas_b200.topk_gating(state["logits"], c["top_k"], c["capacity"], 2,
                                                                 c["train"])
        out = {"l_aux": l_aux, "ec_idx": ec_idx, "weights": weights, "select": select}
        if c["train"]:
            (out["grad"],) = torch.autograd.grad((l_aux, weights), (state["logits"],), state["grads"])
        return out
    if kind == "permute":
        rows, row_map = permute(state["x"], state["ids"])
        y = unpermute(rows, row_map, state["probs"])
        gx, gp = torch.autograd.grad(y, (state["x"], state["probs"]), state["grad"])
        return {"rows": rows, "row_map": row_map, "y": y, "grad_x": gx, "grad_probs": gp}
    if kind == "m_grouped":
        return m_grouped_gemm(state["a"], state["b"], state["sizes"], trans_b=c["trans_b"])
    if kind == "k_grouped":
        return k_grouped_gemm(state["a"], state["b"], state["sizes"])
    if kind == "moe16":
        w, ids = ops.route_softmax_topk(state["logits"], c["top_k"], True)
        return fused_moe(state["x"], state["w1"], state["w2"], w, ids, out_dtype=DTYPES[c["dtype"]])
    w, ids = biased_grouped_topk(state["x"], state["logits"], state["bias"], c["top_k"], True, c["groups"],
                                 c["topk_group"])
    sorted_ids, expert_ids, padded = moe_align_block_size(ids, c["block"], c["experts"], c["experts"])
    return {"weights": w, "ids": ids, "sorted_ids": sorted_ids, "expert_ids": expert_ids, "padded": padded}


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def _hit(tokens, top_k, experts, skew=0.0):
    """Experts that get at least one row."""
    if not skew:
        return experts * (1.0 - (1.0 - top_k / experts) ** tokens)
    rng = np.random.RandomState(0)                       # one fixed sample of the skewed routing
    scores = rng.randn(tokens, experts) - skew * np.log(np.arange(1, experts + 1))
    return float(np.unique(np.argsort(-scores, axis=1)[:, :top_k]).size)


def work(case):
    c, kind = case, case["kind"]
    size = DTYPES[c.get("dtype", "bf16")].itemsize
    if kind in ("moe", "decode", "moe16"):
        t, h, i, e, k = c["tokens"], c["hidden"], c["inter"], c["experts"], c["top_k"]
        weight = 2.0 if kind == "moe16" else 1.0 + 4.0 / (128 * 128)
        return {"bytes": _hit(t, k, e, ZIPF if kind == "decode" else 0.0) * 3 * i * h * weight + 2 * t * h * size + 4 * t * e,
                "flops": 6.0 * t * k * h * i}
    if kind == "linear":
        t, n, k = c["tokens"], c["n"], c["k"]
        return {"bytes": t * k * size + n * k * (1 + 4 / (128 * 128)) + 2 * t * n, "flops": 2.0 * t * n * k}
    if kind == "gating":
        t, e, k = c["tokens"], c["experts"], c["top_k"]
        slots = max(2, math.ceil(t / e * c["capacity"] * k)) * e
        b = t * e * size + t * k * (4 + size) + 8 * slots
        if c["train"]:                                   # logits again, weight gradients in, logit gradients out
            b += 2 * t * e * size + t * k * size
        return {"bytes": b, "flops": 4.0 * t * e * (2 if c["train"] else 1)}
    if kind == "permute":
        t, h, k = c["tokens"], c["hidden"], c["top_k"]
        rows = t * k * (1.0 - c["dropped"])
        # permute t + rows, unpermute rows + t; backward: grad t, rows (for the probabilities), rows out; rows in, t out
        return {"bytes": (4 * t + 5 * rows) * h * size, "flops": 6.0 * rows * h}
    if kind == "m_grouped":
        r, n, k = c["rows"], c["n"], c["k"]
        return {"bytes": 2.0 * (r * k + r * n + min(c["groups"], r) * n * k), "flops": 2.0 * r * n * k}
    if kind == "k_grouped":
        r, m, n = c["rows"], c["m"], c["n"]
        return {"bytes": 2.0 * (r * m + r * n + c["groups"] * m * n), "flops": 2.0 * r * m * n}
    t, e, k = c["tokens"], c["experts"], c["top_k"]
    layout = t * k + e * (c["block"] - 1)
    return {"bytes": t * e * size + 8 * t * k + 4 * layout + 4 * layout / c["block"], "flops": 20.0 * t * e}


def _seconds(case):
    """Roughly what a pass takes at the rates of this card: 6.5 TB/s; 3.3 PFLOP/s in FP8, half of that in 16 bits."""
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (3.3e15 if case["kind"] in ("moe", "decode", "linear") else 1.65e15))


def tolerance(case):
    kind = case["kind"]
    if kind in ("moe", "decode", "moe16"):
        # 16-bit intermediates between two GEMMs; FP8: a sum in another order moves some of them across a rounding
        # boundary of the e4m3 re-quantisation
        return {"rel": 1e-2}
    if kind in ("linear", "m_grouped", "k_grouped"):
        return {"rel": 4e-3}                             # fp32 sums, one rounding to 16 bits
    if kind == "gating":
        return {"rel": 1e-5 if case["dtype"] == "fp32" else 1e-3}
    if kind == "permute":
        return {"rel": 1e-5 if case["dtype"] == "fp32" else 4e-3}
    return {"rel": 1e-5}                                 # routing weights; ids and layout are whole numbers
