"""The work that users of this framework have it do, as cases that can be timed.

Six paths, each over the range of sizes it is called with:

  nvfp4      NVFP4 grouped GEMM over padded per-expert batches; with "dynamic" the activations
             arrive in bf16 / fp32 and their global scale and quantisation are part of the call
  moe        the masked MoE layer (quantise, GEMM1, SiLU * up, quantise, GEMM2)
  megamoe    the routed MoE layer (top-k routing, dispatch, experts, combine)
  mxfp8      quantise activations to MXFP8, then the grouped GEMM over row-concatenated groups
  int4       bf16 activations x int4 weights, grouped
  dense      one fp16 / bf16 matrix product

A case is a dict of plain values.  Weights are quantised when the state is made, as a program
does when it loads a model; activations are new for every state.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import mosaicist_b200.torch_ops  # noqa: F401  (registers torch.ops.mosaicist_sm100a.*)
from mosaicist_b200 import ops
from mosaicist_b200.moe import MegaMoE, fold_alphas, moe_masked


# ---- the cases ---------------------------------------------------------------------------


def listed():
    return [
        # a decode step of a few sequences per expert through one projection: launch latency
        dict(name="nvfp4_decode", path="nvfp4", l=8, m=128, n=2048, k=2048, rows="few", rows_seed=1, dynamic=False, x="bf16"),
        # the headline grouped GEMM: 8 experts x 512 rows, operands already quantised
        dict(name="nvfp4_headline", path="nvfp4", l=8, m=512, n=2048, k=2048, rows="full", rows_seed=0, dynamic=False, x="bf16"),
        # a prefill projection with dynamic activation scales: ragged batches of up to 2048 rows
        dict(name="nvfp4_prefill_dynamic", path="nvfp4", l=8, m=2048, n=4096, k=7168, rows="ragged", rows_seed=2, dynamic=True, x="bf16"),
        # the masked layer in decode, as a graph of torch operators calls it
        dict(name="moe_decode", path="moe", l=8, m=128, k=2048, n=1024, rows="few", rows_seed=3, torch_op=True, folded=False),
        # the masked layer at the size of the end-to-end benchmark, scales folded at load time
        dict(name="moe_batch", path="moe", l=8, m=512, k=2048, n=1024, rows="full", rows_seed=0, torch_op=False, folded=True),
        # a decode step of 16 sequences through 256 experts: weight streaming
        dict(name="megamoe_decode", path="megamoe", tokens=16, experts=256, topk=8, hidden=7168, n=2048),
        # the routed layer's benchmark: a prefill of 8192 tokens
        dict(name="megamoe_prefill", path="megamoe", tokens=8192, experts=256, topk=8, hidden=7168, n=2048),
        # skewed expert loads (Zipf 1.2) in MXFP8, activations quantised on the way
        dict(name="mxfp8_zipf", path="mxfp8", groups=32, total=16384, zipf=1.2, n=4096, k=7168, x="bf16"),
        # weight-only int4: a batch of 64 experts, then the same weights in a decode step
        dict(name="int4_batch", path="int4", groups=64, lo=64, hi=512, rows_seed=4, n=2048, k=7168, group_size=128),
        dict(name="int4_decode", path="int4", groups=64, lo=1, hi=16, rows_seed=5, n=2048, k=7168, group_size=128),
        # dense half precision: the square benchmark, and a small product with no round size
        dict(name="dense_8192", path="dense", m=8192, n=8192, k=8192, dtype="fp16"),
        dict(name="dense_odd", path="dense", m=777, n=1048, k=3080, dtype="bf16"),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(v) // step * step))


#: the largest listed case in each resource; drawn cases stay under it
_MAX_FLOPS = 5.0e12
_MAX_BYTES = 5.0e9


def draw(rng):
    while True:
        path = rng.choice(["nvfp4", "moe", "megamoe", "mxfp8", "int4", "dense"])
        seed = rng.randrange(1 << 20)
        if path == "nvfp4":
            case = dict(path=path, l=_log(rng, 1, 32), m=_log(rng, 128, 2048, 128), n=_log(rng, 128, 8192, 128),
                        k=_log(rng, 256, 8192, 64), rows=rng.choice(["full", "ragged", "few"]), rows_seed=seed,
                        dynamic=rng.random() < 0.4, x=rng.choice(["bf16", "f32"]))
        elif path == "moe":
            # rows beyond masked_m come back undefined from moe_masked and as zeros from the operator
            rows = rng.choice(["full", "ragged", "few"])
            torch_op = rows != "full" or rng.random() < 0.3
            case = dict(path=path, l=_log(rng, 1, 32), m=_log(rng, 128, 1024, 128), k=_log(rng, 512, 7168, 128),
                        n=_log(rng, 256, 4096, 64), rows=rows, rows_seed=seed, torch_op=torch_op,
                        folded=not torch_op and rng.random() < 0.7)
        elif path == "megamoe":
            case = dict(path=path, tokens=_log(rng, 1, 8192), experts=rng.choice([32, 64, 128, 160, 256]),
                        topk=rng.choice([1, 2, 4, 6, 8]), hidden=_log(rng, 1024, 7168, 128), n=_log(rng, 256, 2048, 128))
        elif path == "mxfp8":
            groups = _log(rng, 2, 64)
            case = dict(path=path, groups=groups, total=max(groups, _log(rng, 16, 16384)), zipf=rng.choice([0.0, 0.6, 1.2]),
                        n=_log(rng, 256, 4096, 128), k=_log(rng, 512, 7168, 128), x=rng.choice(["bf16", "f32"]))
        elif path == "int4":
            hi = _log(rng, 4, 512)
            case = dict(path=path, groups=_log(rng, 2, 64), lo=max(1, hi // 8), hi=hi, rows_seed=seed,
                        n=_log(rng, 256, 4096, 256), k=_log(rng, 512, 7168, 128), group_size=rng.choice([64, 128]))
        else:
            case = dict(path=path, m=_log(rng, 1, 8192), n=_log(rng, 64, 8192, 8), k=_log(rng, 64, 8192, 8),
                        dtype=rng.choice(["fp16", "bf16"]))
        w = work(case)
        if w["flops"] <= _MAX_FLOPS and w["bytes"] <= _MAX_BYTES:
            return case


def _rows(case):
    """Rows of each group: part of the case, so that every state of it does the same work."""
    if case["path"] == "mxfp8":
        w = 1.0 / np.arange(1, case["groups"] + 1) ** case["zipf"]
        rows = np.maximum(1, np.floor(w / w.sum() * case["total"])).astype(int)
        rows[0] = max(1, rows[0] + case["total"] - rows.sum())
        return rows.tolist()
    rng = np.random.default_rng(case["rows_seed"])
    if case["path"] == "int4":
        return rng.integers(case["lo"], case["hi"] + 1, case["groups"]).tolist()
    l, m = case["l"], case["m"]
    if case["rows"] == "full":
        return [m] * l
    if case["rows"] == "few":
        return rng.integers(0, 17, l).clip(1 if l == 1 else 0).tolist()
    return rng.integers(m // 4, m + 1, l).tolist()


# ---- the work that cannot be left out ------------------------------------------------------


def _nvfp4_bytes(values):
    return values * (0.5 + 1.0 / 16)


def work(case):
    p = case["path"]
    if p == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2.0 * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}
    if p == "megamoe":
        t, e, kk, h, n = (case[x] for x in ("tokens", "experts", "topk", "hidden", "n"))
        used = e * (1.0 - (1.0 - kk / e) ** t)      # experts that get a token, on average
        return {"bytes": used * _nvfp4_bytes(3 * n * h) + t * (4 * h + 4 * e), "flops": 2.0 * t * kk * 3 * n * h}
    rows = _rows(case)
    total, used = sum(rows), sum(r > 0 for r in rows)
    if p == "nvfp4":
        n, k = case["n"], case["k"]
        # the global scale is that of the whole padded batch
        a = case["l"] * case["m"] * k * (4 if case["x"] == "f32" else 2) if case["dynamic"] else _nvfp4_bytes(total * k)
        return {"bytes": a + _nvfp4_bytes(used * n * k) + 2.0 * total * n, "flops": 2.0 * total * n * k}
    if p == "moe":
        n, k = case["n"], case["k"]
        return {"bytes": 4.0 * total * k + _nvfp4_bytes(used * 3 * n * k), "flops": 2.0 * total * 3 * n * k}
    n, k = case["n"], case["k"]
    if p == "mxfp8":
        a = total * k * (4 if case["x"] == "f32" else 2)
        return {"bytes": a + used * n * k * (1 + 1.0 / 32) + 2.0 * total * n, "flops": 2.0 * total * n * k}
    weights = used * n * k * (0.5 + 2.0 / case["group_size"])
    return {"bytes": 2.0 * total * (k + n) + weights, "flops": 2.0 * total * n * k}


def tolerance(case):
    # bf16 results: one rounding is 2^-9 relative; the layers round the intermediate to bf16 and to
    # e2m1, where another order of fp32 sums moves a value to the neighbouring step now and then
    if case["path"] == "dense" and case["dtype"] == "fp16":
        return {"rel": 2e-3}
    return {"rel": 1e-2}


# ---- inputs --------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, shape, dtype, std=1.0):
    return torch.randn(shape, device="cuda", dtype=dtype, generator=gen).mul_(std)


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _nvfp4_weights(gen, l, n, k, std=0.02):
    """(q, scales, global scale) of N(0, std) weights, a few groups at a time."""
    q = torch.empty((l, n, k // 2), dtype=torch.uint8, device="cuda")
    sf = torch.empty((l, n // 128, k // 64, 32, 16), dtype=torch.uint8, device="cuda")
    gs = torch.empty((l,), dtype=torch.float32, device="cuda")
    step = max(1, (1 << 29) // (n * k))
    for g in range(0, l, step):
        w = _randn(gen, (min(step, l - g), n, k), torch.bfloat16, std)
        s = ops.global_scale_for(w)
        q[g:g + step], sf[g:g + step] = ops.quantize_nvfp4(w, s)
        gs[g:g + step] = s
    return q, sf, gs


def _layout(rows):
    """128-aligned offsets of row-concatenated groups and the rows they take."""
    offsets, total = [], 0
    for r in rows:
        offsets.append(total)
        total += (r + 127) // 128 * 128
    return offsets, max(total, 128)


def _a2_scale(l, std):
    """Global scale of silu(gate) * up for gate and up of N(0, std)."""
    return torch.full((l,), 2688.0 / max(1.0, (4.0 * std) ** 2), device="cuda")


def prepare(case, seed):
    gen = _gen(seed)
    p = case["path"]
    f32 = dict(dtype=torch.float32, device="cuda")
    if p == "dense":
        dt = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
        std = case["k"] ** -0.5
        return dict(run=_run_dense, a=_randn(gen, (case["m"], case["k"]), dt, std),
                    b=_randn(gen, (case["k"], case["n"]), dt, std))
    if p == "megamoe":
        t, e, kk, h, n = (case[x] for x in ("tokens", "experts", "topk", "hidden", "n"))
        one = torch.ones((e,), **f32)
        w1 = _nvfp4_weights(gen, e, 2 * n, h)
        w2 = _nvfp4_weights(gen, e, h, n)
        layer = MegaMoE(*w1, one, *w2, one, torch.full((e,), 2688.0 / 5.0, **f32), _a2_scale(e, 0.02 * h ** 0.5),
                        topk=kk, max_tokens=t)
        return dict(run=_run_megamoe, layer=layer, tokens=_randn(gen, (t, h), torch.bfloat16),
                    logits=_randn(gen, (t, e), torch.float32))
    rows = _rows(case)
    if p == "nvfp4":
        l, m, n, k = (case[x] for x in ("l", "m", "n", "k"))
        w = _nvfp4_weights(gen, l, n, k)
        x = _randn(gen, (l, m, k), torch.float32 if case["x"] == "f32" else torch.bfloat16)
        state = dict(w=w, alpha=torch.rand((l,), device="cuda", generator=gen) + 0.5, masked_m=_i32(rows),
                     out=torch.zeros((l, m, n), dtype=torch.bfloat16, device="cuda"))
        if case["dynamic"]:
            return dict(state, run=_run_nvfp4_dynamic, x=x)
        gs = ops.global_scale_for(x)
        state["alpha"] = state["alpha"] / (gs * w[2])
        return dict(state, run=_run_nvfp4, a=ops.quantize_nvfp4(x, gs))
    if p == "moe":
        l, m, n, k = (case[x] for x in ("l", "m", "n", "k"))
        w1 = _nvfp4_weights(gen, l, 2 * n, k)
        w2 = _nvfp4_weights(gen, l, k, n)
        alpha = torch.rand((2, l), device="cuda", generator=gen) + 0.5
        hidden = _randn(gen, (l, m, k), torch.bfloat16)
        args = (hidden, *w1, alpha[0].contiguous(), *w2, alpha[1].contiguous(), _i32(rows),
                torch.full((l,), 2688.0 / 5.0, **f32), _a2_scale(l, 0.03 * k ** 0.5))
        if case["torch_op"]:
            return dict(run=_run_moe_op, args=args)
        folded = fold_alphas(w1[2], args[4], w2[2], args[8], args[10], args[11]) if case["folded"] else None
        return dict(run=_run_moe, args=args, folded=folded)
    n, k = case["n"], case["k"]
    offsets, total = _layout(rows)
    state = dict(offsets=_i32(offsets), rows=_i32(rows), out=torch.zeros((total, n), dtype=torch.bfloat16, device="cuda"))
    if p == "mxfp8":
        b_q = torch.empty((len(rows), n, k), dtype=torch.uint8, device="cuda")
        b_sf = torch.empty((len(rows), n // 128, k // 128, 32, 16), dtype=torch.uint8, device="cuda")
        for g in range(len(rows)):
            b_q[g], b_sf[g] = ops.quantize_mxfp8(_randn(gen, (n, k), torch.bfloat16, 0.02))
        dt = torch.float32 if case["x"] == "f32" else torch.bfloat16
        return dict(state, run=_run_mxfp8, x=_randn(gen, (total, k), dt), b_q=b_q, b_sf=b_sf)
    gsz = case["group_size"]
    return dict(state, run=_run_int4, a=_randn(gen, (total, k), torch.bfloat16),
                b_q=torch.randint(0, 256, (len(rows), n, k // 2), dtype=torch.uint8, device="cuda", generator=gen),
                scales=_randn(gen, (len(rows), n, k // gsz), torch.bfloat16, 0.02).abs_(), group_size=gsz)


# ---- one pass ------------------------------------------------------------------------------


def _run_dense(s):
    return ops.gemm_f16(s["a"], s["b"])


def _run_megamoe(s):
    return s["layer"].forward(s["tokens"], s["logits"])


def _run_nvfp4(s):
    a_q, a_sf = s["a"]
    b_q, b_sf, _ = s["w"]
    return ops.masked_grouped_gemm(a_q, a_sf, b_q, b_sf, s["alpha"], s["masked_m"], out=s["out"])


def _run_nvfp4_dynamic(s):
    b_q, b_sf, b_gs = s["w"]
    gs = ops.global_scale_for(s["x"])
    a_q, a_sf = ops.quantize_nvfp4(s["x"], gs, s["masked_m"])
    return ops.masked_grouped_gemm(a_q, a_sf, b_q, b_sf, s["alpha"] / (gs * b_gs), s["masked_m"], out=s["out"])


def _run_moe(s):
    return moe_masked(*s["args"], folded_alphas=s["folded"])


def _run_moe_op(s):
    return torch.ops.mosaicist_sm100a.moe_masked(*s["args"])


def _run_mxfp8(s):
    a_q, a_sf = ops.quantize_mxfp8(s["x"], group_offsets=s["offsets"], group_rows=s["rows"])
    return ops.ragged_grouped_gemm_mxfp8(a_q, a_sf, s["b_q"], s["b_sf"], s["offsets"], s["rows"], out=s["out"])


def _run_int4(s):
    return ops.mixed_grouped_gemm_int4(s["a"], s["b_q"], s["scales"], s["offsets"], s["rows"],
                                       group_size=s["group_size"], out=s["out"])


def run(state):
    return state["run"](state)
