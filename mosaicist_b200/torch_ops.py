"""The hot-path operators as torch custom operators (`torch.ops.mosaicist_sm100a.*`), for callers
that build graphs of torch operators (tracing, FakeTensor shape propagation) instead of calling
`mosaicist_b200.ops` directly:

    grouped_gemm_nvfp4         masked grouped GEMM, the operands of the reference's
                               masked_grouped_gemm (masked_gemm.py:104-123) and of FlashInfer's
                               grouped_gemm_nt_masked call site (ref_flashinfer_gemm.py:25-31)
    grouped_gemm_nvfp4_ragged  the same arithmetic over row-concatenated groups
    quantize_nvfp4             quantize_nvfp4 (nvfp4.py:39-57) with scales in the MMA tiling
    silu_mul_quantize_nvfp4    silu_mul (nvfp4.py:81-88) + quantize_nvfp4
    global_scale_for           global_scale_for (nvfp4.py:29-36)
    quantize_mxfp8             e4m3 values + one ue8m0 scale per 32, scales in the MMA tiling
    grouped_gemm_mxfp8_ragged  the MXFP8 grouped GEMM over row-concatenated groups
    gemm_f16                   the dense fp16 / bf16 problem (hopper_gemm/ref_cutedsl.py:50-74)
    grouped_gemm_bf16_int4_ragged   bf16 x int4 grouped GEMM (problems.py:75-87)
    moe_masked                 the masked MoE layer, arguments of the reference's moe_masked
                               (experiments/flashinfer-megamoe-sm100a/moe.py:47-79)

Each is the corresponding C-ABI entry point; their kernels are native (host_ops/host_ops.cpp), so that
a call costs the dispatcher and the launch.  Here are their schemas and shape functions: operators
can be traced without a GPU, and without the native module where that cannot be built.  Operators
return fresh tensors, so rows a masked call leaves untouched come back as zeros.  None has a derivative.
"""

from __future__ import annotations

import warnings

import torch

from . import _lib

if "_LIBRARY" in globals():     # the module is being reloaded
    _LIBRARY._destroy()
_LIBRARY = torch.library.Library("mosaicist_sm100a", "DEF")
for _schema in (
        "grouped_gemm_nvfp4(Tensor a_q, Tensor a_sf, Tensor b_q, Tensor b_sf, Tensor? alpha, Tensor? masked_m) -> Tensor",
        "grouped_gemm_nvfp4_ragged(Tensor a_q, Tensor a_sf, Tensor b_q, Tensor b_sf, Tensor group_offsets, "
        "Tensor group_rows, Tensor? alpha, Tensor? row_scale) -> Tensor",
        "quantize_nvfp4(Tensor x, Tensor global_scale, Tensor? masked_m) -> (Tensor, Tensor)",
        "silu_mul_quantize_nvfp4(Tensor gateup, Tensor global_scale, Tensor? masked_m) -> (Tensor, Tensor)",
        "global_scale_for(Tensor x) -> Tensor",
        "quantize_mxfp8(Tensor x) -> (Tensor, Tensor)",
        "grouped_gemm_mxfp8_ragged(Tensor a_q, Tensor a_sf, Tensor b_q, Tensor b_sf, Tensor group_offsets, "
        "Tensor group_rows, Tensor? alpha, Tensor? row_scale) -> Tensor",
        "gemm_f16(Tensor a, Tensor b) -> Tensor",
        "grouped_gemm_bf16_int4_ragged(Tensor a, Tensor b_q, Tensor scales, Tensor group_offsets, Tensor group_rows, "
        "Tensor? alpha, int group_size) -> Tensor",
        "moe_masked(Tensor hidden, Tensor w1_q, Tensor w1_sf, Tensor w1_gs, Tensor w1_alpha, Tensor w2_q, Tensor w2_sf, "
        "Tensor w2_gs, Tensor w2_alpha, Tensor masked_m, Tensor input_global_scale, Tensor a2_global_scale) -> Tensor"):
    _LIBRARY.define(_schema, tags=(torch.Tag.pt2_compliant_tag,))

try:
    _lib.host_ops()     # registers the kernels
except (ImportError, OSError, RuntimeError) as _why:
    warnings.warn(f"the operators mosaicist_sm100a::* can be traced but not run: {_why}")
_OPS = torch.ops.mosaicist_sm100a
grouped_gemm_nvfp4 = _OPS.grouped_gemm_nvfp4
grouped_gemm_nvfp4_ragged = _OPS.grouped_gemm_nvfp4_ragged
quantize_nvfp4 = _OPS.quantize_nvfp4
silu_mul_quantize_nvfp4 = _OPS.silu_mul_quantize_nvfp4
global_scale_for = _OPS.global_scale_for
quantize_mxfp8 = _OPS.quantize_mxfp8
grouped_gemm_mxfp8_ragged = _OPS.grouped_gemm_mxfp8_ragged
gemm_f16 = _OPS.gemm_f16
grouped_gemm_bf16_int4_ragged = _OPS.grouped_gemm_bf16_int4_ragged
moe_masked = _OPS.moe_masked


def _fake(name):
    return torch.library.register_fake(f"mosaicist_sm100a::{name}", lib=_LIBRARY)


@_fake("grouped_gemm_nvfp4")
def _(a_q, a_sf, b_q, b_sf, alpha, masked_m):
    return a_q.new_empty((a_q.shape[0], a_q.shape[1], b_q.shape[1]), dtype=torch.bfloat16)


@_fake("grouped_gemm_nvfp4_ragged")
def _(a_q, a_sf, b_q, b_sf, group_offsets, group_rows, alpha, row_scale):
    return a_q.new_empty((a_q.shape[0], b_q.shape[1]), dtype=torch.bfloat16)


def _quantized_shapes(l, m, k):
    return (l, m, k // 2), (l, m // 128, k // 64, 32, 16)


@_fake("quantize_nvfp4")
def _(x, global_scale, masked_m):
    qs, ss = _quantized_shapes(*x.shape)
    return x.new_empty(qs, dtype=torch.uint8), x.new_empty(ss, dtype=torch.uint8)


@_fake("silu_mul_quantize_nvfp4")
def _(gateup, global_scale, masked_m):
    l, m, n2 = gateup.shape
    qs, ss = _quantized_shapes(l, m, n2 // 2)
    return gateup.new_empty(qs, dtype=torch.uint8), gateup.new_empty(ss, dtype=torch.uint8)


@_fake("global_scale_for")
def _(x):
    return x.new_empty((x.shape[0],), dtype=torch.float32)


@_fake("quantize_mxfp8")
def _(x):
    rows, k = x.shape
    return x.new_empty((rows, k), dtype=torch.uint8), x.new_empty(((rows + 127) // 128, k // 128, 32, 16), dtype=torch.uint8)


@_fake("grouped_gemm_mxfp8_ragged")
def _(a_q, a_sf, b_q, b_sf, group_offsets, group_rows, alpha, row_scale):
    return a_q.new_empty((a_q.shape[0], b_q.shape[1]), dtype=torch.bfloat16)


@_fake("gemm_f16")
def _(a, b):
    return a.new_empty((a.shape[0], b.shape[1]))


@_fake("grouped_gemm_bf16_int4_ragged")
def _(a, b_q, scales, group_offsets, group_rows, alpha, group_size):
    return a.new_empty((a.shape[0], b_q.shape[1]), dtype=torch.bfloat16)


@_fake("moe_masked")
def _(hidden, w1_q, w1_sf, w1_gs, w1_alpha, w2_q, w2_sf, w2_gs, w2_alpha, masked_m, input_global_scale,
      a2_global_scale):
    return hidden.new_empty(hidden.shape, dtype=torch.bfloat16)
