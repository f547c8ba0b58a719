"""Host-side operators over torch CUDA tensors, named after the reference functions they
replace (experiments/flashinfer-megamoe-sm100a/*.py).  torch supplies device memory and
the stream; all arithmetic happens in libmosaicist_sm100a.so.  The functions here are the
documented signatures; argument checks, allocation and the launch are native
(host_ops/host_ops.cpp).
"""

from __future__ import annotations

from dataclasses import dataclass

import torch

from . import _lib

_host_ops = _lib.native


@dataclass(frozen=True)
class GemmConfig:
    """Knobs of the persistent block-scaled GEMM.  The reference's GemmConfig
    (masked_gemm.py:52-76) tunes block_k / stages of a one-tile-per-CTA kernel; here K
    staging is fixed at 128 bytes per row and the knobs are the tile width, the ring
    depth, the tile order and the persistent grid size.  Zero means library default."""
    tile_n: int = 0
    stages: int = 0
    raster: int = 0
    max_ctas: int = 0
    cta_pair: int = 0
    sf_warps: int = 0

    def c(self, epilogue: int = _lib.EPI_PLAIN) -> _lib.GemmCfg:
        return _lib.GemmCfg(self.tile_n, self.stages, self.raster, self.max_ctas, epilogue,
                            self.cta_pair, self.sf_warps)


def _ptr(t):
    return None if t is None else t.data_ptr()


def _need(t: torch.Tensor, name: str, dtypes, shape=None):
    if not t.is_cuda:
        raise ValueError(f"{name} must be a CUDA tensor")
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous")
    if t.dtype not in dtypes:
        raise ValueError(f"{name} has dtype {t.dtype}, expected one of {dtypes}")
    if shape is not None and tuple(t.shape) != tuple(shape):
        raise ValueError(f"{name} has shape {tuple(t.shape)}, expected {tuple(shape)}")


_BYTES = (torch.uint8, torch.int8, torch.float8_e4m3fn, torch.float8_e8m0fnu)
if hasattr(torch, "float4_e2m1fn_x2"):
    _BYTES = _BYTES + (torch.float4_e2m1fn_x2,)


def _stream():
    return torch.cuda.current_stream().cuda_stream


class Plan:
    """A validated call with its foreign-function arguments already built: running it costs
    one ctypes call on the current stream.  Holds references to the tensors involved."""

    def __init__(self, fn, args, out, keep):
        self._fn, self._args, self.out, self._keep = fn, args, out, keep

    def __call__(self):
        code = self._fn(*self._args, torch.cuda.current_stream().cuda_stream)
        if code:
            _lib.check(code)
        return self.out


def masked_grouped_gemm(a_q, a_sf, b_q, b_sf, alpha=None, masked_m=None,
                        config: GemmConfig = GemmConfig(), out=None) -> torch.Tensor:
    """See masked_grouped_gemm_plan; validates, launches once and returns `out`."""
    return _host_ops.masked_grouped_gemm(a_q, a_sf, b_q, b_sf, alpha, masked_m, config, out)


def masked_grouped_gemm_plan(a_q, a_sf, b_q, b_sf, alpha=None, masked_m=None,
                             config: GemmConfig = GemmConfig(), out=None) -> Plan:
    """out[l, m, n] = bf16(alpha[l] * dequant(A)[l] @ dequant(B)[l].T), rows >= masked_m[l]
    left untouched.  Same operands as masked_grouped_gemm (masked_gemm.py:104-123):
    a_q (l, m, k/2) packed e2m1, a_sf (l, m/128, k/64, 32, 16) e4m3 in the MMA tiling,
    b_q (l, n, k/2), b_sf (l, n/128, k/64, 32, 16), alpha (l,) f32, masked_m (l,) i32."""
    _need(a_q, "a_q", _BYTES)
    _need(b_q, "b_q", _BYTES)
    l, m, kh = a_q.shape
    n = b_q.shape[1]
    k = kh * 2
    _need(b_q, "b_q", _BYTES, (l, n, kh))
    _need(a_sf, "a_sf", _BYTES, (l, m // 128, k // 64, 32, 16))
    _need(b_sf, "b_sf", _BYTES, (l, n // 128, k // 64, 32, 16))
    if alpha is not None:
        _need(alpha, "alpha", (torch.float32,), (l,))
    if masked_m is not None:
        _need(masked_m, "masked_m", (torch.int32,), (l,))
    if out is None:
        out = torch.empty((l, m, n), dtype=torch.bfloat16, device=a_q.device)
    else:
        _need(out, "out", (torch.bfloat16,), (l, m, n))
    cfg = config.c()
    args = (_ptr(a_q), _ptr(a_sf), _ptr(b_q), _ptr(b_sf), _ptr(alpha), _ptr(masked_m), _ptr(out),
            l, m, n, k, cfg)
    return Plan(_lib.load().msc_grouped_gemm_nvfp4, args, out,
                (a_q, a_sf, b_q, b_sf, alpha, masked_m, cfg))


def ragged_grouped_gemm_nvfp4(a_q, a_sf, b_q, b_sf, group_offsets, group_rows, alpha=None,
                              row_scale=None, config: GemmConfig = GemmConfig(), out=None):
    """NVFP4 grouped GEMM over row-concatenated groups: group g owns rows
    [group_offsets[g], +group_rows[g]) of a_q (rows_total, k/2) and out (rows_total, n);
    offsets are multiples of 128.  Per-group arithmetic as masked_grouped_gemm."""
    return _host_ops.ragged_grouped_gemm(False, a_q, a_sf, b_q, b_sf, group_offsets, group_rows, alpha, row_scale,
                                         config, out)


def ragged_grouped_gemm_mxfp8(a_q, a_sf, b_q, b_sf, group_offsets, group_rows, alpha=None,
                              row_scale=None, config: GemmConfig = GemmConfig(), out=None):
    """MXFP8 grouped GEMM (e4m3 values, ue8m0 scale per 32) over row-concatenated groups.
    a_q (rows_total, k) e4m3, a_sf (ceil(rows_total/128), k/128, 32, 16) ue8m0, b_q (l, n, k),
    b_sf (l, n/128, k/128, 32, 16)."""
    return _host_ops.ragged_grouped_gemm(True, a_q, a_sf, b_q, b_sf, group_offsets, group_rows, alpha, row_scale,
                                         config, out)


def quantize_nvfp4(x, global_scale, masked_m=None, tiled_scales: bool = True):
    """(l, m, k) bf16/f32 -> (q (l, m, k/2) packed e2m1, sf e4m3).  Arithmetic of
    quantize_nvfp4 (nvfp4.py:39-57) / quantize_nvfp4_pallas (quantize_kernels.py:119).
    With tiled_scales the scales come out in the MMA tiling (l, m/128, k/64, 32, 16),
    otherwise row-major (l, m, k/16) as the reference kernel writes them.  Rows at or
    beyond masked_m[l] are left untouched."""
    return _host_ops.quantize_nvfp4(x, global_scale, masked_m, tiled_scales, False)


def silu_mul_quantize_nvfp4(gateup, global_scale, masked_m=None, tiled_scales: bool = True):
    """(l, m, 2n) bf16 -> NVFP4 of silu(gate) * up, gate = first n columns, activation kept in
    fp32 up to the quantiser (nvfp4.py:81-88; silu_mul_quantize_nvfp4_pallas,
    quantize_kernels.py:162)."""
    return _host_ops.quantize_nvfp4(gateup, global_scale, masked_m, tiled_scales, True)


def quantize_nvfp4_ragged(x, global_scale, group_offsets, group_rows, silu: bool = False,
                          out=None):
    """Ragged-layout quantiser: x (rows_total, k) -> q (rows_total, k/2) and tiled scales
    (ceil(rows_total/128), k/64, 32, 16); with silu, x is (rows_total, 2k) gate|up.  `out`
    may carry preallocated (q, sf)."""
    return _host_ops.quantize_nvfp4_ragged(x, global_scale, group_offsets, group_rows, silu, out)


def global_scale_for(x, numerator: float = 2688.0, out=None):
    """(l, ...) bf16/f32 -> (l,) f32: numerator / max|x[l]|, a maximum of 0 counted as 1 -
    global_scale_for (nvfp4.py:29-36; 2688 = 6 * 448)."""
    return _host_ops.global_scale_for(x, numerator, out)


def quantize_mxfp8(x, tiled_scales: bool = True, group_offsets=None, group_rows=None, out=None):
    """(rows, k) bf16/f32 -> (q (rows, k) e4m3 bytes, sf ue8m0 bytes): one power-of-two scale per
    32 K-elements, the smallest with blockmax / scale <= 448 (structure of the reference's
    block-scaled FP8 quantiser, flashinfer-megamoe-sm90a/quant.py:47-75, with the MX scale rule).
    Scales come out in the MMA tiling (ceil(rows/128), k/128, 32, 16) or row-major (rows, k/32).
    With group_offsets / group_rows only rows inside a group are written (tiled scales)."""
    return _host_ops.quantize_mxfp8(x, tiled_scales, group_offsets, group_rows, out)


def to_mma_scale_layout(sf):
    """(groups, mn, k_scales) row-major scale bytes -> (groups, ceil(mn/128), k_scales/4, 32, 16)
    (a 2-D input is treated as one group and returns 4-D), as to_mma_scale_layout
    (nvfp4.py:121-131)."""
    _need(sf, "sf", _BYTES)
    squeeze = sf.dim() == 2
    if squeeze:
        sf = sf.unsqueeze(0)
    g, mn, ks = sf.shape
    out = torch.empty((g, (mn + 127) // 128, ks // 4, 32, 16), dtype=sf.dtype, device=sf.device)
    _lib.check(_lib.load().msc_sf_swizzle(_ptr(sf), _ptr(out), g, mn, ks, _stream()))
    return out[0] if squeeze else out


def gemm_f16(a, b, out=None, max_ctas: int = 0):
    """C = A @ B for 2-D fp16 or bf16 CUDA tensors, A (m, k) and B (k, n) row-major (rows may be
    strided: a column slice of a wider matrix works as is), fp32 accumulation, output in the
    input dtype.  The reference's dense problem (experiments/hopper_gemm/ref_cutedsl.py:50-74).

    The order of a row's sums depends on k and on whether there are more than 128 rows, and on nothing
    else: with m <= 128 and k >= 4096 the contraction is summed as two halves, otherwise in one run.  So
    a column shard has the bits of the whole product, and so have row blocks on one side of 128 rows; a
    row computed in a batch of up to 128 and again in a larger one may differ in its last bit from
    k = 4096 on."""
    return _host_ops.gemm_f16(a, b, out, max_ctas)


def dequant_int4(b_q, scales, group_size: int = 128, out=None):
    """(l, n, k/2) packed int4 + (l, n, k/group_size) bf16 scales -> (l, n, k) bf16, the multiply
    done in bf16 (ports/hopper_mixed_dtype_grouped_gemm/problems.py:75-81)."""
    return _host_ops.dequant_int4(b_q, scales, group_size, out)


def ragged_grouped_gemm_bf16(a, b, group_offsets, group_rows, alpha=None, out=None, max_ctas: int = 0):
    """out[off_g + r] = bf16(alpha_g * a[off_g + r] @ b[g].T), r < group_rows[g]; a (rows_total, k)
    bf16, b (l, n, k) bf16, fp32 accumulation."""
    return _host_ops.ragged_grouped_gemm_bf16(a, b, group_offsets, group_rows, alpha, out, max_ctas)


def mixed_grouped_gemm_int4(a, b_q, scales, group_offsets, group_rows, alpha=None, group_size: int = 128,
                            workspace=None, out=None, fused: bool | None = None, max_ctas: int = 0):
    """bf16 activations x int4 weights (ports/hopper_mixed_dtype_grouped_gemm/problems.py:75-87).

    fused (default whenever k and group_size are multiples of 64): one kernel, converter warps
    expand each stage of packed weights to bf16 in registers and put them into tensor memory as
    the MMA's A operand; the weights cross HBM once, as int4.  Otherwise two launches: expand the weights to
    bf16 (`workspace`, (l, n, k) bf16, reusable while the weights do not change) and run the
    grouped bf16 GEMM.  Both produce the same bits."""
    return _host_ops.mixed_grouped_gemm_int4(a, b_q, scales, group_offsets, group_rows, alpha, group_size, workspace,
                                             out, fused, max_ctas)


def swiglu_interleave_w1(w1_q, w1_sf):
    """w1 (l, 2n, k/2) + tiled scales -> the copy the tokens-on-N fused GEMM1 reads
    (GemmConfig(cta_pair=3)): gate and up rows interleaved in blocks of 64."""
    _need(w1_q, "w1_q", _BYTES)
    l, n2, kh = w1_q.shape
    _need(w1_sf, "w1_sf", _BYTES, (l, n2 // 128, kh // 32, 32, 16))
    out_q, out_sf = torch.empty_like(w1_q), torch.empty_like(w1_sf)
    _lib.check(_lib.load().msc_swiglu_interleave_w1(_ptr(w1_q), _ptr(w1_sf), _ptr(out_q), _ptr(out_sf), l, n2,
                                                    kh * 2, _stream()))
    return out_q, out_sf


def ragged_gemm1_swiglu_quantize(a_q, a_sf, w1_q, w1_sf, group_offsets, group_rows, alpha, out_global_scale,
                                 config: GemmConfig = GemmConfig(), out=None):
    """GEMM1 + SiLU(gate) * up + NVFP4 requantisation in one kernel (the reference's
    gemm1_silu_quantize, gemm1_silu_quantize.py:94): returns (d_q (rows_total, n/2),
    d_sf tiled (rows_total/128, n/64, 32, 16)) with n = w1 rows / 2, bit-identical to the GEMM
    followed by the stand-alone SiLU quantiser."""
    return _host_ops.ragged_gemm1_swiglu_quantize(a_q, a_sf, w1_q, w1_sf, group_offsets, group_rows, alpha,
                                                  out_global_scale, config, out)
