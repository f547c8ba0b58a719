// Device helpers of the NVFP4 quantiser shared by the stand-alone quantise kernels and the
// MoE dispatch kernel: the arithmetic of quantize_nvfp4
// (experiments/flashinfer-megamoe-sm100a/nvfp4.py:39-57) on 64 values at a time, and the
// address of a scale word in the 128-row MMA tiling (nvfp4.py:121-131).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "ptx.cuh"

namespace msc {

__device__ __forceinline__ float e4m3_to_float(uint8_t b) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(b, __NV_E4M3);
  return __half2float(__half(h));
}

// Offset of scale (row, kblock/4 word) in the tiled layout (row_tiles, kwords, 32, 16):
// row = 128 t + 32 a + b  ->  [t, c, b, 4 a + d], d = kblock % 4.
__device__ __forceinline__ size_t tiled_sf_word(int row, int kword, int kwords) {
  const int t = row >> 7, a = (row >> 5) & 3, b = row & 31;
  return (((size_t)t * kwords + kword) * 32 + b) * 16 + 4 * a;
}

// silu(gate) * up = gate / (1 + 2^(-gate log2 e)) * up in fp32 (nvfp4.py:81-88), with the
// approximate exponential and reciprocal the reference's own kernel uses
// (quantize_kernels.py:50-69): the result only feeds the e2m1 / e4m3 quantiser, a few ulp are
// far below its steps, and the accurate expf + IEEE reciprocal cost five times the
// instructions.  Every kernel that activates goes through this one function, so the fused and
// the stand-alone paths keep producing the same bytes.
__device__ __forceinline__ float silu_mul(float gate, float up) {
  float e, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(__fmul_rn(gate, -1.4426950408889634f)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(__fadd_rn(1.0f, e)));
  return __fmul_rn(__fmul_rn(s, gate), up);
}

// a / b by one correction step: q = RN(a rb), r = RN(a - q b), q' = RN(q + r rb).  The method is
// Markstein's (P. W. Markstein, Computation of elementary functions on the IBM RISC System/6000
// processor, IBM J. Res. Dev. 34(1), 1990): with rb = RN(1 / b), q within one ulp of a / b, and r exact,
// q' is a / b correctly rounded.  r is exact while nothing over- or underflows (q finite, q * b and r
// within fp32's exponents).  q may miss by more than one ulp where a's significand is the smaller one,
// so what this file relies on is tested on the device over all significands against __fdiv_rn
// (tests/test_division_gpu.py): the quotients that become scales, bit for bit, and the e2m1 values of
// quotients around every rounding boundary.  The block quantiser divides 16 values by the same step,
// so the reciprocal is shared.
template <bool GUARD = true>
__device__ __forceinline__ float div_rn_shared_rcp(float a, float b, float rb) {
  const float q = __fmul_rn(a, rb);
  const float r = __fmaf_rn(-q, b, a);
  const float qc = __fmaf_rn(r, rb, q);
  // keep +-inf instead of inf - inf; a block whose largest quotient is finite needs no guard
  // (a NaN element comes out NaN either way)
  return (!GUARD || fabsf(q) <= 3.0e38f) ? qc : q;
}

// Two fp32 values in one 64-bit register pair: Blackwell's packed fp32 instructions round each
// half exactly as the scalar ones do, at half the issue slots.
__device__ __forceinline__ uint64_t pair_f32(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpair_f32(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// 16 values / step -> 8 bytes of e2m1.  The reference's clip to [-6, 6] is what the saturating
// conversion does to finite and infinite values alike, so it is not repeated here.
template <bool GUARD>
__device__ __forceinline__ void pack_block(const float* v, float safe, float rsafe, uint32_t* w) {
  const uint64_t r2 = pair_f32(rsafe, rsafe), n2 = pair_f32(-safe, -safe);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t word = 0;
#pragma unroll
    for (int pr = 0; pr < 4; ++pr) {
      const int i = h * 8 + pr * 2;
      float2 x;
      if (GUARD) {
        x.x = div_rn_shared_rcp<true>(v[i], safe, rsafe);
        x.y = div_rn_shared_rcp<true>(v[i + 1], safe, rsafe);
      } else {   // the same three operations on two values at a time: q(-b) is -(qb) exactly
        const uint64_t a2 = pair_f32(v[i], v[i + 1]);
        const uint64_t q2 = mul_f32x2(a2, r2);
        x = unpair_f32(fma_f32x2(fma_f32x2(q2, n2, a2), r2, q2));
      }
      const __nv_fp4x2_storage_t b2 = __nv_cvt_float2_to_fp4x2(x, __NV_E2M1, cudaRoundNearest);
      word |= (uint32_t)b2 << (8 * pr);
    }
    w[h] = word;
  }
}

// a / b rounded to nearest, through rb = RN(1 / b) where every intermediate is in range for b = 6 (a
// zero or between 1e-30 and 1e30: the remainder of 1e-30 is a multiple of 2^-147), else by division.
__device__ __forceinline__ float div_rn_mid(float a, float b, float rb) {
  if (a == 0.0f || (a >= 1e-30f && a <= 1e30f)) return div_rn_shared_rcp<false>(a, b, rb);
  return __fdiv_rn(a, b);
}
// The block maximum's share of a scale, amax / 6, and the step that a scale stands for, sf / gs with sf
// an e4m3 value (0 or 2^-9 .. 448): both as __fdiv_rn gives them.
__device__ __forceinline__ float amax_over_6(float amax) {
  return div_rn_mid(amax, 6.0f, 0.16666667163372039794921875f);   // RN(1/6)
}
__device__ __forceinline__ float scale_step(float sf, float gs) {
  return (gs >= 1e-25f && gs <= 1e25f) ? div_rn_shared_rcp<false>(sf, gs, __frcp_rn(gs)) : __fdiv_rn(sf, gs);
}

// Quantises one block of 16 fp32 values, whose largest magnitude is `amax`, into 8 bytes of
// e2m1 and its e4m3 scale byte.
__device__ __forceinline__ void quantize_16_amax(const float* v, float amax, float gs, uint2& q8, uint32_t& sfb) {
  // divisions by 6 and by the group's gs: their reciprocals are constant or shared by the
  // thread's blocks, so the correctly rounded quotient takes three instructions
  float s = __fmul_rn(amax_over_6(amax), gs);
  s = fminf(fmaxf(s, 0.0f), 448.0f);
  sfb = (uint32_t)(uint8_t)__nv_cvt_float_to_fp8(s, __NV_SATFINITE, __NV_E4M3);
  const float sf = e4m3_to_float((uint8_t)sfb);
  const float step = scale_step(sf, gs);
  // A dead block (step == 0) must yield x / 1 * 0 = +-0 with the sign of x, as the reference
  // computes: with divisor 1 and "reciprocal" 0 the shared-reciprocal division returns exactly
  // that (q = x * 0, remainder x, correction x * 0 + q), so no separate multiply is needed.
  const bool dead = step == 0.0f;
  const float safe = dead ? 1.0f : step;
  const float rsafe = dead ? 0.0f : __frcp_rn(step);
  // the largest quotient of the block bounds all of them: only a block where it overflows (an
  // infinite element, a step that underflowed) takes the per-element overflow guard
  uint32_t w[2];
  if (__fmul_rn(amax, rsafe) <= 3.0e38f) pack_block<false>(v, safe, rsafe, w);
  else pack_block<true>(v, safe, rsafe, w);
  q8 = make_uint2(w[0], w[1]);
}

// Largest magnitude of 16 values, NaNs left out (a block of NaNs counts as 0).
__device__ __forceinline__ float amax_f32x16(const float* v) {
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  return amax;
}
// The same of 16 bf16 values in eight words, two at a time.
__device__ __forceinline__ float amax_bf16x16(const uint32_t* w) {
  __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
  for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
  const float2 f = __bfloat1622float2(m);
  return fmaxf(fmaxf(0.0f, f.x), f.y);
}
__device__ __forceinline__ void unpack_bf16x16(const uint32_t* w, float* v) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ void quantize_16(const float* v, float gs, uint2& q8, uint32_t& sfb) {
  quantize_16_amax(v, amax_f32x16(v), gs, q8, sfb);
}

// MXFP8: biased exponent byte of the block scale for a block maximum `amax` >= 0, the smallest
// power of two with amax / scale <= 448 = 1.75 * 2^8, from the bits of amax.
__device__ __forceinline__ uint32_t mx_scale_byte(float amax) {
  const uint32_t bits = __float_as_uint(amax);
  const int E = (int)(bits >> 23) - 127;                       // -127 for zero and subnormals
  int e = E - 8 + ((bits & 0x7fffffu) > 0x600000u ? 1 : 0);     // mantissa above 1.75
  e = max(-127, min(127, e));
  return (uint32_t)(e + 127);
}
// 16 values / scale -> 16 bytes of e4m3.  1 / scale = 2^(127 - byte) is a normal fp32 number for
// every byte the rule can produce (byte <= 247), so x / scale is one exact multiplication (or one
// rounding into the fp32 subnormals, far below e4m3's reach); the saturating conversion is the
// clip to +-448 followed by round-to-nearest-even, two values per instruction.
__device__ __forceinline__ uint4 mx_pack_16(const float* v, uint32_t sfb) {
  const float inv = __uint_as_float((254u - sfb) << 23);
  const uint64_t i2 = pair_f32(inv, inv);
  uint32_t w[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const float2 a = unpair_f32(mul_f32x2(pair_f32(v[4 * h], v[4 * h + 1]), i2));
    const float2 b = unpair_f32(mul_f32x2(pair_f32(v[4 * h + 2], v[4 * h + 3]), i2));
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(a, __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(b, __NV_SATFINITE, __NV_E4M3);
    w[h] = lo | (hi << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// The four lanes that own the four blocks of one 64-element unit (lane & 3 = block index)
// assemble their scale bytes into one 32-bit word, valid in the lane with (lane & 3) == 0.
__device__ __forceinline__ uint32_t gather_scale_word(uint32_t sfb) {
  uint32_t w = sfb;
  w |= __shfl_down_sync(0xffffffffu, sfb, 1) << 8;
  w |= __shfl_down_sync(0xffffffffu, sfb, 2) << 16;
  w |= __shfl_down_sync(0xffffffffu, sfb, 3) << 24;
  return w;
}

// Loads 16 consecutive bf16 values (32 bytes, 16-byte aligned) as fp32.
__device__ __forceinline__ void load16_bf16(const __nv_bfloat16* src, float* v) {
  const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint4 raw = ld_ordered(s4 + i);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      v[i * 8 + j * 2] = f.x;
      v[i * 8 + j * 2 + 1] = f.y;
    }
  }
}

}  // namespace msc
