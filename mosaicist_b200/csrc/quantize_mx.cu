// MXFP8 quantisation and the per-group global scale of NVFP4 (both HBM-bound).
//
// MXFP8 (OCP Microscaling): e4m3 values with one power-of-two scale (ue8m0: a biased exponent
// byte, 2^(b - 127)) per 32 K-elements.  Structure of the reference's block-scaled FP8
// quantiser (experiments/flashinfer-megamoe-sm90a/quant.py:47-75: scale from the block
// maximum, q = x / scale clipped to the e4m3 range) with the MX scale rule:
//   scale = 2^e,  e = the smallest integer with blockmax <= 448 * 2^e, clamped to [-127, 127]
//   q     = e4m3_rne( clip(x / scale, -448, 448) )
// e is found from the bits of blockmax (blockmax = m 2^E, 1 <= m < 2, 448 = 1.75 * 2^8:
// e = E - 8 + (m > 1.75)), so no logarithm or division can round it the wrong way; x / 2^e is
// exact.  A block of zeros (or of values below 2^-126) gets the smallest scale, byte 0.
//
// The kernel is quantize_rows_kernel (quantize_rows.cuh).
//
// Global scale (experiments/flashinfer-megamoe-sm100a/nvfp4.py:29-36): gs[g] = numerator /
// max|x| over group g, a maximum of 0 counted as 1.  |x| as fp32 bit patterns orders like
// unsigned integers, so the groups' maxima are reduced with atomicMax into the output array
// itself and a second, one-block kernel turns them into the quotient in place.
#include "quantize_rows.cuh"

namespace msc {

// max |x| per group into out[g] (as fp32 bit patterns, which order like unsigned integers).
__global__ void __launch_bounds__(256)
amax_groups_kernel(const void* __restrict__ x, int f32_in, long long per_group, unsigned int* __restrict__ out) {
  const int g = blockIdx.y;
  const long long vecs = per_group >> 3;                        // 8 elements per step
  float m = 0.0f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < vecs; i += (long long)gridDim.x * blockDim.x) {
    if (f32_in) {
      const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(x) + g * per_group) + 2 * i;
      const float4 a = __ldg(src), b = __ldg(src + 1);
      m = fmaxf(m, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))));
      m = fmaxf(m, fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
    } else {
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(x) + g * per_group) + i);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  __shared__ float warp_max[8];
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 1; i < 8; ++i) m = fmaxf(m, warp_max[i]);
    atomicMax(out + g, __float_as_uint(m));
  }
}

__global__ void amax_to_scale_kernel(float* __restrict__ inout, int l, float numerator) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= l) return;
  const float amax = inout[g];
  inout[g] = __fdiv_rn(numerator, amax == 0.0f ? 1.0f : amax);
}

int quantize_mxfp8_rows(const void* x, int x_dtype, const int32_t* group_offsets, const int32_t* group_rows,
                        void* q, void* sf, int sf_layout, int l, long long rows, int k, void* stream) {
  if (!x || !q || !sf) return fail(MSC_ERR_BAD_ARG, "NULL pointer");
  if (rows <= 0 || k <= 0) return fail(MSC_ERR_BAD_ARG, "sizes must be positive");
  if (k % 128) return fail(MSC_ERR_BAD_ARG, "k=%d must be a multiple of 128", k);
  if (x_dtype != 0 && x_dtype != 1) return fail(MSC_ERR_UNSUPPORTED, "x_dtype must be 0 (bf16) or 1 (f32)");
  if (sf_layout & ~(1 | MSC_SF_ZERO_REST))
    return fail(MSC_ERR_BAD_ARG, "sf_layout must be 0 or 1, plus MSC_SF_ZERO_REST where wanted");
  if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(q) % 8 ||
      reinterpret_cast<uintptr_t>(sf) % 4)
    return fail(MSC_ERR_BAD_ARG, "x must be 16-byte aligned, q 8-byte aligned, sf 4-byte aligned");
  if (rows > 0x7fffff00LL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
  QuantParams p = {};
  p.x = x; p.q = static_cast<uint8_t*>(q); p.sf = static_cast<uint8_t*>(sf);
  p.group_rows = group_rows; p.group_offsets = group_offsets;
  p.l = l; p.k = k; p.rows_total = (int)rows;
  p.tiled = sf_layout & 1;
  p.zero_rest = (sf_layout & MSC_SF_ZERO_REST) != 0;
  return launch_quantize_rows<FMT_MXFP8>(p, x_dtype ? IN_F32 : IN_BF16, 0, static_cast<cudaStream_t>(stream));
}

}  // namespace msc

extern "C" {

int msc_mxfp8_quantize(const void* x, int x_dtype, void* q, void* sf, int sf_layout, int rows, int k,
                       void* stream) {
  return msc::quantize_mxfp8_rows(x, x_dtype, nullptr, nullptr, q, sf, sf_layout, 0, rows, k, stream);
}

int msc_mxfp8_quantize_ragged(const void* x, int x_dtype, const int32_t* group_offsets,
                              const int32_t* group_rows, void* q, void* sf, int l, int rows_total, int k,
                              void* stream) {
  if (!group_offsets || !group_rows || l <= 0)
    return msc::fail(MSC_ERR_BAD_ARG, "group_offsets, group_rows and l > 0 are required");
  return msc::quantize_mxfp8_rows(x, x_dtype, group_offsets, group_rows, q, sf, 1, l, rows_total, k, stream);
}

int msc_amax_global_scale(const void* x, int x_dtype, int l, long long elems_per_group, float numerator,
                          float* global_scale, void* stream) {
  if (!x || !global_scale) return msc::fail(MSC_ERR_BAD_ARG, "NULL pointer");
  if (l <= 0 || elems_per_group <= 0) return msc::fail(MSC_ERR_BAD_ARG, "sizes must be positive");
  if (elems_per_group % 8) return msc::fail(MSC_ERR_BAD_ARG, "elems_per_group must be a multiple of 8");
  if (l > 65535) return msc::fail(MSC_ERR_UNSUPPORTED, "l=%d exceeds 65535 groups", l);
  if (x_dtype != 0 && x_dtype != 1) return msc::fail(MSC_ERR_UNSUPPORTED, "x_dtype must be 0 (bf16) or 1 (f32)");
  if (reinterpret_cast<uintptr_t>(x) % 16) return msc::fail(MSC_ERR_BAD_ARG, "x must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MSC_CUDA_OK(cudaMemsetAsync(global_scale, 0, sizeof(float) * l, st));
  // enough blocks per group to fill the machine a few times over, never more than the group has work for
  const long long vecs = elems_per_group / 8;
  long long per_group = (vecs + 256 * 8 - 1) / (256 * 8);
  const long long want = (long long)msc::num_sms() * 8 / l + 1;
  if (per_group > want) per_group = want;
  if (per_group < 1) per_group = 1;
  msc::amax_groups_kernel<<<dim3((unsigned)per_group, (unsigned)l), 256, 0, st>>>(
      x, x_dtype, elems_per_group, reinterpret_cast<unsigned int*>(global_scale));
  MSC_CUDA_OK(cudaGetLastError());
  msc::amax_to_scale_kernel<<<(l + 255) / 256, 256, 0, st>>>(global_scale, l, numerator);
  MSC_CUDA_OK(cudaGetLastError());
  return MSC_OK;
}

}  // extern "C"
