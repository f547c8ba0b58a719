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

#include <algorithm>

namespace msc {

// max |x| per group into out[g] (as fp32 bit patterns, which order like unsigned integers).
// Bound by HBM.  A block takes `rounds` pieces of 1024 16-byte vectors, four loads of a thread in
// flight, and blocks walk the batch from its END: the quantiser that follows starts at the
// beginning, which then is what L2 still holds.  8 x 2048 x 7168 bf16, cold: 66 -> 50 us (4.7 TB/s)
// against one load in flight per thread, all groups walked at once.
template <bool F32>
__global__ void __launch_bounds__(256)
amax_groups_kernel(const uint4* __restrict__ x, long long vecs, int rounds, unsigned int* __restrict__ out) {
  grid_launch_dependents();
  const int g = gridDim.y - 1 - blockIdx.y;
  const uint4* src = x + (size_t)g * vecs;
  long long i = (long long)(gridDim.x - 1 - blockIdx.x) * rounds * 1024 + threadIdx.x;
  float m = 0.0f;
  for (int r = 0; r < rounds; ++r, i += 1024) {
    uint4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = i + j * 256 < vecs ? __ldg(src + i + j * 256) : make_uint4(0u, 0u, 0u, 0u);
    if (F32) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        m = fmaxf(m, fmaxf(fmaxf(fabsf(__uint_as_float(v[j].x)), fabsf(__uint_as_float(v[j].y))),
                           fmaxf(fabsf(__uint_as_float(v[j].z)), fabsf(__uint_as_float(v[j].w)))));
    } else {
      __nv_bfloat162 h = __float2bfloat162_rn(0.0f);   // (a NaN never replaces a number)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v[j]);
        h = __hmax2(h, __hmax2(__hmax2(__habs2(p[0]), __habs2(p[1])), __hmax2(__habs2(p[2]), __habs2(p[3]))));
      }
      m = fmaxf(m, fmaxf(__low2float(h), __high2float(h)));
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  __shared__ float warp_max[8];
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmaxf(m, warp_max[w]);
    atomicMax(out + g, __float_as_uint(m));
  }
}

__global__ void amax_to_scale_kernel(float* __restrict__ inout, int l, float numerator) {
  grid_dependency_wait();
  grid_launch_dependents();
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
  // up to four pieces of 16 KB per block, as long as every SM still gets its eight blocks
  const long long vecs = elems_per_group / (x_dtype ? 4 : 8);
  const long long pieces = (vecs + 1023) / 1024;
  const int sms = msc::num_sms();
  if (sms <= 0) return msc::fail(MSC_ERR_CUDA, "could not query the SM count");
  const long long per_sm = pieces * l / (8LL * sms);
  const long long least = (pieces + 0x7ffffffeLL) / 0x7fffffffLL;   // the grid's x extent is 31 bits
  const long long rounds = std::max(least, std::min(4LL, std::max(1LL, per_sm)));
  const dim3 grid((unsigned)((pieces + rounds - 1) / rounds), (unsigned)l);
  const uint4* src = static_cast<const uint4*>(x);
  unsigned int* bits = reinterpret_cast<unsigned int*>(global_scale);
  if (x_dtype) msc::amax_groups_kernel<true><<<grid, 256, 0, st>>>(src, vecs, (int)rounds, bits);
  else msc::amax_groups_kernel<false><<<grid, 256, 0, st>>>(src, vecs, (int)rounds, bits);
  MSC_CUDA_OK(cudaGetLastError());
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t lc = msc::pdl_launch_config((l + 255) / 256, 256, 0, st, attr);
  MSC_CUDA_OK(cudaLaunchKernelEx(&lc, msc::amax_to_scale_kernel, global_scale, l, numerator));
  return MSC_OK;
}

}  // extern "C"
