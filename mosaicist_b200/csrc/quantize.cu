// NVFP4 quantisation kernels (HBM-bound): activations -> packed e2m1 + one e4m3 scale per
// 16 K-elements, with the scales written either row-major or directly in the 128-row MMA
// tiling the GEMM reads; SiLU(gate)*up fused in front of the same quantiser; and the
// stand-alone scale re-tiling kernel.
//
// Arithmetic follows quantize_nvfp4 (experiments/flashinfer-megamoe-sm100a/nvfp4.py:39-57):
//   sf   = e4m3( clip(amax / 6 * gs, 0, 448) )        per block of 16
//   step = f32(sf) / gs
//   q    = e2m1_rne( clip(x / step, -6, 6) )           (0 when step == 0)
// every operation in IEEE fp32 (explicit _rn intrinsics, so no contraction or approximate
// division can change a rounding).  The kernel is quantize_rows_kernel (quantize_rows.cuh).
#include "quantize_rows.cuh"

namespace msc {

// (groups, mn, kwords*4) row-major scale bytes -> (groups, ceil(mn/128), kwords, 32, 16),
// padding rows zero.  One thread per 32-bit word of the output.
__global__ void __launch_bounds__(256)
sf_swizzle_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int groups, int mn,
                  int kwords) {
  const int tiles = (mn + 127) >> 7;
  const long long total = (long long)groups * tiles * kwords * 128;
  const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= total) return;
  // w enumerates [g][t][c][b][a]: consecutive threads write consecutive words
  const int a = (int)(w & 3);
  const int b = (int)((w >> 2) & 31);
  long long rest = w >> 7;
  const int c = (int)(rest % kwords);
  rest /= kwords;
  const int t = (int)(rest % tiles);
  const int g = (int)(rest / tiles);
  const int row = t * 128 + a * 32 + b;
  uint32_t val = 0;
  if (row < mn)
    val = __ldg(reinterpret_cast<const uint32_t*>(src + ((size_t)g * mn + row) * kwords * 4) + c);
  reinterpret_cast<uint32_t*>(dst)[w] = val;
}

// The same re-tiling through shared memory: a CTA takes 32 bytes (8 words) of each of a tile's
// 128 rows - two lanes read one full sector of a row - and writes eight 512-byte chunks of the
// tiling with one 16-byte store per thread.  The tile's rows sit at a 9-word pitch, so the
// column reads of the second phase fall in 32 different banks.  With rows_used (device, one
// group only) tiles at or beyond that row are left alone.  Needs kwords % 4 == 0 and 16-byte
// aligned pointers.
__global__ void __launch_bounds__(256)
sf_swizzle_tile_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int groups, int mn,
                       int kwords, const int* __restrict__ rows_used) {
  __shared__ uint32_t tile[128 * 9];
  const int tiles = (mn + 127) >> 7;
  const int cgroups = (kwords + 7) >> 3;
  const int cg = blockIdx.x % cgroups;
  const int rest = blockIdx.x / cgroups;
  const int t = rest % tiles, g = rest / tiles;
  if (rows_used && t * 128 >= __ldg(rows_used)) return;   // uniform over the CTA
  {
    const int row_l = threadIdx.x >> 1, half = threadIdx.x & 1;
    const int row = t * 128 + row_l, c0 = cg * 8 + half * 4;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row < mn && c0 < kwords)
      v = __ldg(reinterpret_cast<const uint4*>(src + ((size_t)g * mn + row) * kwords * 4 + (size_t)c0 * 4));
    uint32_t* d = tile + row_l * 9 + half * 4;
    d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
  }
  __syncthreads();
  const int cc = threadIdx.x >> 5, b = threadIdx.x & 31;
  const int c = cg * 8 + cc;
  if (c < kwords) {
    const uint4 o = make_uint4(tile[b * 9 + cc], tile[(32 + b) * 9 + cc], tile[(64 + b) * 9 + cc],
                               tile[(96 + b) * 9 + cc]);
    *reinterpret_cast<uint4*>(dst + ((((size_t)g * tiles + t) * kwords + c) * 32 + b) * 16) = o;
  }
}

int launch_sf_swizzle(const void* sf_rowmajor, void* sf_tiled, int groups, int mn, int kwords,
                      const int* rows_used, cudaStream_t stream) {
  const long long tiles = (mn + 127) / 128;
  const bool by_tiles = kwords % 4 == 0 && reinterpret_cast<uintptr_t>(sf_rowmajor) % 16 == 0 &&
                        reinterpret_cast<uintptr_t>(sf_tiled) % 16 == 0;
  if (by_tiles) {
    const long long blocks = (long long)groups * tiles * ((kwords + 7) / 8);
    if (blocks > 0x7fffffffLL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
    sf_swizzle_tile_kernel<<<(unsigned)blocks, 256, 0, stream>>>(
        static_cast<const uint8_t*>(sf_rowmajor), static_cast<uint8_t*>(sf_tiled), groups, mn, kwords,
        groups == 1 ? rows_used : nullptr);
  } else {
    const long long total = (long long)groups * tiles * kwords * 128;
    const long long blocks = (total + 255) / 256;
    if (blocks > 0x7fffffffLL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
    sf_swizzle_kernel<<<(unsigned)blocks, 256, 0, stream>>>(
        static_cast<const uint8_t*>(sf_rowmajor), static_cast<uint8_t*>(sf_tiled), groups, mn, kwords);
  }
  MSC_CUDA_OK(cudaGetLastError());
  return MSC_OK;
}

int quantize_nvfp4_rows(const void* x, int x_dtype, const float* gs, const int32_t* group_offsets,
                        const int32_t* group_rows, void* q, void* sf, int sf_layout, int l,
                        long long rows_total, int m_stride, int k, int silu, void* zero_out, void* stream) {
  if (!x || !gs || !q || !sf) return fail(MSC_ERR_BAD_ARG, "NULL pointer");
  if (l <= 0 || rows_total <= 0 || k <= 0) return fail(MSC_ERR_BAD_ARG, "sizes must be positive");
  if (k % 64) return fail(MSC_ERR_BAD_ARG, "k=%d must be a multiple of 64", k);
  if (x_dtype != 0 && x_dtype != 1) return fail(MSC_ERR_UNSUPPORTED, "x_dtype must be 0 (bf16) or 1 (f32)");
  if (silu && x_dtype != 0) return fail(MSC_ERR_UNSUPPORTED, "the fused SiLU form takes bf16 input");
  if (sf_layout & ~(1 | MSC_SF_ZERO_REST))
    return fail(MSC_ERR_BAD_ARG, "sf_layout must be 0 or 1, plus MSC_SF_ZERO_REST where wanted");
  if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(q) % 16 ||
      reinterpret_cast<uintptr_t>(sf) % 4)
    return fail(MSC_ERR_BAD_ARG, "x and q must be 16-byte aligned, sf 4-byte aligned");
  if (rows_total > 0x7fffff00LL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
  QuantParams p = {};
  p.x = x; p.gs = gs; p.group_rows = group_rows; p.group_offsets = group_offsets;
  p.q = static_cast<uint8_t*>(q); p.sf = static_cast<uint8_t*>(sf);
  p.zero_out = static_cast<__nv_bfloat16*>(zero_out);
  p.l = l; p.k = k; p.rows_total = (int)rows_total;
  p.tiled = sf_layout & 1;
  p.zero_rest = (sf_layout & MSC_SF_ZERO_REST) != 0;
  return launch_quantize_rows<FMT_NVFP4>(p, silu ? IN_SILU : x_dtype ? IN_F32 : IN_BF16, m_stride,
                                         static_cast<cudaStream_t>(stream));
}

}  // namespace msc

extern "C" {

int msc_nvfp4_quantize(const void* x, int x_dtype, const float* global_scale,
                       const int32_t* masked_m, void* q, void* sf, int sf_layout, int l, int m,
                       int k, void* stream) {
  if (m <= 0) return msc::fail(MSC_ERR_BAD_ARG, "m must be positive");
  if ((sf_layout & 1) && m % 128)
    return msc::fail(MSC_ERR_BAD_ARG, "tiled scales need m %% 128 == 0 in the masked layout");
  return msc::quantize_nvfp4_rows(x, x_dtype, global_scale, nullptr, masked_m, q, sf, sf_layout, l,
                              (long long)l * m, m, k, 0, nullptr, stream);
}

int msc_nvfp4_silu_mul_quantize(const void* gateup, const float* global_scale,
                                const int32_t* masked_m, void* q, void* sf, int sf_layout, int l,
                                int m, int n, void* stream) {
  if (m <= 0) return msc::fail(MSC_ERR_BAD_ARG, "m must be positive");
  if ((sf_layout & 1) && m % 128)
    return msc::fail(MSC_ERR_BAD_ARG, "tiled scales need m %% 128 == 0 in the masked layout");
  return msc::quantize_nvfp4_rows(gateup, 0, global_scale, nullptr, masked_m, q, sf, sf_layout, l,
                              (long long)l * m, m, n, 1, nullptr, stream);
}

int msc_nvfp4_quantize_ragged(const void* x, int x_dtype, const float* global_scale,
                              const int32_t* group_offsets, const int32_t* group_rows, void* q,
                              void* sf, int l, int rows_total, int k, int silu, void* stream) {
  if (!group_offsets || !group_rows)
    return msc::fail(MSC_ERR_BAD_ARG, "group_offsets and group_rows are required");
  return msc::quantize_nvfp4_rows(x, x_dtype, global_scale, group_offsets, group_rows, q, sf, 1, l,
                                  rows_total, 0, k, silu, nullptr, stream);
}

int msc_quantize_rows(int format, const void* x, int x_form, const float* global_scale,
                      const int32_t* group_offsets, const int32_t* group_rows, void* q, void* sf,
                      int sf_layout, void* zero_out_bf16, int l, int rows_total, int m_stride, int k,
                      void* stream) {
  if (x_form < 0 || x_form > 2) return msc::fail(MSC_ERR_UNSUPPORTED, "x_form must be 0 (bf16), 1 (f32) or 2 (gate | up)");
  if (group_offsets && !group_rows)
    return msc::fail(MSC_ERR_BAD_ARG, "group_offsets needs group_rows");
  if (format == 0) {
    if (!group_offsets) {
      if (m_stride <= 0) return msc::fail(MSC_ERR_BAD_ARG, "m must be positive");
      if ((sf_layout & 1) && m_stride % 128)
        return msc::fail(MSC_ERR_BAD_ARG, "tiled scales need m %% 128 == 0 in the masked layout");
      if (rows_total > (long long)l * m_stride)
        return msc::fail(MSC_ERR_BAD_ARG, "rows_total=%d exceeds l * m_stride", rows_total);
    }
    if (zero_out_bf16 && (x_form == 2 || reinterpret_cast<uintptr_t>(zero_out_bf16) % 16))
      return msc::fail(MSC_ERR_BAD_ARG, "zero_out takes the shape of x and 16-byte alignment");
    return msc::quantize_nvfp4_rows(x, x_form == 1, global_scale, group_offsets, group_rows, q, sf, sf_layout, l,
                                    rows_total, m_stride, k, x_form == 2, zero_out_bf16, stream);
  }
  if (format != 1) return msc::fail(MSC_ERR_UNSUPPORTED, "format must be 0 (NVFP4) or 1 (MXFP8)");
  if (x_form == 2 || zero_out_bf16) return msc::fail(MSC_ERR_UNSUPPORTED, "not built for MXFP8");
  if (!group_offsets != !group_rows || (group_offsets && l <= 0))
    return msc::fail(MSC_ERR_BAD_ARG, "group_offsets, group_rows and l > 0 go together");
  return msc::quantize_mxfp8_rows(x, x_form, group_offsets, group_rows, q, sf, sf_layout, l, rows_total, k, stream);
}

int msc_sf_swizzle(const void* sf_rowmajor, void* sf_tiled, int groups, int mn, int k_scales,
                   void* stream) {
  if (!sf_rowmajor || !sf_tiled) return msc::fail(MSC_ERR_BAD_ARG, "NULL pointer");
  if (groups <= 0 || mn <= 0 || k_scales <= 0) return msc::fail(MSC_ERR_BAD_ARG, "sizes must be positive");
  if (k_scales % 4) return msc::fail(MSC_ERR_BAD_ARG, "k_scales=%d must be a multiple of 4", k_scales);
  if (reinterpret_cast<uintptr_t>(sf_rowmajor) % 4 || reinterpret_cast<uintptr_t>(sf_tiled) % 4)
    return msc::fail(MSC_ERR_BAD_ARG, "scale pointers must be 4-byte aligned");
  return msc::launch_sf_swizzle(sf_rowmajor, sf_tiled, groups, mn, k_scales / 4, nullptr,
                                static_cast<cudaStream_t>(stream));
}

}  // extern "C"
