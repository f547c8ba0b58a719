// The row quantiser behind every stand-alone quantise entry point (NVFP4, NVFP4 of
// SiLU(gate) * up, MXFP8): one kernel template over the output format, the input form and the layout
// (masked batches or ragged groups).
//
// A thread owns 16 consecutive K-elements of FOUR rows, the rows 32 a + b (a = 0..3) of a
// 128-row tile: in the 128-row MMA tiling the four scale words of those rows are 16 consecutive
// bytes, so the scales of a tile leave as 16-byte stores of one lane in four (NVFP4) or eight
// (MXFP8) instead of 4-byte words 512 bytes apart, each of which costs an L2 transaction of its
// own.  The loads of the four rows are issued before anything is computed; a warp reads 1 KB of
// a row at a time.  Which rows are live is a property of the quad (its 128-row tile lies in one
// ragged group, unless a group starts inside it) or of the row (masked batches), and the index
// arithmetic of the four blocks is shared: multiplications by precomputed reciprocals instead of
// 64-bit divisions.
//
// Bound by HBM for MXFP8 and by a mix of issue slots and HBM for NVFP4.  Cold, 16384 x 7168,
// against one thread per block with its own row search: MXFP8 bf16 99 -> 62 us (5.7 TB/s), ragged
// groups 138 -> 62 us, fp32 106 -> 97 us; NVFP4 bf16 95 -> 71 us (4.3 TB/s), fp32 103 -> 97 us,
// SiLU * up 132 -> 106 us.  One kernel for both layouts, with the search of single rows inside it, cost
// registers: 9 ragged groups of 666 rows, k 1920, 6.3 -> 6.7 us (6.3 with the search out of line and the
// layouts apart).
#pragma once

#include "host_common.h"
#include "ptx.cuh"
#include "quantize_common.cuh"

namespace msc {

enum : int { FMT_NVFP4 = 0, FMT_MXFP8 = 1 };
enum : int { IN_BF16 = 0, IN_F32 = 1, IN_SILU = 2 };

// n / d for n < 2^31 as one multiplication: mul = ceil(2^(31 + s) / d), s = ceil(log2 d).
struct FastDiv {
  uint32_t mul, shift, d;
  static FastDiv make(uint32_t d) {
    FastDiv f;
    f.d = d;
    uint32_t s = 0;
    while ((1ull << s) < d) ++s;
    f.shift = s ? s - 1 : 0;
    f.mul = s ? (uint32_t)(((1ull << (31 + s)) + d - 1) / d) : 0u;   // d == 1 needs no division
    return f;
  }
  __device__ __forceinline__ uint32_t div(uint32_t n) const { return d == 1 ? n : __umulhi(n, mul) >> shift; }
};

struct QuantParams {
  const void* x;            // (rows_total, k) or, with IN_SILU, (rows_total, 2k) gate | up
  const float* gs;          // (l) per-group global scale (NVFP4)
  const int* group_rows;    // (l) or null: rows at or beyond it are not live
  const int* group_offsets; // (l) ascending, or null: group g starts at g * m_stride
  uint8_t* q;               // (rows_total, k/2) e2m1 pairs or (rows_total, k) e4m3
  uint8_t* sf;              // tiled or row-major scale bytes
  __nv_bfloat16* zero_out;  // (rows_total, k) or null: rows that are not live are set to zero here
  int l, k, rows_total;
  int tiled;                // scale layout
  int zero_rest;            // write zero scales for rows that are not live
  int wide;                 // bit 0: sf is 16-byte aligned, bit 1: q is
  int quads;                // 32 per 128-row tile
  FastDiv kb_div;           // by k / 16
  FastDiv m_div;            // by m_stride (masked layout)
};

// Owner of row `row0` in the ragged layout: the last group whose offset is <= row0 (offsets ascend; an
// empty group shares the offset of the group after it); -1 before the first group.  Also says whether
// a group starts inside the 127 rows after it.  The lanes of a converged warp ask about the same row
// and each compares every 32nd offset.
__device__ __forceinline__ int owner_of_tile(const int* offsets, int l, int row0, bool& shared) {
  const int lane = threadIdx.x & 31;
  int count = 0, upto = 0;
  for (int base = 0; base < l; base += 32) {
    const int g = base + lane;
    const int off = g < l ? ld_ordered(offsets + g) : 0x7fffffff;
    count += __popc(__ballot_sync(0xffffffffu, off <= row0));
    upto += __popc(__ballot_sync(0xffffffffu, off <= row0 + 127));
  }
  shared = upto != count;
  return count - 1;
}
// The same for one thread's row.
__device__ __forceinline__ int owner_of_row(const int* offsets, int l, int row) {
  int lo = -1, hi = l - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (ld_ordered(offsets + mid) <= row) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <int IN>
constexpr int kInWords = IN == IN_BF16 ? 8 : 16;   // 32-bit words of input per block of 16

template <int IN>
__device__ __forceinline__ void load_block(const QuantParams& p, int row, int kb, uint32_t* raw) {
  if (IN == IN_BF16) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.x) + (size_t)row * p.k + kb * 16);
    *reinterpret_cast<uint4*>(raw) = ld_ordered(src);
    *reinterpret_cast<uint4*>(raw + 4) = ld_ordered(src + 1);
  } else if (IN == IN_F32) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const float*>(p.x) + (size_t)row * p.k + kb * 16);
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(raw + 4 * j) = ld_ordered(src + j);
  } else {
    const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(p.x) + (size_t)row * 2 * p.k + kb * 16;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      *reinterpret_cast<uint4*>(raw + 4 * j) = ld_ordered(reinterpret_cast<const uint4*>(base) + j);
      *reinterpret_cast<uint4*>(raw + 8 + 4 * j) = ld_ordered(reinterpret_cast<const uint4*>(base + p.k) + j);
    }
  }
}

// Quantises a block and stores its values if its row is live.  Made by whole warps: returns the scale
// word of the row, valid in lanes 0 mod 4 (NVFP4) or 0 mod 8 (MXFP8), zero bytes where not live.
template <int FMT, int IN>
__device__ __forceinline__ uint32_t quantize_block(const QuantParams& p, int row, int kb, uint32_t* raw, bool live, float gs) {
  float v[16];
  float amax;
  if (IN == IN_BF16) {
    amax = amax_bf16x16(raw);
    unpack_bf16x16(raw, v);
  } else if (IN == IN_F32) {
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(raw[e]);
    amax = amax_f32x16(v);
  } else {
    // row holds [gate (k) | up (k)] in bf16; the activation stays fp32 (nvfp4.py:81-88)
    float up[16];
    unpack_bf16x16(raw, v);
    unpack_bf16x16(raw + 8, up);
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = silu_mul(v[e], up[e]);
    amax = amax_f32x16(v);
  }
  uint32_t sfb = 0;
  if (FMT == FMT_NVFP4) {
    uint2 q8 = make_uint2(0u, 0u);
    if (live) {
      quantize_16_amax(v, amax, gs, q8, sfb);
      *reinterpret_cast<uint2*>(p.q + (size_t)row * (p.k >> 1) + kb * 8) = q8;
    }
    return gather_scale_word(sfb);              // lanes 0 mod 4: bytes of four blocks
  }
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));   // two lanes share a block of 32
  if (live) {
    sfb = mx_scale_byte(amax);
    const uint4 q16 = mx_pack_16(v, sfb);
    uint8_t* dst = p.q + (size_t)row * p.k + kb * 16;
    if (p.wide & 2) {
      *reinterpret_cast<uint4*>(dst) = q16;
    } else {
      reinterpret_cast<uint2*>(dst)[0] = make_uint2(q16.x, q16.y);
      reinterpret_cast<uint2*>(dst)[1] = make_uint2(q16.z, q16.w);
    }
  }
  uint32_t w = sfb;                             // lanes 0 mod 8: bytes of four blocks
  w |= __shfl_down_sync(0xffffffffu, sfb, 2) << 8;
  w |= __shfl_down_sync(0xffffffffu, sfb, 4) << 16;
  w |= __shfl_down_sync(0xffffffffu, sfb, 6) << 24;
  return w;
}
template <int FMT>
constexpr int kScaleLanes = FMT == FMT_NVFP4 ? 4 : 8;   // lanes (blocks of 16) per scale word

// The blocks of a warp that meets a tile inside which a group starts: the GEMMs want groups at
// multiples of 128, the quantisers alone take any ascending offsets.  One row at a time, each with
// its own group.  Out of line, so that it costs the kernel no registers.
template <int FMT, int IN>
__device__ __noinline__ void quantize_shared_tiles(const QuantParams& p, int row_b, int kb, bool have) {
#pragma unroll 1
  for (int a = 0; a < 4; ++a) {
    const int row = row_b + 32 * a;
    bool live = have && row < p.rows_total;
    float gs = 1.0f;
    if (live) {
      const int own = owner_of_row(p.group_offsets, p.l, row);
      live = own >= 0 && row < ld_ordered(p.group_offsets + own) + ld_ordered(p.group_rows + own);
      if (FMT == FMT_NVFP4 && live) gs = ld_ordered(p.gs + own);
    }
    uint32_t raw[kInWords<IN>];
#pragma unroll
    for (int w = 0; w < kInWords<IN>; ++w) raw[w] = 0u;
    if (live) load_block<IN>(p, row, kb, raw);
    if (p.zero_out && have && !live && row < p.rows_total) {
      uint4* dst = reinterpret_cast<uint4*>(p.zero_out + (size_t)row * p.k + kb * 16);
      dst[0] = dst[1] = make_uint4(0u, 0u, 0u, 0u);
    }
    const uint32_t word = quantize_block<FMT, IN>(p, row, kb, raw, live, gs);
    if (!have || (kb & (kScaleLanes<FMT> - 1))) continue;
    const int kw = kb / kScaleLanes<FMT>, kwords = (p.k >> 4) / kScaleLanes<FMT>;
    if (p.tiled) {
      if (live || p.zero_rest) *reinterpret_cast<uint32_t*>(p.sf + tiled_sf_word(row, kw, kwords)) = word;
    } else if (live || (p.zero_rest && row < p.rows_total)) {
      *reinterpret_cast<uint32_t*>(p.sf + ((size_t)row * kwords + kw) * 4) = word;
    }
  }
}

template <int FMT, int IN, bool RAGGED>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const __grid_constant__ QuantParams p) {
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t unit = blockIdx.x * 256u + threadIdx.x;
  const uint32_t quad = p.kb_div.div(unit);
  const int kblocks = (int)p.kb_div.d;
  const int kb = (int)(unit - quad * p.kb_div.d);
  const bool have = (int)quad < p.quads;    // whole warps stay for the shuffles
  const int tile = (int)(quad >> 5), b = (int)(quad & 31u);
  const int row_b = tile * 128 + b;         // row of a = 0

  // which of the four rows are live, and their global scales
  bool live[4];
  float gsv[4];
  if (RAGGED) {
    int g = 0, limit = 0;
    bool shared = false;
    // a warp spans at most two tiles when a row has 32 blocks or more; short rows take more steps
    uint32_t todo = __ballot_sync(0xffffffffu, have);
    while (todo) {
      const int lead = __ffs(todo) - 1;
      const int t = __shfl_sync(0xffffffffu, tile, lead);
      bool inside;
      const int own = owner_of_tile(p.group_offsets, p.l, t * 128, inside);
      shared = shared || inside;
      const uint32_t same = __ballot_sync(0xffffffffu, have && tile == t);
      if (have && tile == t && own >= 0) {
        g = own;
        limit = ld_ordered(p.group_offsets + own) + ld_ordered(p.group_rows + own);
      }
      todo &= ~same;
    }
    if (shared) {                           // the same for the whole warp
      quantize_shared_tiles<FMT, IN>(p, row_b, kb, have);
      return;
    }
    const float gs = FMT == FMT_NVFP4 && have ? ld_ordered(p.gs + g) : 1.0f;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int row = row_b + 32 * a;
      live[a] = have && row < p.rows_total && row < limit;
      gsv[a] = gs;
    }
  } else {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int row = row_b + 32 * a;
      live[a] = have && row < p.rows_total;
      gsv[a] = 1.0f;
      if (FMT == FMT_NVFP4 && live[a]) {
        const int g = (int)p.m_div.div((uint32_t)row);
        gsv[a] = ld_ordered(p.gs + g);
        if (p.group_rows) live[a] = row - g * (int)p.m_div.d < ld_ordered(p.group_rows + g);
      }
    }
  }

  constexpr int kAhead = IN == IN_BF16 ? 4 : 2;    // rows whose loads are issued together
  uint32_t words[4];                               // scale word of each row
#pragma unroll
  for (int a0 = 0; a0 < 4; a0 += kAhead) {
    uint32_t raw[kAhead][kInWords<IN>];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int row = row_b + 32 * (a0 + i);
#pragma unroll
      for (int w = 0; w < kInWords<IN>; ++w) raw[i][w] = 0u;
      if (live[a0 + i]) {
        load_block<IN>(p, row, kb, raw[i]);
      } else if (p.zero_out && have && row < p.rows_total) {
        uint4* dst = reinterpret_cast<uint4*>(p.zero_out + (size_t)row * p.k + kb * 16);
        dst[0] = dst[1] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      words[a0 + i] = quantize_block<FMT, IN>(p, row_b + 32 * (a0 + i), kb, raw[i], live[a0 + i], gsv[a0 + i]);
  }
  if (!have || (kb & (kScaleLanes<FMT> - 1))) return;
  const int kw = kb / kScaleLanes<FMT>, kwords = kblocks / kScaleLanes<FMT>;
  if (p.tiled) {
    uint8_t* dst = p.sf + tiled_sf_word(row_b, kw, kwords);
    const bool all = p.zero_rest || (live[0] && live[1] && live[2] && live[3]);   // dead rows' words are 0
    if (all && (p.wide & 1)) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(words[0], words[1], words[2], words[3]);
    } else {
#pragma unroll
      for (int a = 0; a < 4; ++a)
        if (all || live[a]) reinterpret_cast<uint32_t*>(dst)[a] = words[a];
    }
  } else {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int row = row_b + 32 * a;
      if (live[a] || (p.zero_rest && row < p.rows_total))
        *reinterpret_cast<uint32_t*>(p.sf + ((size_t)row * kwords + kw) * 4) = words[a];
    }
  }
}

// Fills in the index reciprocals and launches; the caller has validated sizes and pointers.
template <int FMT>
int launch_quantize_rows(QuantParams& p, int in_form, int m_stride, cudaStream_t stream) {
  const long long tiles = ((long long)p.rows_total + 127) / 128;
  const int kblocks = p.k / 16;
  const long long units = tiles * 32 * kblocks;
  if (units > 0x7fffff00LL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
  p.quads = (int)(tiles * 32);
  p.wide = (reinterpret_cast<uintptr_t>(p.sf) % 16 == 0 ? 1 : 0) | (reinterpret_cast<uintptr_t>(p.q) % 16 == 0 ? 2 : 0);
  p.kb_div = FastDiv::make((uint32_t)kblocks);
  p.m_div = FastDiv::make((uint32_t)(m_stride > 0 ? m_stride : 1));
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t lc = pdl_launch_config((int)((units + 255) / 256), 256, 0, stream, attr);
  const bool ragged = p.group_offsets != nullptr;
  auto launch = [&](auto kern) { return cudaLaunchKernelEx(&lc, kern, p); };
  if (in_form == IN_BF16)
    MSC_CUDA_OK(ragged ? launch(quantize_rows_kernel<FMT, IN_BF16, true>) : launch(quantize_rows_kernel<FMT, IN_BF16, false>));
  else if (in_form == IN_F32)
    MSC_CUDA_OK(ragged ? launch(quantize_rows_kernel<FMT, IN_F32, true>) : launch(quantize_rows_kernel<FMT, IN_F32, false>));
  else if constexpr (FMT == FMT_NVFP4)
    MSC_CUDA_OK(ragged ? launch(quantize_rows_kernel<FMT, IN_SILU, true>) : launch(quantize_rows_kernel<FMT, IN_SILU, false>));
  return MSC_OK;
}

}  // namespace msc
