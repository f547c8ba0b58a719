// Pieces shared by the block-scaled GEMM kernels: launch parameters, the tile walker and the
// debug-build trace hooks.
#pragma once

#include "host_common.h"
#include "ptx.cuh"

#include <cuda_bf16.h>

namespace msc {

enum : int { KIND_NVFP4 = 0, KIND_MXFP8 = 1 };

struct GemmParams {
  const uint8_t* sfa;        // [row_tiles][sf_chunks][512]
  const uint8_t* sfb;        // [l][n/128][sf_chunks][512]
  const float* alpha;        // [l] or null
  const float* alpha_gs_a;   // [l] or null, with alpha_gs_b: the group's factor is
  const float* alpha_gs_b;   // alpha / (alpha_gs_a * alpha_gs_b), the two-level scales' fold
  const float* row_scale;    // [rows_total] or null
  const int* group_rows;     // [l] or null (= m_stride)
  const int* group_offsets;  // [l] or null (= g * m_stride)
  __nv_bfloat16* out;        // [rows_total][n]
  int* status;
  int l, m_stride, n;
  int rows_total;            // rows of a_q / out: no group may reach beyond them
  int k_stages;              // ceil(k_bytes / 128)
  int sf_chunks;             // scale chunks along K per 128-row tile
  int raster;
  // fused SwiGLU + requantise epilogue (B holds gate rows then up rows, n = 2 x width):
  uint8_t* out_q;            // (rows_total, n/4) packed e2m1 of silu(gate) * up
  uint8_t* out_sf;           // its e4m3 scales, tiled (rows_total/128, n/128, 32, 16)
  const float* out_gs;       // [l] global scale of the activation
  // row-scatter epilogue: row r goes to scatter_base[code >> 26] + (code & 0x3ffffff) * n bf16,
  // code = row_dest[r]; negative codes are skipped
  const int* row_dest;       // [rows_total] or null
  uint8_t* scatter_base[16]; // unused entries are null: rows coded for them are skipped
  int scatter_count;         // destinations in use; codes naming another one are refused
  int scatter_rows;          // rows every destination holds; codes beyond them are refused
#ifdef MSC_DEBUG
  unsigned long long* trace;  // [cta][8 tiles][3 roles][2] clock64 stamps, then [cta][2] at the end
  int debug_flags;            // 1: skip global stores, 2: skip scale loads/copies, 4: skip MMAs
#endif
};

#ifdef MSC_DEBUG
extern unsigned long long* g_trace;
extern int g_debug_flags;
#define MSC_STAMP(role, tl, which)                                                        \
  do {                                                                                    \
    if (p.trace && (tl) < 8 && (threadIdx.x & 31) == 0)                                                            \
      p.trace[(((size_t)blockIdx.x * 8 + (tl)) * 3 + (role)) * 2 + (which)] = clock64();  \
  } while (0)
#define MSC_FLAG(bit) (p.debug_flags & (bit))
// fine stamps: [cta][32] after the per-CTA begin/end pairs; taken for tile 1, K stage 4
#define MSC_FINE(slot)                                                                     \
  do {                                                                                     \
    if (p.trace && tl == 1 && kb == 4)                                                     \
      p.trace[(size_t)gridDim.x * 50 + (size_t)blockIdx.x * 32 + (slot)] = clock64();      \
  } while (0)
#else
#define MSC_FINE(slot) do {} while (0)
#define MSC_STAMP(role, tl, which) do {} while (0)
#define MSC_FLAG(bit) false
#endif

// Factor of a group's accumulators.
__device__ __forceinline__ float group_alpha(const GemmParams& p, int g) {
  if (!p.alpha) return 1.0f;
  const float a = ld_ordered(p.alpha + g);
  if (!p.alpha_gs_a) return a;
  return __fdiv_rn(a, __fmul_rn(ld_ordered(p.alpha_gs_a + g), ld_ordered(p.alpha_gs_b + g)));
}

// Finds the group of a tile, 32 groups at a time: lane i of the (converged) warp holds the running
// tile count at group i of the current window, so that passing a group costs a share of one load and
// five shuffles instead of two dependent loads of its own.  For the kernels that meet hundreds of
// groups: a batch of 256 of which a decode step uses 100 spent 1000 cycles per tile in each role on
// the walk.  With a handful of groups the plain walk of TileCursor is ahead (8 groups of 512 rows:
// 15.3 against 15.7 us).  Tiles are asked for in increasing order.
// KEEP: the lanes also hold their groups' rows and offsets.  An epilogue that has no registers to
// spare and time to wait reads the two words of the found group again (from L2: the operand ring
// leaves L1 no room).
template <bool KEEP>
struct GroupWindow {
  int next = 0;    // first group behind the window
  int end = 0;     // tiles of all groups up to there
  int end_l = 0;   // tiles up to and including this lane's group
  int rows_l = 0, off_l = 0;
  // load(g, rows, off) reads the tables, tiles_of(rows) counts; first = tile id the group starts at
  template <class Load, class Tiles>
  __device__ __forceinline__ bool find(int l, int t, Load load, Tiles tiles_of, int& g, int& rows, int& off, int& first) {
    const int lane = threadIdx.x & 31;
    while (t >= end) {
      if (next >= l) return false;
      int incl = 0;
      if (next + lane < l) {
        load(next + lane, rows_l, off_l);
        incl = tiles_of(rows_l);
      }
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
      }
      end_l = end + incl;
      end = __shfl_sync(0xffffffffu, end_l, 31);
      next += 32;
    }
    const int i = __ffs(__ballot_sync(0xffffffffu, t < end_l)) - 1;
    g = next - 32 + i;
    // every lane the same: the broadcast tells the compiler that the role bodies stay warp-uniform
    if (!KEEP) load(g, rows_l, off_l);
    rows = __shfl_sync(0xffffffffu, rows_l, KEEP ? i : 0);
    off = __shfl_sync(0xffffffffu, off_l, KEEP ? i : 0);
    first = __shfl_sync(0xffffffffu, end_l, i) - tiles_of(rows);
    return true;
  }
};

// Rows and offset of a group.  A group table that reaches beyond the buffers (an overflowing
// expert-parallel step, a stale table after a timed-out wait) is cut to what the buffers hold.
__device__ __forceinline__ void load_group(const int* group_rows, const int* group_offsets, int rows_total, int g,
                                           int& rows, int& off) {
  rows = max(ld_ordered(group_rows + g), 0);
  off = ld_ordered(group_offsets + g);
  if (off < 0 || off >= rows_total) rows = 0;
  else if (rows > rows_total - off) rows = rows_total - off;
}

// Walks the flattened (group, m-tile, n-tile) space in increasing tile id.
struct TileCursor {
  int g = 0, base = 0, mtiles = 0, rows = 0, off = 0;
  int mshift = 7;  // log2 of the rows one tile covers: 7 for one CTA, 8 for a CTA pair
  bool primed = false;
  __device__ __forceinline__ bool seek(const GemmParams& p, int ntiles, int t, int& mt, int& nt) {
    while (true) {
      if (!primed) {
        if (g >= p.l) return false;
        // every lane reads the same words, both loads under way before either is waited for; the
        // broadcasts tell the compiler that all lanes agree
        const int r = p.group_rows ? ld_ordered(p.group_rows + g) : p.m_stride;
        const int o = p.group_offsets ? ld_ordered(p.group_offsets + g) : g * p.m_stride;
        rows = __shfl_sync(0xffffffffu, r, 0);
        off = __shfl_sync(0xffffffffu, o, 0);
        if (rows < 0) rows = 0;
        if (p.m_stride > 0 && rows > p.m_stride) rows = p.m_stride;
        // a group table that reaches beyond the buffers (an overflowing expert-parallel step,
        // a stale table after a timed-out wait) is cut to what the buffers hold
        if (off < 0 || off >= p.rows_total) rows = 0;
        else if (rows > p.rows_total - off) rows = p.rows_total - off;
        mtiles = (rows + (1 << mshift) - 1) >> mshift;
        primed = true;
      }
      const int tiles = mtiles * ntiles;
      if (t < base + tiles) break;
      base += tiles;
      ++g;
      primed = false;
    }
    const int u = t - base;
    if (p.raster == 0) {
      mt = u / ntiles;
      nt = u - mt * ntiles;
    } else {
      nt = u / mtiles;
      mt = u - nt * mtiles;
    }
    return true;
  }
};

// Body of the block-scaled entry points (gemm_blockscaled.cu): k_bytes and chunk size follow from
// kind; gs_a / gs_b as in GemmParams.
int grouped_gemm(int kind, const void* a_q, const void* a_sf, const void* b_q, const void* b_sf,
                 const float* alpha, const int32_t* group_offsets, const int32_t* group_rows,
                 const float* row_scale, void* out, int l, long long rows_total, int m_stride, int n, int k,
                 const msc_gemm_cfg* cfg_in, void* stream_v, const float* gs_a = nullptr,
                 const float* gs_b = nullptr);

// Launcher of the CTA-pair kernel (gemm_blockscaled_pair.cu).
int launch_pair_gemm(int kind, const void* a_q, const void* b_q, long long rows_total, long long k_bytes,
                     const GemmParams& p, int stages, int max_ctas, cudaStream_t stream,
                     bool sf_by_warps);

// Launcher of the tokens-on-N kernel (gemm_blockscaled_swap.cu): row-concatenated groups.
int launch_swap_gemm(int kind, const void* a_q, const void* b_q, long long rows_total, long long k_bytes,
                     const GemmParams& p, int max_ctas, cudaStream_t stream);

}  // namespace msc
