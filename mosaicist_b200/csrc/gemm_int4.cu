// Grouped GEMM of bf16 activations with int4 weights, the weights expanded on their way into the
// tensor core: out[off_g + r] = bf16(alpha_g * a[off_g + r] . dequant(b[g])^T), dequant(b) =
// bf16( bf16(q) * scale ) (the reference's rounding order,
// ports/hopper_mixed_dtype_grouped_gemm/problems.py:75-87).
//
// The WEIGHTS are the MMA's M side and live in TENSOR MEMORY: a converter thread owns one weight
// row (TMEM lane), reads its packed nibbles from a swizzled shared-memory stage with 16-byte
// loads, expands 128 of them in registers and writes them with tcgen05.st as the A operand of the
// next eight MMAs.  The expanded weights therefore never touch shared memory - writing them
// there and reading them back for the MMA is what bounded the kernel that kept them on the N side
// (128 rows x 64 K cost 32 KB of shared-memory traffic per stage and 512-row tiles to amortise
// it).  The TOKENS are the N side, at a granularity of 16 (32 for pairs), so a group of a few rows
// costs a narrow MMA and not a 256- or 512-row tile: in a decode step the kernel streams the packed
// weights at the rate the converters or HBM allow.
//
// Roles (one CTA per SM; PAIR: two CTAs share an MMA of 256 weight rows, each expanding its own
// 128 and loading half of the tokens):
//   CONV (8 or 16) converter warps: lane quadrant w % 4, taking the 128-K stages in turn
//   EPI (8 or 4) epilogue warps: the accumulator is the output transposed (lane = output column,
//                       TMEM column = token): 32 x 32 pieces are turned around in shared memory
//   1 MMA warp, 1 producer warp for the packed weights, 1 for the tokens
// Rings: packed weights in stages of 256 K (16 KB: 128 bytes per row, whole 128-byte lines); tokens
// and expanded weights in stages of 128 K that share their barriers ("full": the tokens' bytes and
// the converter warps' arrivals; "empty": one commit).  Warps that only wait sleep between probes:
// their polling took a third of the issue slots from the converters.
//
// Finding a tile's group 32 at a time (GroupWindow) instead of walking the table took the passes of
// 64 groups, n = 2048, k = 7168 from 177 to 150 - 160 us (1 - 16 rows per group) and from 577 to
// 538 - 560 us (64 - 512 rows) back to back.  Before that, cold (the kernel before it, weights expanded into shared
// memory as the N-side operand of 512-row tiles, in brackets): 1 - 16 rows per group 182 us (469),
// 65 - 128 rows 241 us (472), 64 - 512 rows 417 - 441 us (595), 1320 - 1390 TFLOP/s.  With hundreds
// of rows the tensor pipe is the limit (it runs into the power cap); with a few rows it is the
// fixed cost of an MMA, about 65 cycles to fetch 128 rows x 16 K of A whatever N is, 107 us there.
#include "gemm_common.cuh"

namespace msc {

struct Int4Params {
  const __nv_bfloat16* scales;   // (l, n, k / group_size)
  const float* alpha;            // (l) or null
  const int* group_rows;
  const int* group_offsets;
  __nv_bfloat16* out;            // (rows_total, n)
  int* status;
  int l, n, rows_total;
  int kblocks;                   // k / 64
  int group_blocks;              // group_size / 64
};

template <bool PAIR, int TMAX, int PSTAGES, int CONV, int EPI>
struct Int4Smem {
  static constexpr int kStages = 4;                        // 128-K stages: tokens + expanded weights
  static constexpr int kTokHalf = TMAX / (PAIR ? 2 : 1) * 128;   // this CTA's tokens x 64 K
  static constexpr int kTok = 2 * kTokHalf;
  static constexpr int kPacked = 128 * 128;                // 128 weight rows x 256 K
  static constexpr int kThreads = (CONV + EPI + 3) * 32;
  static constexpr int kOffTok = 1024;
  static constexpr int kOffPacked = kOffTok + kStages * kTok;
  static constexpr int kOffC = kOffPacked + PSTAGES * kPacked;
  static constexpr int kBoxPitch = 36 * 4;                 // a token's 32 fp32 columns, padded
  static constexpr int kBoxBytes = 32 * kBoxPitch;
  static constexpr int kAlloc = kOffC + EPI * kBoxBytes + 1024;
  static_assert(kAlloc <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
};

// Walks (group, token tile, weight tile) in increasing tile id; weight tiles vary fastest.  A
// group's rows are split evenly over the fewest tiles of at most TMAX tokens: an MMA's time
// follows its tokens while the expansion of the weights costs the same for every tile, so no tile
// should be a sliver.
template <int TMAX, int GRAIN>
struct Int4Cursor {
  int g = 0, rows = 0, off = 0, width = 0;
  GroupWindow<true> win;
  static __device__ __forceinline__ int tile_width(int rows) {
    const int tiles = (rows + TMAX - 1) / TMAX;
    return tiles ? ((rows + tiles - 1) / tiles + GRAIN - 1) / GRAIN * GRAIN : GRAIN;
  }
  __device__ __forceinline__ bool seek(const Int4Params& p, int ntiles, int t, int& tt, int& nt) {
    int first;
    if (!win.find(p.l, t,
                  [&](int gi, int& r, int& o) { load_group(p.group_rows, p.group_offsets, p.rows_total, gi, r, o); },
                  [=](int r) { const int w = tile_width(r); return (r + w - 1) / w * ntiles; }, g, rows, off, first))
      return false;
    width = tile_width(rows);
    const int u = t - first;
    tt = u / ntiles;
    nt = u - tt * ntiles;
    return true;
  }
  // tokens of tile tt, and the MMA's N (a multiple of GRAIN)
  __device__ __forceinline__ int tokens(int tt) const { return min(width, rows - tt * width); }
  __device__ __forceinline__ int mma_n(int tt) const { return (tokens(tt) + GRAIN - 1) / GRAIN * GRAIN; }
};

// Eight nibbles of a word -> eight bf16 products with the scale, in K order.  The steps are those of
// CUTLASS's int4 -> bf16 converter (cutlass/numeric_conversion.h, a published trick): the nibble with its
// sign bit flipped is q + 8; put into the mantissa of 128.0 it reads 136 + q, and subtracting 136
// is exact.  One byte permutation brings the two nibbles of a byte (one from the word, one from the
// word shifted right by four) under one mask.
// Written out in PTX so that it stays one shift, four permutations, four LOP3 and eight packed bf16
// operations: left to the compiler, the two constants of the mask cost a second LOP3 each.
__device__ __forceinline__ void expand_8(uint32_t w, uint32_t scale2, uint32_t mask, uint32_t one2, uint32_t* out) {
  asm("{\n"
      " .reg .b32 h, p0, p1, p2, p3, c;\n"
      " shr.u32 h, %4, 4;\n"
      " mov.b32 c, 0xC308C308;\n"                      // -136, -136
      " prmt.b32 p0, %4, h, 0x4400;\n"
      " prmt.b32 p1, %4, h, 0x5511;\n"
      " prmt.b32 p2, %4, h, 0x6622;\n"
      " prmt.b32 p3, %4, h, 0x7733;\n"
      " lop3.b32 p0, p0, %6, 0x43084308, 0x6A;\n"      // (p & mask) ^ 136.0 with the nibble flipped
      " lop3.b32 p1, p1, %6, 0x43084308, 0x6A;\n"
      " lop3.b32 p2, p2, %6, 0x43084308, 0x6A;\n"
      " lop3.b32 p3, p3, %6, 0x43084308, 0x6A;\n"
      " fma.rn.bf16x2 p0, p0, %7, c;\n"
      " fma.rn.bf16x2 p1, p1, %7, c;\n"
      " fma.rn.bf16x2 p2, p2, %7, c;\n"
      " fma.rn.bf16x2 p3, p3, %7, c;\n"
      " mul.rn.bf16x2 %0, p0, %5;\n"
      " mul.rn.bf16x2 %1, p1, %5;\n"
      " mul.rn.bf16x2 %2, p2, %5;\n"
      " mul.rn.bf16x2 %3, p3, %5;\n"
      "}\n"
      : "=r"(out[0]), "=r"(out[1]), "=r"(out[2]), "=r"(out[3])
      : "r"(w), "r"(scale2), "r"(mask), "r"(one2));
}

template <bool PAIR, int TMAX, int PSTAGES, int CONV, int EPI>
__device__ __forceinline__ void gemm_int4_body(const CUtensorMap& tmap_w, const CUtensorMap& tmap_t64,
                                               const CUtensorMap& tmap_t16, const Int4Params& p) {
  using L = Int4Smem<PAIR, TMAX, PSTAGES, CONV, EPI>;
  constexpr int S = L::kStages;
  constexpr int kCtas = PAIR ? 2 : 1;
  constexpr int kGrain = PAIR ? 32 : 16;
  constexpr int kTileRows = 128 * kCtas;                   // weight rows of a tile
  constexpr bool kTwoAcc = TMAX <= 128;                    // two accumulators of 128 columns fit
  constexpr int kACol0 = 256;                              // expanded weights: S x 64 columns
  constexpr int kPhases = CONV / 4;                        // converter warps per lane quadrant
  static_assert(kPhases == 2 || kPhases == 4, "a packed stage is read by two warps of each quadrant");
  constexpr int kMmaWarp = CONV + EPI, kWeightWarp = kMmaWarp + 1, kTokenWarp = kMmaWarp + 2;
  using Cursor = Int4Cursor<TMAX, kGrain>;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const uint32_t bar_full = sbase;                         // S x 8 (the leader's are used)
  const uint32_t bar_empty = bar_full + 8 * S;             // S x 8
  const uint32_t bar_packed = bar_empty + 8 * S;           // PSTAGES x 8: packed weights landed
  const uint32_t bar_unpacked = bar_packed + 8 * PSTAGES;  // PSTAGES x 8: and have been read
  const uint32_t bar_acc_full = bar_unpacked + 8 * PSTAGES;   // 2 x 8
  const uint32_t bar_acc_empty = bar_acc_full + 16;        // 2 x 8 (the leader's are used)
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sgen + 512);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(sgen + 516);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const bool leader = rank == 0;
  const int unit = blockIdx.x / kCtas, units = gridDim.x / kCtas;
  const int ntiles = p.n / kTileRows;
  const int kunits = (p.kblocks + 1) >> 1;                 // 128-K stages of a tile; the last may hold 64 K
  auto arrive_leader = [](uint32_t bar) {
    if (PAIR) mbar_arrive_cluster(bar & kLeaderMask);
    else mbar_arrive(bar);
  };
  auto commit = [](uint32_t bar) {
    if (PAIR) tc_commit_pair(bar, 3);
    else tc_commit(bar);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar_full + 8 * s, 1 + 4 * kCtas);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < PSTAGES; ++s) {
      mbar_init(bar_packed + 8 * s, 1);
      mbar_init(bar_unpacked + 8 * s, 8);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, EPI * kCtas);
    }
    *abort_flag = 0u;
    fence_barrier_init();
  }
  if (warp == kWeightWarp && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_t64);
    tma_prefetch_desc(&tmap_t16);
  }
  if (warp == 0) {
    if (PAIR) {
      tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  grid_dependency_wait();
  grid_launch_dependents();

  if (warp == kWeightWarp) {
    // ------------------------------ packed weights ------------------------------
    Cursor cur;
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int t = unit; ok; t += units) {
      int tt, nt;
      if (!cur.seek(p, ntiles, t, tt, nt)) break;
      const int row0 = cur.g * p.n + nt * kTileRows + (int)rank * 128;
      for (int kb = 0; kb < p.kblocks; kb += 4) {
        ok = warp_wait_relaxed(bar_unpacked + 8 * s, ph ^ 1u, abort_flag, p.status, 1, 100);
        if (!ok) break;
        if (elect_one()) {
          mbar_arrive_expect_tx(bar_packed + 8 * s, L::kPacked);
          tma_load_2d(sbase + L::kOffPacked + s * L::kPacked, &tmap_w, bar_packed + 8 * s, kb * 32, row0);
        }
        __syncwarp();
        if (++s == PSTAGES) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == kTokenWarp) {
    // ------------------------------ tokens --------------------------------------
    Cursor cur;
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int t = unit; ok; t += units) {
      int tt, nt;
      if (!cur.seek(p, ntiles, t, tt, nt)) break;
      const int share = cur.mma_n(tt) / kCtas;              // rows this CTA loads, a multiple of 16
      const int row0 = cur.off + tt * cur.width + (int)rank * share;
      const int wide = share >> 6;                          // 64-row boxes, then 16-row boxes
      for (int u = 0; u < kunits; ++u) {
        ok = warp_wait_relaxed(bar_empty + 8 * s, ph ^ 1u, abort_flag, p.status, 2, 60);
        if (!ok) break;
        const uint32_t full = bar_full + 8 * s;
        const int halves = min(2, p.kblocks - 2 * u);
        if (elect_one()) {
          if (leader) mbar_arrive_expect_tx(full, (uint32_t)(halves * share * 128 * kCtas));
          for (int h = 0; h < halves; ++h) {
            const uint32_t dst = sbase + L::kOffTok + s * L::kTok + h * L::kTokHalf;
            const int x = (2 * u + h) * 128;
            for (int i = 0; i < wide; ++i) {
              if (PAIR) tma_load_2d_pair(dst + i * 8192, &tmap_t64, full, x, row0 + 64 * i);
              else tma_load_2d(dst + i * 8192, &tmap_t64, full, x, row0 + 64 * i);
            }
            for (int r = wide * 64; r < share; r += 16) {
              if (PAIR) tma_load_2d_pair(dst + r * 128, &tmap_t16, full, x, row0 + r);
              else tma_load_2d(dst + r * 128, &tmap_t16, full, x, row0 + r);
            }
          }
        }
        __syncwarp();
        if (++s == S) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------ MMA issuer (leader only) --------------------
    if (leader) {
      Cursor cur;
      uint32_t s = 0, ph = 0;
      int tl = 0;
      bool ok = true;
      const uint64_t tdesc0 = operand_desc_sw128(sbase + L::kOffTok);
      for (int t = unit; ok; t += units, ++tl) {
        int tt, nt;
        if (!cur.seek(p, ntiles, t, tt, nt)) break;
        // fp32 accumulate, bf16 operands, both K-major
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(cur.mma_n(tt) >> 3) << 17) |
                               (uint32_t(kTileRows >> 4) << 24);
        const int buf = kTwoAcc ? (tl & 1) : 0;
        const uint32_t use = kTwoAcc ? (uint32_t)(tl >> 1) : (uint32_t)tl;
        ok = warp_wait(bar_acc_empty + 8 * buf, (use & 1u) ^ 1u, abort_flag, p.status, 3);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + buf * 128;
        for (int u = 0; u < kunits; ++u) {
          ok = warp_wait(bar_full + 8 * s, ph, abort_flag, p.status, 4);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t tdesc = tdesc0 + s * (L::kTok >> 4);
          const uint32_t a = tmem_base + kACol0 + s * 64;
          const bool two = 2 * u + 1 < p.kblocks;
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {   // K = 16: eight TMEM columns, 32 bytes of a token row
              if (j == 4 && !two) break;
              const uint64_t b = tdesc + (j >> 2) * (L::kTokHalf >> 4) + 2 * (j & 3);
              if (PAIR) tc_mma_f16_ts_pair(acc, a + 8 * j, b, idesc, (u | j) ? 1u : 0u);
              else tc_mma_f16_ts(acc, a + 8 * j, b, idesc, (u | j) ? 1u : 0u);
            }
            commit(bar_empty + 8 * s);
          }
          __syncwarp();
          if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (ok && elect_one()) commit(bar_acc_full + 8 * buf);
        __syncwarp();
      }
    }
  } else if (warp < CONV) {
    // ------------------------------ converters (both CTAs) ----------------------
    // The warps of a quadrant take the 128-K stages in turn.  A packed stage holds two of them; a
    // tile with an odd number leaves a place empty, which counts as a turn (somebody has to say that
    // the packed stage has been read) but takes no ring stage.
    Cursor cur;
    const int quad = warp & 3, phase = warp >> 2;
    const int row = quad * 32 + lane;                       // of this CTA's 128 weight rows
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    const int groups_k = p.kblocks / p.group_blocks;
    const int step_groups = 2 * kPhases / p.group_blocks, step_rem = 2 * kPhases % p.group_blocks;
    const bool shared_scale = p.group_blocks % 2 == 0, whole_steps = step_rem == 0;
    const int places = (kunits + 1) & ~1;
    uint32_t mask, one2;                                    // kept in registers
    asm volatile("mov.b32 %0, 0x000F000F;" : "=r"(mask));
    asm volatile("mov.b32 %0, 0x3F803F80;" : "=r"(one2));   // 1.0, 1.0
    const uint32_t src0 = sbase + L::kOffPacked + row * 128;
    const uint32_t swz = (uint32_t)(row & 7) << 4;
    uint32_t turn = phase;        // this warp's next place, counted from the start of the tile
    uint32_t stage0 = 0;          // ring stages used by earlier tiles
    uint32_t ps = phase >> 1, pph = 0;   // packed stage of the next turn: kPhases / 2 on at every turn
    bool ok = true;
    for (int t = unit; ok; t += units) {
      int tt, nt;
      if (!cur.seek(p, ntiles, t, tt, nt)) break;
      const __nv_bfloat16* srow = p.scales + ((size_t)cur.g * p.n + nt * kTileRows + (int)rank * 128 + row) * groups_k;
      // Scales of this warp's two 64-K blocks (one, when a scale group covers both), requested one
      // turn ahead: volatile, so that the load stays where it is and is not moved down to its use.
      // Past the tile's last block the pointer stays where it is and the value is not used.
      int grp[2], rem[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        grp[i] = (int)(2 * turn + i) / p.group_blocks;
        rem[i] = (int)(2 * turn + i) % p.group_blocks;
      }
      uint16_t sc[2], sc_next[2] = {0, 0};
      auto load_scales = [&](uint16_t (&v)[2]) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i == 1 && shared_scale) break;
          if (grp[i] < groups_k) asm volatile("ld.global.u16 %0, [%1];" : "=h"(v[i]) : "l"(srow + grp[i]));
          grp[i] += step_groups;
          if (!whole_steps) {
            rem[i] += step_rem;
            if (rem[i] >= p.group_blocks) {
              rem[i] -= p.group_blocks;
              ++grp[i];
            }
          }
        }
      };
      load_scales(sc_next);
      for (; turn < (uint32_t)places; turn += kPhases) {
#pragma unroll
        for (int i = 0; i < 2; ++i) sc[i] = sc_next[shared_scale ? 0 : i];
        load_scales(sc_next);
        ok = warp_wait(bar_packed + 8 * ps, pph, abort_flag, p.status, 5);
        if (!ok) break;
        const uint32_t read = bar_unpacked + 8 * ps, src = src0 + ps * L::kPacked;
        ps += kPhases / 2;
        if (ps >= PSTAGES) { ps -= PSTAGES; pph ^= 1u; }
        if (turn >= (uint32_t)kunits) {                     // the empty place
          if (lane == 0) mbar_arrive(read);
          continue;
        }
        uint4 q[4];                                         // 16 bytes = 32 weights each
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(q[c].x), "=r"(q[c].y), "=r"(q[c].z), "=r"(q[c].w)
                       : "r"(src + (((phase & 1) * 64 + c * 16) ^ swz)) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(read);
        const uint32_t st = stage0 + turn;
        const uint32_t s = st % S;
        const uint32_t a = tmem_base + lane_base + kACol0 + s * 64;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t s2 = (uint32_t)sc[c >> 1] * 0x00010001u;
          uint32_t v[16];
          expand_8(q[c].x, s2, mask, one2, v);
          expand_8(q[c].y, s2, mask, one2, v + 4);
          expand_8(q[c].z, s2, mask, one2, v + 8);
          expand_8(q[c].w, s2, mask, one2, v + 12);
          if (c == 0) {
            ok = warp_wait(bar_empty + 8 * s, ((st / S) & 1u) ^ 1u, abort_flag, p.status, 6);
            if (!ok) break;
            tc_fence_after_sync();
          }
          tmem_st_32x32b_x16(a + c * 16, v);   // (a second half beyond K is written and not multiplied)
        }
        if (!ok) break;
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) arrive_leader(bar_full + 8 * s);
      }
      if (!ok) break;
      turn -= places;
      stage0 += kunits;
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ------------------------
    Cursor cur;
    int tl = 0;
    const int quad = warp & 3, half = (warp - CONV) >> 2;
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    const uint32_t box = sbase + L::kOffC + (warp - CONV) * L::kBoxBytes;
    constexpr int kHalves = EPI / 4;                        // warps of a quadrant share the tokens
    constexpr int kChunks = (TMAX + 32 * kHalves - 1) / (32 * kHalves);   // 32-token chunks of a warp
    for (int t = unit;; t += units, ++tl) {
      int tt, nt;
      if (!cur.seek(p, ntiles, t, tt, nt)) break;
      const int tn = cur.tokens(tt);
      const int buf = kTwoAcc ? (tl & 1) : 0;
      const uint32_t use = kTwoAcc ? (uint32_t)(tl >> 1) : (uint32_t)tl;
      const float alpha = p.alpha ? ld_ordered(p.alpha + cur.g) : 1.0f;   // arrives during the main loop
      if (!warp_wait_relaxed(bar_acc_full + 8 * buf, use & 1u, abort_flag, p.status, 7, 400)) break;
      tc_fence_after_sync();
      const int nchunks = (tn + 31) >> 5;
      // the accumulator goes back before anything is stored: 32 tokens of this lane's column at a
      // time, scaled and rounded, two tokens per register
      uint32_t pk[kChunks][16];
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
        if (kHalves * i + half >= nchunks) break;
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem_base + lane_base + buf * 128 + (kHalves * i + half) * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * e]) * alpha, __uint_as_float(v[2 * e + 1]) * alpha);
          pk[i][e] = *reinterpret_cast<const uint32_t*>(&h);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_leader(bar_acc_empty + 8 * buf);
      const int col0 = nt * kTileRows + (int)rank * 128 + quad * 32;
      const size_t row0 = (size_t)cur.off + (size_t)tt * cur.width;
      const int piece = lane & 3;
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
        const int ci = kHalves * i + half;
        if (ci >= nchunks) break;
        __syncwarp();   // the previous chunk has been read out of the box
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(box + (2 * e) * L::kBoxPitch + lane * 4), "r"(pk[i][e] << 16) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(box + (2 * e + 1) * L::kBoxPitch + lane * 4), "r"(pk[i][e] & 0xffff0000u) : "memory");
        }
        __syncwarp();
        // four lanes take a token's 32 columns, eight each: 64 bytes, two full sectors
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int tl_ = r * 8 + (lane >> 2);
          uint32_t f[8];
#pragma unroll
          for (int h = 0; h < 2; ++h)
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(f[4 * h]), "=r"(f[4 * h + 1]), "=r"(f[4 * h + 2]), "=r"(f[4 * h + 3])
                         : "r"(box + tl_ * L::kBoxPitch + piece * 32 + h * 16) : "memory");
          const int tok = ci * 32 + tl_;
          if (tok < tn) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) w[h] = __byte_perm(f[2 * h], f[2 * h + 1], 0x7632);   // upper halves
            *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + ((row0 + tok) * (size_t)p.n + col0) * 2 + piece * 16) =
                make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // a wait gave up somewhere: give loads still in flight time to land before the shared memory
    // they target is released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (PAIR) cluster_sync();
  if (warp == 0) {
    tc_fence_after_sync();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

template <int TMAX, int PSTAGES, int CONV, int EPI>
__global__ void __launch_bounds__(Int4Smem<false, TMAX, PSTAGES, CONV, EPI>::kThreads, 1)
gemm_int4_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_t64,
                 const __grid_constant__ CUtensorMap tmap_t16, const Int4Params p) {
  gemm_int4_body<false, TMAX, PSTAGES, CONV, EPI>(tmap_w, tmap_t64, tmap_t16, p);
}
template <int TMAX, int PSTAGES, int CONV, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Int4Smem<true, TMAX, PSTAGES, CONV, EPI>::kThreads, 1)
gemm_int4_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_t64,
                      const __grid_constant__ CUtensorMap tmap_t16, const Int4Params p) {
  gemm_int4_body<true, TMAX, PSTAGES, CONV, EPI>(tmap_w, tmap_t64, tmap_t16, p);
}

template <bool PAIR, int TMAX, int PSTAGES, int CONV, int EPI>
static int launch_int4(const CUtensorMap* maps, const Int4Params& p, int max_ctas, cudaStream_t stream) {
  using L = Int4Smem<PAIR, TMAX, PSTAGES, CONV, EPI>;
  constexpr int kCtas = PAIR ? 2 : 1;
  int units = (max_ctas > 0 ? max_ctas : num_sms()) / kCtas;
  if (units <= 0) return fail(MSC_ERR_CUDA, "could not query the SM count");
  const long long tiles = ((long long)(p.rows_total + TMAX - 1) / TMAX + p.l) * (p.n / (128 * kCtas));
  if (units > tiles) units = (int)tiles;
  auto kern = [] {
    if constexpr (PAIR) return gemm_int4_pair_kernel<TMAX, PSTAGES, CONV, EPI>;
    else return gemm_int4_kernel<TMAX, PSTAGES, CONV, EPI>;
  }();
  if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), L::kAlloc)) return rc;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t lc = pdl_launch_config(units * kCtas, L::kThreads, L::kAlloc, stream, attr);
  MSC_CUDA_OK(cudaLaunchKernelEx(&lc, kern, maps[0], maps[1], maps[2], p));
  return MSC_OK;
}

}  // namespace msc

extern "C" int msc_grouped_gemm_bf16_int4_ragged(const void* a, const void* b_q, const void* scales,
                                                 const float* alpha, const int32_t* group_offsets,
                                                 const int32_t* group_rows, void* out, int l,
                                                 int rows_total, int n, int k, int group_size,
                                                 int max_ctas, void* stream) {
  using namespace msc;
  if (!a || !b_q || !scales || !out || !group_offsets || !group_rows)
    return fail(MSC_ERR_BAD_ARG, "NULL pointer");
  if (l <= 0 || rows_total <= 0 || n <= 0 || k <= 0) return fail(MSC_ERR_BAD_ARG, "sizes must be positive");
  if (n % 256) return fail(MSC_ERR_BAD_ARG, "n=%d must be a multiple of 256", n);
  if (k % 64) return fail(MSC_ERR_BAD_ARG, "k=%d must be a multiple of 64", k);
  if (group_size <= 0 || group_size % 64 || k % group_size)
    return fail(MSC_ERR_UNSUPPORTED,
                "group_size=%d must be a multiple of 64 that divides k (use msc_int4_dequant_bf16 + "
                "msc_grouped_gemm_bf16_ragged otherwise)", group_size);
  if (reinterpret_cast<uintptr_t>(out) % 16) return fail(MSC_ERR_BAD_ARG, "out must be 16-byte aligned");
  Int4Params p = {};
  p.status = status_word();
  if (!p.status) return fail(MSC_ERR_CUDA, "status word unavailable on this device");
  CUtensorMap maps[3];
  int rc = make_tmap_bytes_2d(&maps[0], b_q, (uint64_t)l * n, (uint64_t)k / 2, 128);
  if (rc) return rc;
  rc = make_tmap_bytes_2d(&maps[1], a, (uint64_t)rows_total, (uint64_t)k * 2, 64);
  if (rc) return rc;
  rc = make_tmap_bytes_2d(&maps[2], a, (uint64_t)rows_total, (uint64_t)k * 2, 16);
  if (rc) return rc;
  p.scales = static_cast<const __nv_bfloat16*>(scales);
  p.alpha = alpha;
  p.group_rows = group_rows;
  p.group_offsets = group_offsets;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.l = l;
  p.n = n;
  p.rows_total = rows_total;
  p.kblocks = k / 64;
  p.group_blocks = group_size / 64;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Pairs share the tokens between two SMs and take 256 of them per tile: the form for groups of
  // hundreds of rows, where the MMAs set the pace (64 groups of 64 - 512 rows, n = 2048, k = 7168:
  // 417 - 441 us against 609 us with single CTAs).  Single CTAs with 16 converter warps and
  // narrower tiles are ahead where the expansion sets it, groups within one 128-row block (1 - 16
  // rows: 182 against 205 us), and where there are so few tiles that half the pairs would idle.
  const long long avg = rows_total / l;
  const long long pair_tiles = (long long)l * ((avg + 255) / 256) * (n / 256);
  if (avg <= 128 || 4 * pair_tiles <= num_sms()) return launch_int4<false, 128, 4, 16, 4>(maps, p, max_ctas, st);
  return launch_int4<true, 256, 3, 8, 8>(maps, p, max_ctas, st);
}
