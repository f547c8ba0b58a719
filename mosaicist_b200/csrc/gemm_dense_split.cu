// Dense 16-bit GEMM for problems with too few 256-row pair tiles to fill the chip: smaller tiles,
// and the contraction split over the CTAs of a cluster.
//
// One tile of 128 rows per cluster, no persistence.  A cluster is `splits` CTAs, each with its share
// of the K stages; every CTA then puts its fp32 accumulator into its own shared memory (the operand
// ring is free by then), and after one cluster barrier each sums a slice of the tile's rows over
// distributed shared memory, in the order of the splits, rounds once and stores.  No workspace, no
// second launch, the same sum every time.
//
// What bounds such a problem in the persistent kernel (gemm_dense_f16.cu) is the serial chain of
// one tile: 48 stages of 32 KB into each of 40 SMs while 108 idle.  Here the tile and the split are
// chosen so that the stages of a CTA are few and cheap.  bf16, inputs from HBM, back to back, us
// (persistent kernel in brackets): 16 x 1024 x 1024 4.4 (8.2), 64 x 4096 x 4096 10.5 (22.6),
// 512^3 4.1 (6.7), 1024 x 1024 x 8192 21.8 (40.7), 128 x 8192 x 8192 26.2 (41.5; 20.5 at the rate
// of HBM), 777 x 1048 x 3080 18.9 (22.8; its rows start off 128-byte lines, which doubles the
// cost of a stage in the copy engine: 777 x 1024 x 3072 takes 10.5 (18.4)).  CTA pairs with 256-row tiles,
// split the same way, were 1 - 60 % slower than these tiles on all but one of 25 shapes and are not
// built.
#include "gemm_dense.h"

#include <cuda_fp16.h>

namespace msc {

struct DenseSplitParams {
  void* c;
  int* status;
  int m, n, ldc;
  int m_tiles;
  int k_stages;     // ceil(K / 64)
  int splits;
  int a_box_rows;   // rows of A a load brings: 128, less when the matrix has fewer
  int is_bf16;
};

template <int TN>
struct DenseSplitSmem {
  static constexpr int kBoxes = TN / 64;                    // 64-column boxes of B per stage
  static constexpr int kA = 128 * 128;
  static constexpr int kB = kBoxes * 8192;
  static constexpr int kStages = 196608 / (kA + kB);        // 8 x 24 KB or 6 x 32 KB
  static constexpr int kOffA = 1024;
  static constexpr int kOffB = kOffA + kStages * kA;
  static constexpr int kOffAcc = 1024;                      // over the ring: [128][kPitch] fp32
  static constexpr int kPitch = TN + 4;                     // 16-byte writes of a column of rows: no conflict
  static constexpr int kThreads = 10 * 32;
  static constexpr int kAlloc = 1024 + kStages * (kA + kB) + 1024;
  static_assert(128 * kPitch * 4 <= kStages * (kA + kB), "the accumulator does not fit over the ring");
  static_assert(kAlloc <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
};

template <int TN>
__global__ void __launch_bounds__(DenseSplitSmem<TN>::kThreads, 1)
gemm_dense_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        const DenseSplitParams p) {
  using L = DenseSplitSmem<TN>;
  constexpr int S = L::kStages;
  constexpr int kMmaWarp = 8, kProducerWarp = 9;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sbase = (raw + 1023u) & ~1023u;
  uint8_t* sgen = smem_raw + (sbase - raw);
  const uint32_t bar_full = sbase;                 // S x 8
  const uint32_t bar_empty = bar_full + 8 * S;     // S x 8
  const uint32_t bar_acc = bar_empty + 8 * S;      // 8
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sgen + 512);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(sgen + 516);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int split = (int)cluster_ctarank();
  const int tile = blockIdx.x / p.splits;
  const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
  const int row0 = mt * 128;
  const int kb0 = (int)((long long)p.k_stages * split / p.splits);
  const int kb1 = (int)((long long)p.k_stages * (split + 1) / p.splits);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_acc, 1);
    *abort_flag = 0u;
    fence_barrier_init();
  }
  if (warp == kProducerWarp && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  grid_dependency_wait();
  grid_launch_dependents();

  if (warp == kProducerWarp) {
    uint32_t s = 0, ph = 0;
    const uint32_t a_bytes = (uint32_t)p.a_box_rows * 128u;
    const int col = nt * TN * 2;   // byte column of B
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!warp_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, p.status, 1)) break;
      const uint32_t full = bar_full + 8 * s;
      if (elect_one()) {
        mbar_arrive_expect_tx(full, a_bytes + L::kB);
        const uint32_t a_dst = sbase + L::kOffA + s * L::kA, b_dst = sbase + L::kOffB + s * L::kB;
        tma_load_2d(a_dst, &tmap_a, full, kb * 128, row0);
#pragma unroll
        for (int i = 0; i < L::kBoxes; ++i) tma_load_2d(b_dst + i * 8192, &tmap_b, full, col + i * 128, kb * 64);
      }
      __syncwarp();
      if (++s == S) { s = 0; ph ^= 1u; }
    }
  } else if (warp == kMmaWarp) {
    // fp32 accumulate, A K-major, B MN-major
    const uint32_t idesc = (1u << 4) | (p.is_bf16 ? ((1u << 7) | (1u << 10)) : 0u) | (1u << 16) |
                           (uint32_t(TN >> 3) << 17) | (uint32_t(128 >> 4) << 24);
    const uint64_t adesc0 = operand_desc_sw128(sbase + L::kOffA);
    const uint64_t bdesc0 = operand_desc_mn_sw128(sbase + L::kOffB, 8192u);
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      ok = warp_wait(bar_full + 8 * s, ph, abort_flag, p.status, 3);
      if (!ok) break;
      tc_fence_after_sync();
      const uint64_t adesc = adesc0 + s * (L::kA >> 4), bdesc = bdesc0 + s * (L::kB >> 4);
      if (elect_one()) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t accumulate = (kb > kb0 || j) ? 1u : 0u;
          tc_mma_f16(tmem_base, adesc + 2 * j, bdesc + 128 * j, idesc, accumulate);
        }
        tc_commit(bar_empty + 8 * s);
      }
      __syncwarp();
      if (++s == S) { s = 0; ph ^= 1u; }
    }
    if (ok && elect_one()) tc_commit(bar_acc);
    __syncwarp();
  } else {
    // ------------------------------ accumulator -> shared memory ----------------
    // every load has been consumed and every MMA has completed once bar_acc flips, so the ring's
    // memory is free
    const int quad = warp & 3, slab = warp >> 2;
    if (warp_wait(bar_acc, 0, abort_flag, p.status, 4)) {
      tc_fence_after_sync();
      constexpr int kChunks = TN / 64;   // 32-column chunks per warp
      const uint32_t src = tmem_base + (uint32_t(quad * 32) << 16) + slab * (TN / 2);
      const uint32_t dst = sbase + L::kOffAcc + ((quad * 32 + lane) * L::kPitch + slab * (TN / 2)) * 4;
      uint32_t v[kChunks][32];
#pragma unroll
      for (int c = 0; c < kChunks; ++c) tmem_ld_32x32b_x32(src + c * 32, v[c]);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int q = 0; q < 8; ++q)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (c * 32 + q * 4) * 4),
                       "r"(v[c][4 * q]), "r"(v[c][4 * q + 1]), "r"(v[c][4 * q + 2]), "r"(v[c][4 * q + 3]) : "memory");
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  if (p.splits > 1) cluster_sync();   // the partial sums of the whole cluster are in place
  else __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem_base, TN);
  if (*abort_flag) {
    // a wait gave up: give loads still in flight time to land; what is stored then is reported as
    // wrong through the status word
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }

  // ------------------------------ sum, round, store --------------------------------
  // this CTA's share of the rows that exist, eight columns per thread and step
  const int rows = min(max(p.m - row0, 0), 128);
  const int share = (rows + p.splits - 1) / p.splits;
  const int r_end = min(rows, (split + 1) * share);
  constexpr int kVecs = TN / 8;
  const int u_end = r_end * kVecs;
  constexpr int kAhead = 2;   // steps of a thread whose loads are in flight together
  for (int u0 = split * share * kVecs + (int)threadIdx.x; u0 < u_end; u0 += kAhead * L::kThreads) {
    float acc[kAhead][8];
    uint32_t local[kAhead];
#pragma unroll
    for (int h = 0; h < kAhead; ++h) {
      const int u = min(u0 + h * L::kThreads, u_end - 1);
      const int r = u / kVecs, vc = u - r * kVecs;
      local[h] = sbase + L::kOffAcc + (r * L::kPitch + vc * 8) * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[h][i] = 0.0f;
    }
#pragma unroll 4
    for (int j = 0; j < p.splits; ++j) {
      float f[kAhead][8];
#pragma unroll
      for (int h = 0; h < kAhead; ++h) {
        const uint32_t src = cluster_map_shared(local[h], (uint32_t)j);
        ld_shared_cluster_v4(src, f[h]);
        ld_shared_cluster_v4(src + 16, f[h] + 4);
      }
#pragma unroll
      for (int h = 0; h < kAhead; ++h)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[h][i] = __fadd_rn(acc[h][i], f[h][i]);
    }
#pragma unroll
    for (int h = 0; h < kAhead; ++h) {
      const int u = u0 + h * L::kThreads;
      const int r = u / kVecs, col = nt * TN + (u - r * kVecs) * 8;
      if (u >= u_end || col >= p.n) continue;               // n is a multiple of 8
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (p.is_bf16) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(acc[h][2 * i], acc[h][2 * i + 1]);
          w[i] = *reinterpret_cast<const uint32_t*>(&pr);
        } else {
          const __half2 pr = __floats2half2_rn(acc[h][2 * i], acc[h][2 * i + 1]);
          w[i] = *reinterpret_cast<const uint32_t*>(&pr);
        }
      }
      *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.c) + (size_t)(row0 + r) * p.ldc + col) =
          make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  __syncwarp();
  if (p.splits > 1) cluster_sync();   // nobody leaves while its sums may still be read
}

template <int TN>
static int launch_split(const CUtensorMap& ta, const CUtensorMap& tb, const DenseSplitParams& p, int ctas,
                        cudaStream_t stream) {
  using L = DenseSplitSmem<TN>;
  auto kern = gemm_dense_split_kernel<TN>;
  if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(kern), L::kAlloc)) return rc;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t lc = pdl_launch_config(ctas, L::kThreads, L::kAlloc, stream, attr);
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.splits;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  lc.numAttrs = 2;
  MSC_CUDA_OK(cudaLaunchKernelEx(&lc, kern, ta, tb, p));
  return MSC_OK;
}

int launch_dense_split(const DenseForm& form, const void* a, const void* b, void* c, int m, int n, int k, int lda,
                       int ldb, int ldc, int is_bf16, int* status, cudaStream_t stream) {
  const int k_stages = (k + 63) / 64;
  if (form.splits < 1 || form.splits > k_stages || form.splits > 8)
    return fail(MSC_ERR_BAD_ARG, "splits=%d does not fit a cluster or %d stages of K", form.splits, k_stages);
  if (form.tile_n != 64 && form.tile_n != 128) return fail(MSC_ERR_BAD_ARG, "tile_n=%d must be 64 or 128", form.tile_n);
  DenseSplitParams p;
  p.a_box_rows = m >= 128 ? 128 : (m + 7) / 8 * 8;
  CUtensorMap ta, tb;
  int rc = make_tmap_pitched_2d(&ta, a, (uint64_t)m, (uint64_t)k * 2, (uint64_t)lda * 2, (uint32_t)p.a_box_rows);
  if (rc) return rc;
  rc = make_tmap_pitched_2d(&tb, b, (uint64_t)k, (uint64_t)n * 2, (uint64_t)ldb * 2, 64);
  if (rc) return rc;
  p.c = c;
  p.status = status;
  p.m = m; p.n = n; p.ldc = ldc;
  p.m_tiles = (m + 127) / 128;
  p.k_stages = k_stages;
  p.splits = form.splits;
  p.is_bf16 = is_bf16;
  const long long ctas = (long long)p.m_tiles * ((n + form.tile_n - 1) / form.tile_n) * form.splits;
  if (ctas > 0x7fffffffLL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
  return form.tile_n == 64 ? launch_split<64>(ta, tb, p, (int)ctas, stream) : launch_split<128>(ta, tb, p, (int)ctas, stream);
}

// The form that a model of the time, fitted to 25 shapes on a B200 (m, n, k from 1 to 8192, both
// kernels), puts lowest: a fixed part plus K stages of a CTA times the price of a stage.  A stage
// costs what the copy engine takes for its bytes, about twice that for an operand whose rows are
// not whole 128-byte lines apart.  Only launches of one wave are considered: the tiles of a second
// one start over (4096 x 512 x 256: 4.9 us with 128 CTAs, 7.5 us with 256).
//
// Whether the contraction is split depends on m and k alone: every form without a split adds up in
// the same order, so a column shard of a product has the bits of the whole product, and has to keep
// them.  Two splits from K = 4096 on for matrices of up to 128 rows, whatever n is: 64 x 4096 x 4096
// 12.5 -> 10.5 us, 128 x 8192 x 8192 26.6 -> 26.2 us; from that K on many waves of half tiles are
// still no slower than the persistent kernel, which loads and multiplies 256 rows.
DenseForm pick_dense_form(int m, int n, int k, int lda, int ldb) {
  const long long stages = (k + 63) / 64;
  const long long sms = num_sms();
  if (sms <= 0) return DenseForm{0, 0};
  const bool split = m <= 128 && k >= 4096;
  const bool a_off = (long long)lda * 2 % 128, b_off = (long long)ldb * 2 % 128;
  // ns per stage, and what an operand off its lines adds
  auto stage_ns = [&](int base, int a_extra, int b_extra) { return base + (a_off ? a_extra : 0) + (b_off ? b_extra : 0); };
  const long long tiles256 = (long long)((m + 255) / 256) * ((n + 255) / 256);
  DenseForm best{0, 0};
  long long best_ns = 3800 + (tiles256 + sms / 2 - 1) / (sms / 2) * stages * stage_ns(350, 45, 45);
  if (split) best_ns = 0x7fffffffffffffffLL;
  const int rows = m < 128 ? m : 128;
  for (int wide = 1; wide <= 2; ++wide) {
    const long long ctas = (long long)((m + 127) / 128) * ((n + 64 * wide - 1) / (64 * wide)) * (split ? 2 : 1);
    const long long waves = (ctas + sms - 1) / sms;
    if (waves > 1 && !split) continue;
    const long long per_cta = split ? (stages + 1) / 2 : stages;
    // the accumulator goes through shared memory, with two splits twice
    const long long ns = 1900 + 800 * wide * rows / 128 + (split ? 800 + 1000 * wide * rows / 128 : 0) +
                         per_cta * (wide == 1 ? stage_ns(155, 115, 60) : stage_ns(200, 85, 85));
    if (waves * ns < best_ns) {
      best_ns = waves * ns;
      best = DenseForm{64 * wide, split ? 2 : 1};
    }
  }
  return best;
}

}  // namespace msc
