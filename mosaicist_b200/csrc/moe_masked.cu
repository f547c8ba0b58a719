// The masked MoE layer as one call (moe_masked, experiments/flashinfer-megamoe-sm100a/moe.py:47-79):
// three launches back to back on the stream, each with its set-up under the tail of the one before
// it.  Everything that used to be a launch of its own around them is folded in: the two-level
// scales into the GEMMs' epilogues, the zeros of rows that are not live into the quantiser, and
// the intermediates are slices of one workspace that is never cleared (scale bytes of rows that
// are not live only reach accumulator rows that are not stored).
#include "gemm_common.cuh"

namespace msc {

struct MaskedLayout {
  size_t a_q, a_sf, d_q, d_sf, gateup, total;
};

static MaskedLayout masked_layout(long long l, long long m, long long k, long long n) {
  auto up = [](long long b) { return (size_t)((b + 255) / 256 * 256); };
  const bool fused = 2 * n % 256 == 0;
  MaskedLayout w;
  w.a_q = 0;
  w.a_sf = w.a_q + up(l * m * k / 2);
  w.d_q = w.a_sf + up(l * m * k / 16);
  w.d_sf = w.d_q + up(l * m * n / 2);
  w.gateup = w.d_sf + up(l * m * n / 16);
  w.total = w.gateup + (fused ? 0 : up(l * m * n * 4));
  return w;
}

}  // namespace msc

extern "C" {

size_t msc_moe_masked_workspace(int l, int m, int k, int n) {
  if (l <= 0 || m <= 0 || k <= 0 || n <= 0) return 0;
  return msc::masked_layout(l, m, k, n).total;
}

int msc_moe_masked(const void* hidden, const void* w1_q, const void* w1_sf, const float* w1_gs,
                   const float* w1_alpha, const void* w2_q, const void* w2_sf, const float* w2_gs,
                   const float* w2_alpha, const int32_t* masked_m, const float* input_gs,
                   const float* a2_gs, const float* g1_alpha, const float* g2_alpha, void* workspace,
                   size_t workspace_bytes, void* out, int zero_rest, int l, int m, int k, int n,
                   void* stream) {
  using namespace msc;
  if (!hidden || !w1_q || !w1_sf || !w2_q || !w2_sf || !masked_m || !input_gs || !a2_gs || !workspace || !out)
    return fail(MSC_ERR_BAD_ARG, "NULL pointer");
  if (!g1_alpha != !g2_alpha || (!g1_alpha && (!w1_gs || !w1_alpha || !w2_gs || !w2_alpha)))
    return fail(MSC_ERR_BAD_ARG, "either both folded alphas or all global scales and alphas are needed");
  if (l <= 0 || m <= 0 || k <= 0 || n <= 0) return fail(MSC_ERR_BAD_ARG, "sizes must be positive");
  if (m % 128) return fail(MSC_ERR_BAD_ARG, "m=%d must be a multiple of 128", m);
  if (n % 64 || k % 128) return fail(MSC_ERR_BAD_ARG, "n=%d must be a multiple of 64 and k=%d of 128", n, k);
  if (reinterpret_cast<uintptr_t>(workspace) % 256) return fail(MSC_ERR_BAD_ARG, "workspace must be 256-byte aligned");
  const MaskedLayout w = masked_layout(l, m, k, n);
  if (workspace_bytes < w.total) return fail(MSC_ERR_BAD_ARG, "the workspace needs %zu bytes", w.total);
  if ((long long)l * m > 0x7fffff00LL) return fail(MSC_ERR_UNSUPPORTED, "problem too large for one launch");
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  const int rows = l * m;
  const float* gs1a = g1_alpha ? nullptr : input_gs;
  const float* gs2a = g1_alpha ? nullptr : a2_gs;
  int rc = quantize_nvfp4_rows(hidden, 0, input_gs, nullptr, masked_m, ws + w.a_q, ws + w.a_sf, 1, l, rows, m, k, 0,
                               zero_rest ? out : nullptr, stream);
  if (rc) return rc;
  if (2 * n % 256 == 0) {
    int* status = status_word();
    if (!status) return fail(MSC_ERR_CUDA, "status word unavailable on this device");
    GemmParams p = {};
    p.sfa = ws + w.a_sf;
    p.sfb = static_cast<const uint8_t*>(w1_sf);
    p.alpha = g1_alpha ? g1_alpha : w1_alpha;
    p.alpha_gs_a = gs1a;
    p.alpha_gs_b = w1_gs;
    p.group_rows = masked_m;
    p.status = status;
    p.l = l;
    p.m_stride = m;
    p.rows_total = rows;
    p.n = 2 * n;
    p.k_stages = (k / 2 + 127) / 128;
    p.sf_chunks = k / 64;
    p.out_q = ws + w.d_q;
    p.out_sf = ws + w.d_sf;
    p.out_gs = a2_gs;
#ifdef MSC_DEBUG
    p.trace = g_trace;
    p.debug_flags = g_debug_flags;
#endif
    rc = launch_pair_gemm(KIND_NVFP4, ws + w.a_q, w1_q, rows, k / 2, p, 0, 0, static_cast<cudaStream_t>(stream), false);
  } else {
    rc = grouped_gemm(KIND_NVFP4, ws + w.a_q, ws + w.a_sf, w1_q, w1_sf, g1_alpha ? g1_alpha : w1_alpha, nullptr, masked_m,
                      nullptr, ws + w.gateup, l, rows, m, 2 * n, k, nullptr, stream, gs1a, w1_gs);
    if (rc) return rc;
    rc = quantize_nvfp4_rows(ws + w.gateup, 0, a2_gs, nullptr, masked_m, ws + w.d_q, ws + w.d_sf, 1, l, rows, m, n, 1,
                             nullptr, stream);
  }
  if (rc) return rc;
  return grouped_gemm(KIND_NVFP4, ws + w.d_q, ws + w.d_sf, w2_q, w2_sf, g1_alpha ? g2_alpha : w2_alpha, nullptr, masked_m,
                      nullptr, out, l, rows, m, k, n, nullptr, stream, gs2a, w2_gs);
}

}  // extern "C"
