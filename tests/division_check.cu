// Device side of test_division_gpu.py: counts the operands for which the quantisers' quotients differ
// from __fdiv_rn.  Every loop is over a fixed number of operands; nothing is indexed by data.
#include "../mosaicist_b200/csrc/quantize_common.cuh"

using namespace msc;

constexpr int kSignificands = 1 << 23;
__device__ unsigned long long g_bad[3];
__device__ unsigned long long g_seen[3];

__device__ void add(int which, unsigned long long bad, unsigned long long seen) {
  atomicAdd(&g_bad[which], bad);
  atomicAdd(&g_seen[which], seen);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// amax / 6: all significands of one exponent (0: subnormals)
__global__ void check_six(int exponent) {
  unsigned long long bad = 0, seen = 0;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < kSignificands; m += gridDim.x * blockDim.x) {
    const float a = __uint_as_float(((unsigned)exponent << 23) | (unsigned)m);
    bad += !same(amax_over_6(a), __fdiv_rn(a, 6.0f));
    ++seen;
  }
  add(0, bad, seen);
}

// sf / gs: every e4m3 scale by all significands of one exponent of gs
__global__ void check_step(int exponent) {
  unsigned long long bad = 0, seen = 0;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < kSignificands; m += gridDim.x * blockDim.x) {
    const float gs = __uint_as_float(((unsigned)exponent << 23) | (unsigned)m);
    for (int b = 0; b <= 0x7e; ++b) {
      const float sf = e4m3_to_float((uint8_t)b);
      bad += !same(scale_step(sf, gs), __fdiv_rn(sf, gs));
      ++seen;
    }
  }
  add(1, bad, seen);
}

// e2m1 of x / step: all significands of one exponent of the step, x within eight ulp of every rounding
// boundary of e2m1 times the step, both signs, through pack_block
__global__ void check_values(int exponent) {
  unsigned long long bad = 0, seen = 0;
  const float edge[8] = {0.25f, 0.75f, 1.25f, 1.75f, 2.5f, 3.5f, 5.0f, 6.0f};
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < kSignificands; m += gridDim.x * blockDim.x) {
    const float step = __uint_as_float(((unsigned)exponent << 23) | (unsigned)m);
    const float rcp = __frcp_rn(step);
    for (int e = 0; e < 8; ++e) {
      const unsigned mid = __float_as_uint(__fmul_rn(edge[e], step));
      float v[16];
      for (int i = 0; i < 16; ++i) {
        const float x = __uint_as_float(mid + (unsigned)i - 8u);
        v[i] = (i & 1) ? -x : x;
      }
      uint32_t w[2], want[2] = {0, 0};
      pack_block<false>(v, step, rcp, w);
      for (int i = 0; i < 16; i += 2) {
        const float2 q = make_float2(__fdiv_rn(v[i], step), __fdiv_rn(v[i + 1], step));
        want[i >> 3] |= (uint32_t)__nv_cvt_float2_to_fp4x2(q, __NV_E2M1, cudaRoundNearest) << (8 * ((i & 7) >> 1));
      }
      for (int h = 0; h < 2; ++h)
        for (int n = 0; n < 8; ++n) bad += ((w[h] ^ want[h]) >> (4 * n) & 15u) != 0;
      seen += 16;
    }
  }
  add(2, bad, seen);
}

extern "C" int division_check(int which, int exponent, unsigned long long* bad, unsigned long long* seen) {
  if (which < 0 || which > 2 || exponent < 0 || exponent > 254) return -1;
  unsigned long long zero[3] = {0, 0, 0}, out[3];
  if (cudaMemcpyToSymbol(g_bad, zero, sizeof zero) != cudaSuccess || cudaMemcpyToSymbol(g_seen, zero, sizeof zero) != cudaSuccess) return -2;
  if (which == 0) check_six<<<592, 256>>>(exponent);
  else if (which == 1) check_step<<<592, 256>>>(exponent);
  else check_values<<<592, 256>>>(exponent);
  if (cudaDeviceSynchronize() != cudaSuccess) return -3;
  if (cudaMemcpyFromSymbol(out, g_bad, sizeof out) != cudaSuccess) return -4;
  *bad = out[which];
  if (cudaMemcpyFromSymbol(out, g_seen, sizeof out) != cudaSuccess) return -4;
  *seen = out[which];
  return 0;
}
