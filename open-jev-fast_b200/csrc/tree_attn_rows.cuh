// What the two tcgen05 tree-attention kernels share about a query row: its key ranges as bit masks, and its result where the tiled
// product must not be trusted.
#pragma once
#include "gemm_common.cuh"

namespace ojb {
namespace {

// bits of keys [32 * w, 32 * w + 32) that fall in [lo, hi)
__device__ __forceinline__ uint32_t range_bits(int lo, int hi, int w) {
  const int a = max(lo - w * 32, 0), b = min(hi - w * 32, 32);
  if (a >= b) return 0u;
  return (b == 32 ? 0xffffffffu : ((1u << b) - 1u)) & ~((1u << a) - 1u);
}

// 128 dims (from d0) of O / l of one query row over the keys it sees and no others, by one warp; -> four dims from d0 + 4 * lane.
// The product O += P V takes whole key blocks, with P = 0 for keys a row does not see, and 0 times an infinity or a not-a-number is
// a not-a-number: V of one token would reach rows that do not see it (siblings, other requests of a packed forward). The kernels
// call this for rows with a finite sum of P whose O is not finite. Everything else was finite, so the time (about a tenth
// of a microsecond per key) counts only where such a V occurs; keys whose own scores are not finite have left l not finite.
__device__ __forceinline__ float4 row_over_its_keys(const bf16_t* q, const bf16_t* kt, const bf16_t* vt_t, int N, int d0, int lo0, int hi0,
                                                    int lo1, int hi1, int lo2, int hi2, float scale_log2e, float m_log2e, float inv_l) {
  const int lane = threadIdx.x & 31;
  float qf[8], acc[4] = {0.f, 0.f, 0.f, 0.f};
  unpack8(*reinterpret_cast<const uint4*>(q + lane * 8), qf);
  const bf16_t* v = vt_t + static_cast<int64_t>(d0 + 4 * lane) * N;
  hi0 = min(hi0, N); hi1 = min(hi1, N); hi2 = min(hi2, N);
  const int words = (max(hi0, max(hi1, hi2)) + 31) >> 5;
#pragma unroll 1
  for (int w = 0; w < words; ++w) {
    uint32_t bits = range_bits(lo0, hi0, w) | range_bits(lo1, hi1, w) | range_bits(lo2, hi2, w);
#pragma unroll 1
    for (; bits != 0u; bits &= bits - 1u) {
      const int key = w * 32 + __ffs(bits) - 1;
      float kf[8], s = 0.f;
      unpack8(*reinterpret_cast<const uint4*>(kt + static_cast<int64_t>(key) * 256 + lane * 8), kf);
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(qf[e], kf[e], s);
      const float p = round_bf(exp2f_fast(fmaf(warp_sum(s), scale_log2e, -m_log2e)));
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = fmaf(p, bf2f(v[static_cast<int64_t>(e) * N + key]), acc[e]);
    }
    bool done = true;      // (nothing brings a not-a-number back)
#pragma unroll
    for (int e = 0; e < 4; ++e) done = done && acc[e] != acc[e];
    if (__all_sync(0xffffffffu, done)) break;
  }
  return make_float4(acc[0] * inv_l, acc[1] * inv_l, acc[2] * inv_l, acc[3] * inv_l);
}

}  // namespace
}  // namespace ojb
