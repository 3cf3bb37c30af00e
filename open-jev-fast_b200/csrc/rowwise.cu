// Row-wise and element-wise kernels of the scoring forward: residual add + RMSNorm (with or without split-K partial sums),
// SwiGLU product, activation tables, sigmoid gate product, visibility bit packing, attention q/k/v preparation.
// All of them are HBM-bound streaming kernels: 16-byte accesses, one pass over the data, rows held in registers.
#include "common.cuh"
#include <cuda_fp8.h>
#include <initializer_list>

namespace ojb {
namespace {

constexpr int kRowThreads = 256;
constexpr int kRowVecs = 4;  // 16-byte vectors per thread held in registers -> H <= 256 * 4 * 8 = 8192

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < kRowThreads / 32) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;  // every warp reduces the same 8 partials in the same order -> identical value in all threads
}

// The same for any number of whole warps (red: 32 floats).
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) red[w] = v;
  __syncthreads();
  return warp_sum(lane < static_cast<int>(blockDim.x >> 5) ? red[lane] : 0.f);
}

// One CTA per row. SPLITS == 0: delta is an optional bf16 row; SPLITS > 0: delta = bf16(sum of SPLITS fp32 partial rows).
template <int SPLITS>
__global__ void __launch_bounds__(kRowThreads)
add_rmsnorm_kernel(const bf16_t* __restrict__ x, const bf16_t* __restrict__ delta, const float* __restrict__ parts,
                   int64_t part_stride, const float* __restrict__ w1, const int32_t* __restrict__ rowmask,
                   bf16_t* __restrict__ h_out, bf16_t* __restrict__ hn_out, int H, float eps) {
  pdl_begin();
  __shared__ float red[kRowThreads / 32];
  const int64_t row = blockIdx.x;
  const int nvec = H >> 3;
  float v[kRowVecs][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < kRowVecs; ++i) {
    const int vi = threadIdx.x + i * kRowThreads;
    if (vi < nvec) {
      const int64_t off = row * H + static_cast<int64_t>(vi) * 8;
      unpack8(ldg_stream(x + off), v[i]);
      if constexpr (SPLITS > 0) {
        float d[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = 0.f;
#pragma unroll
        for (int s = 0; s < SPLITS; ++s) {
          const float* pp = parts + s * part_stride + off;
          const uint4 a = ldg_stream(pp), b = ldg_stream(pp + 4);
          d[0] += __uint_as_float(a.x); d[1] += __uint_as_float(a.y); d[2] += __uint_as_float(a.z); d[3] += __uint_as_float(a.w);
          d[4] += __uint_as_float(b.x); d[5] += __uint_as_float(b.y); d[6] += __uint_as_float(b.z); d[7] += __uint_as_float(b.w);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] = round_bf(v[i][e] + round_bf(d[e]));
        *reinterpret_cast<uint4*>(h_out + off) = pack8(v[i]);
      } else if (delta != nullptr) {
        float d[8];
        unpack8(ldg_stream(delta + off), d);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] = round_bf(v[i][e] + d[e]);
        *reinterpret_cast<uint4*>(h_out + off) = pack8(v[i]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[i][e] * v[i][e];
    }
  }
  ss = block_sum_256(ss, red);
  const float rstd = rsqrtf(ss / static_cast<float>(H) + eps);
  const bool keep = rowmask ? (rowmask[row] != 0) : true;
#pragma unroll
  for (int i = 0; i < kRowVecs; ++i) {
    const int vi = threadIdx.x + i * kRowThreads;
    if (vi < nvec) {
      const int col = vi * 8;
      const float4 wa = __ldg(reinterpret_cast<const float4*>(w1 + col));
      const float4 wb = __ldg(reinterpret_cast<const float4*>(w1 + col + 4));
      const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = keep ? (v[i][e] * rstd) * w[e] : 0.f;
      *reinterpret_cast<uint4*>(hn_out + row * H + col) = pack8(o);
    }
  }
}

// e4m3 scale of a row from the largest magnitude that each thread of its block of THREADS has seen: max|x| / 448, 1 for an
// all-zero row. red: one float per warp.
template <int THREADS = kRowThreads>
__device__ __forceinline__ float e4m3_scale(float amax, float* red, float& inv) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) amax = fmaxf(amax, red[w]);
  const float sc = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
  inv = 1.0f / sc;
  return sc;
}
// Eight values times inv, rounded to e4m3 (saturating).
__device__ __forceinline__ uint2 e4m3x8(const float (&f)[8], float inv) {
  uint32_t out[2];
#pragma unroll
  for (int e = 0; e < 8; e += 4) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[e] * inv, f[e + 1] * inv), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[e + 2] * inv, f[e + 3] * inv), __NV_SATFINITE, __NV_E4M3);
    out[e >> 2] = lo | (hi << 16);
  }
  return make_uint2(out[0], out[1]);
}

// Residual stream kept in fp32. One CTA per row: h = x_init (bf16, first norm of a forward) or h + delta, where delta is the
// sum of SPLITS fp32 partial rows (SPLITS > 0) or one bf16 row or nothing; the sum is added in fp32 and h is never rounded.
// hn = bf16(h * rstd * w1): the only rounding is the one the consuming GEMM needs for its operand.
// THREADS = 256 with four 16-byte vectors to a thread, or, for few rows, 1024 with one: one round of loads per row instead of three.
template <int SPLITS, int THREADS, bool E4M3 = false>
__global__ void __launch_bounds__(THREADS)
resnorm_f32_kernel(float* __restrict__ h, const bf16_t* __restrict__ x_init, const bf16_t* __restrict__ delta,
                   const float* __restrict__ parts, int64_t part_stride, const float* __restrict__ w1,
                   const int32_t* __restrict__ rowmask, bf16_t* __restrict__ hn_out, int H, float eps,
                   uint8_t* __restrict__ q_out = nullptr, float* __restrict__ q_scale = nullptr) {
  pdl_begin();
  constexpr int kVecs = kRowThreads * kRowVecs / THREADS;
  __shared__ float red[32];
  const int64_t row = blockIdx.x;
  const int nvec = H >> 3;
  float v[kVecs][8];
  float ss = 0.f;
  // Few rows: the norm's weights and the row mask are asked for with the row, not behind the sum over it (another trip to the L2 on a
  // chain of a few microseconds). 32 / 288 rows, three planes: 3.34 / 5.60 -> 3.09 / 5.37 us. Not with five planes or more: those registers
  // would leave one row of 640 threads to an SM in place of two (6 planes at 192 rows 6.5 us, with early weights 7.5).
  constexpr bool kEarly = THREADS == 1024 && SPLITS < 5;
  float4 wa[kEarly ? kVecs : 1], wb[kEarly ? kVecs : 1];
  const bool keep_early = kEarly && (rowmask ? rowmask[row] != 0 : true);
  if constexpr (kEarly) {
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const int vi = threadIdx.x + i * THREADS;
      if (vi < nvec) {
        wa[i] = __ldg(reinterpret_cast<const float4*>(w1 + vi * 8));
        wb[i] = __ldg(reinterpret_cast<const float4*>(w1 + vi * 8 + 4));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int vi = threadIdx.x + i * THREADS;
    if (vi < nvec) {
      const int64_t off = row * H + static_cast<int64_t>(vi) * 8;
      if (x_init != nullptr) {
        unpack8(ldg_stream(x_init + off), v[i]);
      } else {
        const float4 a = *reinterpret_cast<const float4*>(h + off), b = *reinterpret_cast<const float4*>(h + off + 4);
        v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
        v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
      }
      if constexpr (SPLITS > 0) {
        float d[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) d[e] = 0.f;
#pragma unroll
        for (int s = 0; s < SPLITS; ++s) {
          const float* pp = parts + s * part_stride + off;
          const uint4 a = ldg_stream(pp), b = ldg_stream(pp + 4);
          d[0] += __uint_as_float(a.x); d[1] += __uint_as_float(a.y); d[2] += __uint_as_float(a.z); d[3] += __uint_as_float(a.w);
          d[4] += __uint_as_float(b.x); d[5] += __uint_as_float(b.y); d[6] += __uint_as_float(b.z); d[7] += __uint_as_float(b.w);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] += d[e];
      } else if (delta != nullptr) {
        float d[8];
        unpack8(ldg_stream(delta + off), d);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] += d[e];
      }
      if (x_init != nullptr || SPLITS > 0 || delta != nullptr) {
        *reinterpret_cast<float4*>(h + off) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
        *reinterpret_cast<float4*>(h + off + 4) = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[i][e] * v[i][e];
    }
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / static_cast<float>(H) + eps);
  float amax = 0.f;
  const bool keep = kEarly ? keep_early : (rowmask ? (rowmask[row] != 0) : true);
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int vi = threadIdx.x + i * THREADS;
    if (vi < nvec) {
      const int col = vi * 8;
      if constexpr (!kEarly) {
        wa[0] = __ldg(reinterpret_cast<const float4*>(w1 + col));
        wb[0] = __ldg(reinterpret_cast<const float4*>(w1 + col + 4));
      }
      const float4 x = wa[kEarly ? i : 0], y = wb[kEarly ? i : 0];
      const float w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = keep ? (v[i][e] * rstd) * w[e] : 0.f;
      const uint4 packed = pack8(o);
      if constexpr (E4M3) {
        unpack8(packed, v[i]);
#pragma unroll
        for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[i][e]));
      } else {
        *reinterpret_cast<uint4*>(hn_out + row * H + col) = packed;
      }
    }
  }
  if constexpr (E4M3) {      // the bf16 row, quantised as quantize_rows_e4m3_kernel does it, without its way through memory
    __syncthreads();         // (red is read by every warp of block_sum)
    float inv;
    const float sc = e4m3_scale(amax, red, inv);
    if (threadIdx.x == 0) q_scale[row] = sc;
#pragma unroll
    for (int i = 0; i < kVecs; ++i) {
      const int vi = threadIdx.x + i * THREADS;
      if (vi < nvec) *reinterpret_cast<uint2*>(q_out + row * H + vi * 8) = e4m3x8(v[i], inv);
    }
  }
}

__global__ void act_tables_kernel(bf16_t* __restrict__ silu_tab, float* __restrict__ sig_tab) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 65536u) return;
  const float x = __uint_as_float(i << 16);  // bf16 bit pattern widened to fp32
  silu_tab[i] = f2bf(silu_f(x));
  sig_tab[i] = sigmoid_f(x);
}

// 8 outputs per thread; gate at column c, up at column I + c of the same row.
__global__ void __launch_bounds__(256)
silu_mul_kernel(const bf16_t* __restrict__ gu, const bf16_t* __restrict__ tab, bf16_t* __restrict__ out, int I, int64_t nvec) {
  pdl_begin();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nvec) return;
  const int vec_per_row = I >> 3;
  const int64_t row = i / vec_per_row;
  const int col = static_cast<int>(i - row * vec_per_row) * 8;
  const bf16_t* gp = gu + row * 2 * I + col;
  const uint4 gv = ldg_stream(gp), uv = ldg_stream(gp + I);
  float u[8], o[8];
  unpack8(uv, u);
  if (tab != nullptr) {
    const uint16_t* gs = reinterpret_cast<const uint16_t*>(&gv);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = bf2f(__ldg(tab + gs[e])) * u[e];
  } else {
    float g[8];
    unpack8(gv, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = round_bf(silu_f(g[e])) * u[e];
  }
  *reinterpret_cast<uint4*>(out + row * I + col) = pack8(o);
}

__global__ void __launch_bounds__(256)
gate_mul_kernel(const bf16_t* __restrict__ att, int64_t stride_t, int64_t stride_h, const bf16_t* __restrict__ gate,
                bf16_t* __restrict__ y, int HQ, int D, int64_t nvec) {
  pdl_begin();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nvec) return;
  const int64_t e0 = i * 8;
  const int d = static_cast<int>(e0 % D);
  const int64_t th = e0 / D;
  const int h = static_cast<int>(th % HQ);
  const int64_t t = th / HQ;
  float a[8], g[8], o[8];
  unpack8(ldg_stream(att + h * stride_h + t * stride_t + d), a);
  unpack8(ldg_stream(gate + e0), g);
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = a[e] * round_bf(sigmoid_f(g[e]));
  *reinterpret_cast<uint4*>(y + e0) = pack8(o);
}

// One warp per 32 keys of one row: ballot of the visibility bytes.
__global__ void __launch_bounds__(256) pack_bits_kernel(const uint8_t* __restrict__ vis, int32_t* __restrict__ bits, int64_t nwords, int N) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= nwords) return;
  const int lane = threadIdx.x & 31;
  const int words_per_row = N >> 5;
  const int64_t row = w / words_per_row;
  const int wc = static_cast<int>(w - row * words_per_row);
  const uint32_t b = __ballot_sync(0xffffffffu, vis[row * N + wc * 32 + lane] != 0);
  if (lane == 0) bits[w] = static_cast<int32_t>(b);
}

// One warp per (row, task); tasks = HQ query heads, HKV key heads, HKV value heads. Each lane owns D/32 (<= 8) contiguous
// dims. Rotary partner d <-> d + RD/2 lives RD/(2*per) lanes away.
template <int PER>
__global__ void __launch_bounds__(256)
fullattn_prep_kernel(const bf16_t* __restrict__ proj, const float* __restrict__ qw1, const float* __restrict__ kw1,
                     const bf16_t* __restrict__ cosb, const bf16_t* __restrict__ sinb, bf16_t* __restrict__ qt,
                     bf16_t* __restrict__ kt, bf16_t* __restrict__ vt, bf16_t* __restrict__ vt_t, bf16_t* __restrict__ gate,
                     int64_t N, int HQ, int HKV, int D, int RD, float eps) {
  pdl_begin();
  const int ntask = HQ + 2 * HKV;
  const int64_t wid = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wid >= N * ntask) return;
  const int lane = threadIdx.x & 31;
  const int64_t n = wid / ntask;
  const int task = static_cast<int>(wid - n * ntask);
  const int P = HQ * 2 * D + 2 * HKV * D;
  const int d0 = lane * PER;
  const bf16_t* prow = proj + n * P;
  auto load = [&](const bf16_t* p, float* f) {
    if constexpr (PER == 8) {
      float t[8];
      unpack8(*reinterpret_cast<const uint4*>(p), t);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = t[e];
    } else {
#pragma unroll
      for (int e = 0; e < PER; ++e) f[e] = bf2f(p[e]);
    }
  };
  auto store = [&](bf16_t* p, const float* f) {
    if constexpr (PER == 8) {
      float t[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) t[e] = f[e];
      *reinterpret_cast<uint4*>(p) = pack8(t);
    } else {
#pragma unroll
      for (int e = 0; e < PER; ++e) p[e] = f2bf(f[e]);
    }
  };
  float xv[PER];
  if (task >= HQ + HKV) {  // value head: plain transpose to head-major
    const int kh = task - HQ - HKV;
    load(prow + HQ * 2 * D + HKV * D + kh * D + d0, xv);
    store(vt + (static_cast<int64_t>(kh) * N + n) * D + d0, xv);
    if (vt_t != nullptr) {      // the same values with rows and columns exchanged: [HKV, D, N] (the tcgen05 attention kernel reads V
#pragma unroll                  // blocks as K-major operand tiles, keys contiguous)
      for (int e = 0; e < PER; ++e) vt_t[(static_cast<int64_t>(kh) * D + d0 + e) * N + n] = f2bf(xv[e]);
    }
    return;
  }
  const bool isq = task < HQ;
  const int hh = isq ? task : task - HQ;
  const bf16_t* src = isq ? prow + static_cast<int64_t>(hh) * 2 * D : prow + HQ * 2 * D + static_cast<int64_t>(hh) * D;
  if (isq) {
    float gv[PER];
    load(src + D + d0, gv);
    store(gate + n * (static_cast<int64_t>(HQ) * D) + hh * D + d0, gv);
  }
  load(src + d0, xv);
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < PER; ++e) ss += xv[e] * xv[e];
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss / static_cast<float>(D) + eps);
  const float* w1 = isq ? qw1 : kw1;
  float nv[PER], pv[PER], ov[PER];
#pragma unroll
  for (int e = 0; e < PER; ++e) nv[e] = round_bf((xv[e] * rstd) * __ldg(w1 + d0 + e));
  const int partner = (RD / 2) / PER;  // lane distance of the rotate-half partner
#pragma unroll
  for (int e = 0; e < PER; ++e) pv[e] = __shfl_xor_sync(0xffffffffu, nv[e], partner);
  const bool rope = d0 < RD;
#pragma unroll
  for (int e = 0; e < PER; ++e) {
    if (rope) {
      const float c = bf2f(cosb[n * RD + d0 + e]), s = bf2f(sinb[n * RD + d0 + e]);
      const float rh = (d0 + e < RD / 2) ? -pv[e] : pv[e];
      ov[e] = round_bf(round_bf(nv[e] * c) + round_bf(rh * s));
    } else {
      ov[e] = nv[e];
    }
  }
  bf16_t* dst = isq ? qt : kt;
  store(dst + (static_cast<int64_t>(hh) * N + n) * D + d0, ov);
}

// Operands of the tcgen05 tree attention (head dim 256) from the in-projection: q and k normalised and rotated, head-major; V with
// keys contiguous. The first blocks (8 warps) do q and k: a warp takes kPrepRows rows of one head, so the norm weights are read
// once and the rows' loads are in flight together. The other blocks transpose tiles of 64 keys x 64 dims of V through shared
// memory, so that both sides move in 128-byte pieces.
// Bound by memory: 2 x 2 bytes per q / k / v element, N * (HQ + 2 HKV) * 256 of them. fullattn_prep_kernel, which the attention
// path used before, also copies the gate (the attention now reads it in place), writes V a second time in row order and stores
// the transposed V element by element (2-byte stores N apart): 530 us at 16 672 rows and 19 us at 540, here 123 and 7.2 us.
constexpr int kPrepRows = 4;
constexpr int kPrepTile = 64;

__global__ void __launch_bounds__(256)
attn_operands_kernel(const bf16_t* __restrict__ q_src, int64_t q_ld, const int64_t* __restrict__ q_rows, int NQ,
                     const bf16_t* __restrict__ kv_src, int64_t kv_ld, const float* __restrict__ qw1, const float* __restrict__ kw1,
                     const bf16_t* __restrict__ cosb, const bf16_t* __restrict__ sinb, bf16_t* __restrict__ qt,
                     bf16_t* __restrict__ kt, bf16_t* __restrict__ vt_t, int N, int HQ, int HKV, int RD, float eps, int q_blocks,
                     int k_blocks) {
  pdl_begin();
  constexpr int D = 256;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ bf16_t tile[kPrepTile][kPrepTile + 2];
  const int blk = blockIdx.x;
  if (blk < q_blocks + k_blocks) {
    // block = 8 groups of kPrepRows rows of one head: consecutive blocks take consecutive heads of the same rows
    const bool isq = blk < q_blocks;
    const int heads = isq ? HQ : HKV, rows = isq ? NQ : N;
    const int b = isq ? blk : blk - q_blocks;
    const int hh = b % heads, n0 = (b / heads * 8 + warp) * kPrepRows;
    const bf16_t* src = isq ? q_src + static_cast<int64_t>(hh) * 2 * D : kv_src + static_cast<int64_t>(hh) * D;
    const int64_t ld = isq ? q_ld : kv_ld;
    bf16_t* dst = (isq ? qt : kt) + static_cast<int64_t>(hh) * rows * D;
    const float* w1 = isq ? qw1 : kw1;
    const int d0 = lane * 8;
    uint4 raw[kPrepRows];
#pragma unroll
    for (int r = 0; r < kPrepRows; ++r)
      raw[r] = n0 + r < rows ? ldg_stream(src + (n0 + r) * ld + d0) : make_uint4(0u, 0u, 0u, 0u);
    const float4 wa = __ldg(reinterpret_cast<const float4*>(w1 + d0)), wb = __ldg(reinterpret_cast<const float4*>(w1 + d0 + 4));
    const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
    const bool rope = d0 < RD, first = d0 < RD / 2;
    const int partner = RD / 16;      // lane distance of the rotate-half partner
#pragma unroll
    for (int r = 0; r < kPrepRows; ++r) {
      const int n = n0 + r;
      if (n >= rows) break;
      float x[8], nv[8], pv[8];
      unpack8(raw[r], x);
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += x[e] * x[e];
      ss = warp_sum(ss);
      const float rstd = rsqrtf(ss / static_cast<float>(D) + eps);
#pragma unroll
      for (int e = 0; e < 8; ++e) nv[e] = round_bf((x[e] * rstd) * w[e]);
#pragma unroll
      for (int e = 0; e < 8; ++e) pv[e] = __shfl_xor_sync(0xffffffffu, nv[e], partner);
      if (rope) {
        const int64_t tn = (isq && q_rows != nullptr) ? nearest_row(q_rows[n], N) : n;
        float c[8], s[8];
        unpack8(*reinterpret_cast<const uint4*>(cosb + tn * RD + d0), c);
        unpack8(*reinterpret_cast<const uint4*>(sinb + tn * RD + d0), s);
#pragma unroll
        for (int e = 0; e < 8; ++e) nv[e] = round_bf(nv[e] * c[e]) + round_bf((first ? -pv[e] : pv[e]) * s[e]);
      }
      *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(n) * D + d0) = pack8(nv);
    }
    return;
  }
  const int b = blk - q_blocks - k_blocks, cols = HKV * D / kPrepTile;
  const int c0 = b % cols * kPrepTile, n0 = b / cols * kPrepTile;
  const bf16_t* v = kv_src + static_cast<int64_t>(HKV) * D + c0;
#pragma unroll
  for (int u = 0; u < kPrepTile * kPrepTile / 8 / 256; ++u) {
    const int i = threadIdx.x + u * 256, r = i >> 3, c = (i & 7) * 8;
    if (n0 + r < N) {
      const uint4 x = ldg_stream(v + (n0 + r) * kv_ld + c);
      uint32_t* t = reinterpret_cast<uint32_t*>(&tile[r][c]);
      t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w;
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < kPrepTile * kPrepTile / 8 / 256; ++u) {
    const int i = threadIdx.x + u * 256, c = i >> 3, r = (i & 7) * 8;
    if (n0 + r < N) {      // N is a multiple of 8: all eight keys or none
      alignas(16) bf16_t o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = tile[r + e][c];
      *reinterpret_cast<uint4*>(vt_t + static_cast<int64_t>(c0 + c) * N + n0 + r) = *reinterpret_cast<const uint4*>(o);
    }
  }
}

// Rows rows[i] of one or two matrices, one block per output row; an index outside gives a row of ones (not-a-number) and is reported.
__global__ void __launch_bounds__(256)
gather_rows_kernel(const int64_t* __restrict__ rows, int64_t n_src, const uint4* __restrict__ a, uint4* __restrict__ a_out, int a_vecs,
                   const uint4* __restrict__ b, uint4* __restrict__ b_out, int b_vecs, int32_t* status) {
  pdl_begin();
  const int64_t i = blockIdx.x, n = row_of_index(rows[i], n_src);
  if (n < 0) {
    const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (int c = threadIdx.x; c < a_vecs; c += blockDim.x) a_out[i * a_vecs + c] = ones;
    for (int c = threadIdx.x; c < b_vecs; c += blockDim.x) b_out[i * b_vecs + c] = ones;
    if (threadIdx.x == 0) report_status(status, OJB_DEV_ROW_INDEX);
    return;
  }
  for (int c = threadIdx.x; c < a_vecs; c += blockDim.x) a_out[i * a_vecs + c] = a[n * a_vecs + c];
  for (int c = threadIdx.x; c < b_vecs; c += blockDim.x) b_out[i * b_vecs + c] = b[n * b_vecs + c];
}

// Per-row e4m3 quantisation for the 8-bit GEMM (e4m3_scale, e4m3x8). One CTA per row, two passes over the row (the second one hits
// L1 / L2): for rows too long for the registers.
__global__ void __launch_bounds__(kRowThreads)
quantize_rows_e4m3_kernel(const bf16_t* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale, int K) {
  pdl_begin();
  __shared__ float red[kRowThreads / 32];
  const int64_t row = blockIdx.x;
  const bf16_t* xr = x + row * K;
  float amax = 0.f;
  for (int i = threadIdx.x * 8; i < K; i += kRowThreads * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + i), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
  }
  float inv;
  const float sc = e4m3_scale(amax, red, inv);
  if (threadIdx.x == 0) scale[row] = sc;
  uint8_t* qr = q + row * K;
  for (int i = threadIdx.x * 8; i < K; i += kRowThreads * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + i), f);
    *reinterpret_cast<uint2*>(qr + i) = e4m3x8(f, inv);
  }
}

// The same for rows of up to THREADS * VECS vectors of eight, which stay in registers between the two passes. Bound by memory (3 bytes
// per element): all of a row's loads are in flight at once and none is repeated, and small blocks leave many rows to an SM, so that the
// barrier of one is covered by the loads of others. 4224 rows of 17 408: 46 -> 32 us, 6.8 TB/s; 544 rows: 7.4 -> 4.4.
template <int THREADS, int VECS>
__global__ void __launch_bounds__(THREADS)
quantize_held_rows_e4m3_kernel(const bf16_t* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale, int nvec) {
  pdl_begin();
  __shared__ float red[THREADS / 32];
  const int64_t row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x) + row * nvec + threadIdx.x;
  uint4 v[VECS];
#pragma unroll
  for (int i = 0; i < VECS; ++i)
    v[i] = static_cast<int>(threadIdx.x) + i * THREADS < nvec ? xr[i * THREADS] : make_uint4(0u, 0u, 0u, 0u);
  __nv_bfloat162 mx = __float2bfloat162_rn(0.f);      // (the maximum of bf16 values is one of them)
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
#pragma unroll
    for (int e = 0; e < 4; ++e) mx = __hmax2(mx, __habs2(p[e]));
  }
  const float2 m = __bfloat1622float2(mx);
  float inv;
  const float sc = e4m3_scale<THREADS>(fmaxf(m.x, m.y), red, inv);
  if (threadIdx.x == 0) scale[row] = sc;
  uint2* qr = reinterpret_cast<uint2*>(q) + row * nvec + threadIdx.x;
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    float f[8];
    unpack8(v[i], f);
    if (static_cast<int>(threadIdx.x) + i * THREADS < nvec) qr[i * THREADS] = e4m3x8(f, inv);
  }
}

// One thread per slice: a bulk prefetch into L2, nothing is held or waited for.
__global__ void l2_prefetch_kernel(const uint8_t* __restrict__ base, int64_t nbytes, int chunk) {
  const int64_t off = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * chunk;
  if (off >= nbytes) return;
  const uint32_t sz = static_cast<uint32_t>(nbytes - off < chunk ? nbytes - off : chunk);
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base + off), "r"(sz) : "memory");
}

}  // namespace
}  // namespace ojb

using namespace ojb;

extern "C" int ojb_l2_prefetch(const void* data, int64_t nbytes, int64_t chunk, ojb_stream_t stream) {
  OJB_REQUIRE(data && nbytes >= 0 && chunk >= 16 && chunk % 16 == 0 && chunk <= (1 << 20));
  OJB_REQUIRE((reinterpret_cast<uintptr_t>(data) & 15u) == 0);
  nbytes &= ~static_cast<int64_t>(15);
  if (nbytes == 0) return OJB_OK;
  const int64_t n = ceil_div(nbytes, chunk);
  l2_prefetch_kernel<<<static_cast<unsigned>(ceil_div(n, 128)), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(data), nbytes, static_cast<int>(chunk));
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_abi_version(void) { return 9; }

extern "C" int ojb_add_rmsnorm(const void* x, const void* delta, const float* w1, const int32_t* rowmask, void* h_out,
                               void* hn_out, int64_t rows, int64_t H, float eps, ojb_stream_t stream) {
  if (rows == 0) return OJB_OK;
  OJB_REQUIRE(x && w1 && hn_out && rows > 0 && H > 0 && H % 8 == 0);
  OJB_REQUIRE(delta == nullptr || h_out != nullptr);
  if (H > kRowThreads * kRowVecs * 8) return OJB_ERR_LIMIT;
  launch_kernel(add_rmsnorm_kernel<0>, dim3(static_cast<unsigned>(rows)), dim3(kRowThreads), 0, static_cast<cudaStream_t>(stream), 
      static_cast<const bf16_t*>(x), static_cast<const bf16_t*>(delta), nullptr, 0, w1, rowmask,
      static_cast<bf16_t*>(h_out), static_cast<bf16_t*>(hn_out), static_cast<int>(H), eps);
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_add_rmsnorm_sk(const void* x, const float* parts, int splits, const float* w1, const int32_t* rowmask,
                                  void* h_out, void* hn_out, int64_t rows, int64_t H, float eps, ojb_stream_t stream) {
  if (rows == 0) return OJB_OK;
  OJB_REQUIRE(x && parts && w1 && h_out && hn_out && rows > 0 && H > 0 && H % 8 == 0 && splits >= 1 && splits <= 16);
  if (H > kRowThreads * kRowVecs * 8) return OJB_ERR_LIMIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t ps = rows * H;
#define OJB_SK(S)                                                                                                     \
  case S:                                                                                                             \
    launch_kernel(add_rmsnorm_kernel<S>, dim3(static_cast<unsigned>(rows)), dim3(kRowThreads), 0, st,                                        \
        static_cast<const bf16_t*>(x), nullptr, parts, ps, w1, rowmask, static_cast<bf16_t*>(h_out),                  \
        static_cast<bf16_t*>(hn_out), static_cast<int>(H), eps);                                                      \
    break;
  switch (splits) {
    OJB_SK(1) OJB_SK(2) OJB_SK(3) OJB_SK(4) OJB_SK(5) OJB_SK(6) OJB_SK(7) OJB_SK(8)
    OJB_SK(9) OJB_SK(10) OJB_SK(11) OJB_SK(12) OJB_SK(13) OJB_SK(14) OJB_SK(15) OJB_SK(16)
  }
#undef OJB_SK
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_resnorm_f32(float* h, const void* x_init, const void* delta, const float* parts, int splits,
                               const float* w1, const int32_t* rowmask, void* hn_out, int64_t rows, int64_t H, float eps,
                               ojb_stream_t stream) {
  if (rows == 0) return OJB_OK;
  OJB_REQUIRE(h && w1 && hn_out && rows > 0 && H > 0 && H % 8 == 0 && splits >= 0 && splits <= 16);
  OJB_REQUIRE((splits == 0) == (parts == nullptr));
  OJB_REQUIRE(!(parts && delta) && !(x_init && (parts || delta)));
  if (H > kRowThreads * kRowVecs * 8) return OJB_ERR_LIMIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t ps = rows * H;
  // measured (us, one / six K ranges): 32 rows 3.7 / 5.1 -> 3.1 / 3.9, 288 rows 4.6 / 7.4 -> 4.2 / 7.1, 544 rows 6.9 / 11.5 against
  // 7.8 / 13.0: with two wide rows to an SM a second wave begins
  const bool wide = rows <= 296;
#define OJB_RN_T(S, T, THREADS)                                                                                          \
  launch_kernel(resnorm_f32_kernel<S, T>, dim3(static_cast<unsigned>(rows)), dim3(THREADS), 0, st, h,                    \
                static_cast<const bf16_t*>(x_init), static_cast<const bf16_t*>(delta), parts, ps, w1, rowmask,           \
                static_cast<bf16_t*>(hn_out), static_cast<int>(H), eps, static_cast<uint8_t*>(nullptr),                  \
                static_cast<float*>(nullptr))
#define OJB_RN(S)                                                                                                       \
  case S:                                                                                                               \
    if (wide) OJB_RN_T(S, 1024, static_cast<unsigned>(ceil_div(H / 8, 32) * 32));                                       \
    else OJB_RN_T(S, kRowThreads, kRowThreads);                                                                         \
    break;
  switch (splits) {
    OJB_RN(0) OJB_RN(1) OJB_RN(2) OJB_RN(3) OJB_RN(4) OJB_RN(5) OJB_RN(6) OJB_RN(7) OJB_RN(8)
    OJB_RN(9) OJB_RN(10) OJB_RN(11) OJB_RN(12) OJB_RN(13) OJB_RN(14) OJB_RN(15) OJB_RN(16)
  }
#undef OJB_RN
#undef OJB_RN_T
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_resnorm_f32_e4m3(float* h, const void* x_init, const float* parts, int splits, const float* w1,
                                    const int32_t* rowmask, void* q, float* scale, int64_t rows, int64_t H, float eps,
                                    ojb_stream_t stream) {
  if (rows == 0) return OJB_OK;
  OJB_REQUIRE(h && w1 && q && scale && rows > 0 && H > 0 && H % 8 == 0 && splits >= 0 && splits <= 16);
  OJB_REQUIRE((splits == 0) == (parts == nullptr) && !(x_init && parts));
  if (H > kRowThreads * kRowVecs * 8) return OJB_ERR_LIMIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define OJB_RQ(S)                                                                                                       \
  case S:                                                                                                               \
    launch_kernel(resnorm_f32_kernel<S, kRowThreads, true>, dim3(static_cast<unsigned>(rows)), dim3(kRowThreads), 0, st, h, \
                  static_cast<const bf16_t*>(x_init), static_cast<const bf16_t*>(nullptr), parts, rows * H, w1, rowmask, \
                  static_cast<bf16_t*>(nullptr), static_cast<int>(H), eps, static_cast<uint8_t*>(q), scale);             \
    break;
  switch (splits) {
    OJB_RQ(0) OJB_RQ(1) OJB_RQ(2) OJB_RQ(3) OJB_RQ(4) OJB_RQ(5) OJB_RQ(6) OJB_RQ(7) OJB_RQ(8)
    OJB_RQ(9) OJB_RQ(10) OJB_RQ(11) OJB_RQ(12) OJB_RQ(13) OJB_RQ(14) OJB_RQ(15) OJB_RQ(16)
  }
#undef OJB_RQ
  return launch_status(cudaGetLastError());
}

// ---- embedding rows + rotary tables of a packed tree: the two things the forward needs before its first layer.
// Block n copies row ids[n] of the embedding table to x[n] (an id outside the table gives a zero row) and writes
// cos / sin of pos[n] * inv_freq[j] for the R2 rotary frequencies, each value twice (columns j and j + R2), as the
// reference's rotary module does for text positions: angle and cos / sin in fp32, one rounding to bf16.
__global__ void __launch_bounds__(256)
embed_rope_kernel(const int64_t* __restrict__ ids, const bf16_t* __restrict__ table, int64_t vocab,
                  const int64_t* __restrict__ pos, const float* __restrict__ inv_freq, float scaling,
                  bf16_t* __restrict__ x, bf16_t* __restrict__ cosb, bf16_t* __restrict__ sinb, int H, int R2) {
  pdl_begin();
  const int64_t n = blockIdx.x;
  const int64_t id = ids[n];
  const bool ok = id >= 0 && id < vocab;
  const uint4* src = reinterpret_cast<const uint4*>(table + (ok ? id : 0) * H);
  uint4* dst = reinterpret_cast<uint4*>(x + n * H);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) dst[i] = ok ? __ldg(src + i) : make_uint4(0u, 0u, 0u, 0u);
  const float p = static_cast<float>(pos[n]);
  for (int j = threadIdx.x; j < R2; j += blockDim.x) {
    const float a = inv_freq[j] * p;
    const bf16_t c = f2bf(cosf(a) * scaling), sn = f2bf(sinf(a) * scaling);
    cosb[n * 2 * R2 + j] = c; cosb[n * 2 * R2 + R2 + j] = c;
    sinb[n * 2 * R2 + j] = sn; sinb[n * 2 * R2 + R2 + j] = sn;
  }
}

extern "C" int ojb_embed_rope(const int64_t* ids, const void* table, int64_t vocab, const int64_t* pos, const float* inv_freq,
                              float scaling, void* x, void* cosb, void* sinb, int64_t N, int64_t H, int64_t R2,
                              ojb_stream_t stream) {
  if (N == 0) return OJB_OK;
  OJB_REQUIRE(ids && table && pos && inv_freq && x && cosb && sinb && N > 0 && vocab > 0 && H > 0 && H % 8 == 0 && R2 > 0);
  OJB_REQUIRE((reinterpret_cast<uintptr_t>(table) & 15u) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0);
  launch_kernel(embed_rope_kernel, dim3(static_cast<unsigned>(N)), dim3(256), 0, static_cast<cudaStream_t>(stream), ids,
                static_cast<const bf16_t*>(table), vocab, pos, inv_freq, scaling, static_cast<bf16_t*>(x),
                static_cast<bf16_t*>(cosb), static_cast<bf16_t*>(sinb), static_cast<int>(H), static_cast<int>(R2));
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_act_tables(void* silu_tab, float* sig_tab, ojb_stream_t stream) {
  OJB_REQUIRE(silu_tab && sig_tab);
  act_tables_kernel<<<256, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<bf16_t*>(silu_tab), sig_tab);
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_silu_mul(const void* gu, const void* silu_tab, void* out, int64_t rows, int64_t I, ojb_stream_t stream) {
  OJB_REQUIRE(gu && out && rows >= 0 && I > 0 && I % 8 == 0);
  const int64_t nvec = rows * I / 8;
  if (nvec == 0) return OJB_OK;
  launch_kernel(silu_mul_kernel, dim3(static_cast<unsigned>(ceil_div(nvec, 256))), dim3(256), 0, static_cast<cudaStream_t>(stream), 
      static_cast<const bf16_t*>(gu), static_cast<const bf16_t*>(silu_tab), static_cast<bf16_t*>(out), static_cast<int>(I), nvec);
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_gate_mul(const void* att, int64_t att_stride_t, int64_t att_stride_h, const void* gate, void* y,
                            int64_t T, int64_t HQ, int64_t D, ojb_stream_t stream) {
  OJB_REQUIRE(att && gate && y && T >= 0 && HQ > 0 && D > 0 && D % 8 == 0 && att_stride_t % 8 == 0 && att_stride_h % 8 == 0);
  const int64_t nvec = T * HQ * D / 8;
  if (nvec == 0) return OJB_OK;
  launch_kernel(gate_mul_kernel, dim3(static_cast<unsigned>(ceil_div(nvec, 256))), dim3(256), 0, static_cast<cudaStream_t>(stream), 
      static_cast<const bf16_t*>(att), att_stride_t, att_stride_h, static_cast<const bf16_t*>(gate), static_cast<bf16_t*>(y),
      static_cast<int>(HQ), static_cast<int>(D), nvec);
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_pack_bits(const uint8_t* vis, int32_t* bits, int64_t N, ojb_stream_t stream) {
  OJB_REQUIRE(vis && bits && N > 0 && N % 32 == 0);
  const int64_t nwords = N * (N / 32);
  pack_bits_kernel<<<static_cast<unsigned>(ceil_div(nwords, 8)), 256, 0, static_cast<cudaStream_t>(stream)>>>(vis, bits, nwords,
                                                                                                        static_cast<int>(N));
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_fullattn_prep(const void* proj, const float* qw1, const float* kw1, const void* cosb, const void* sinb,
                                 void* qt, void* kt, void* vt, void* vt_t, void* gate, int64_t N, int64_t HQ, int64_t HKV,
                                 int64_t D, int64_t RD, float eps, ojb_stream_t stream) {
  OJB_REQUIRE(proj && qw1 && kw1 && cosb && sinb && qt && kt && vt && gate && N >= 0 && HQ > 0 && HKV > 0);
  OJB_REQUIRE(D == 256 || D == 128 || D == 64);
  const int per = static_cast<int>(D / 32);
  OJB_REQUIRE(RD > 0 && RD <= D && RD % (2 * per) == 0);
  if (N == 0) return OJB_OK;
  const int64_t warps = N * (HQ + 2 * HKV);
  const unsigned grid = static_cast<unsigned>(ceil_div(warps, 8));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define OJB_PREP(P)                                                                                                     \
  launch_kernel(fullattn_prep_kernel<P>, dim3(grid), dim3(256), 0, st, static_cast<const bf16_t*>(proj), qw1, kw1,                             \
                                                static_cast<const bf16_t*>(cosb), static_cast<const bf16_t*>(sinb),     \
                                                static_cast<bf16_t*>(qt), static_cast<bf16_t*>(kt),                     \
                                                static_cast<bf16_t*>(vt), static_cast<bf16_t*>(vt_t),                   \
                                                static_cast<bf16_t*>(gate), N,                                          \
                                                static_cast<int>(HQ), static_cast<int>(HKV), static_cast<int>(D),       \
                                                static_cast<int>(RD), eps)
  if (per == 8) OJB_PREP(8); else if (per == 4) OJB_PREP(4); else OJB_PREP(2);
#undef OJB_PREP
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_attn_operands(const void* q_src, int64_t q_ld, const int64_t* q_rows, int64_t NQ, const void* kv_src, int64_t kv_ld,
                                 const float* qw1, const float* kw1, const void* cosb, const void* sinb, void* qt, void* kt,
                                 void* vt_t, int64_t N, int64_t HQ, int64_t HKV, int64_t RD, float eps, ojb_stream_t stream) {
  constexpr int D = 256;
  OJB_REQUIRE(q_src && kv_src && qw1 && kw1 && cosb && sinb && qt && kt && vt_t && N > 0 && NQ > 0 && HQ > 0 && HKV > 0);
  OJB_REQUIRE(N % 8 == 0 && N < (1 << 24) && NQ < (1 << 24) && HQ <= 1024 && HKV <= 1024);
  OJB_REQUIRE(q_rows != nullptr || NQ <= N);      // without q_rows query row n takes row n of the rotary tables, which have N
  OJB_REQUIRE(RD > 0 && RD <= D && RD % 16 == 0 && (RD & (RD - 1)) == 0);
  OJB_REQUIRE(q_ld >= HQ * 2 * D && q_ld % 8 == 0 && kv_ld >= HKV * 2 * D && kv_ld % 8 == 0);
  for (const void* p : {q_src, kv_src, static_cast<const void*>(qw1), static_cast<const void*>(kw1), cosb, sinb,
                        static_cast<const void*>(qt), static_cast<const void*>(kt), static_cast<const void*>(vt_t)})
    OJB_REQUIRE((reinterpret_cast<uintptr_t>(p) & 15u) == 0);
  const int64_t q_blocks = ceil_div(NQ, 8 * kPrepRows) * HQ, k_blocks = ceil_div(N, 8 * kPrepRows) * HKV;
  const int64_t v_blocks = ceil_div(N, kPrepTile) * (HKV * D / kPrepTile);
  OJB_REQUIRE(q_blocks + k_blocks + v_blocks < (int64_t{1} << 31));
  launch_kernel(attn_operands_kernel, dim3(static_cast<unsigned>(q_blocks + k_blocks + v_blocks)), dim3(256), 0,
                static_cast<cudaStream_t>(stream), static_cast<const bf16_t*>(q_src), q_ld, q_rows, static_cast<int>(NQ),
                static_cast<const bf16_t*>(kv_src), kv_ld, qw1, kw1, static_cast<const bf16_t*>(cosb),
                static_cast<const bf16_t*>(sinb), static_cast<bf16_t*>(qt), static_cast<bf16_t*>(kt), static_cast<bf16_t*>(vt_t),
                static_cast<int>(N), static_cast<int>(HQ), static_cast<int>(HKV), static_cast<int>(RD), eps,
                static_cast<int>(q_blocks), static_cast<int>(k_blocks));
  return launch_status(cudaGetLastError());
}

extern "C" int ojb_gather_rows(const int64_t* rows, int64_t n_rows, int64_t n_src, const void* a, void* a_out, int64_t a_bytes, const void* b,
                               void* b_out, int64_t b_bytes, int32_t* status, ojb_stream_t stream) {
  if (n_rows == 0) return OJB_OK;
  OJB_REQUIRE(rows && n_rows > 0 && n_rows < (int64_t{1} << 31) && n_src > 0 && a && a_out && a_bytes > 0 && a_bytes % 16 == 0 && a_bytes < (1 << 30));
  OJB_REQUIRE(b ? (b_out && b_bytes > 0 && b_bytes % 16 == 0 && b_bytes < (1 << 30)) : (b_bytes == 0));
  for (const void* p : {a, static_cast<const void*>(a_out), b, static_cast<const void*>(b_out)})
    OJB_REQUIRE((reinterpret_cast<uintptr_t>(p) & 15u) == 0);
  launch_kernel(gather_rows_kernel, dim3(static_cast<unsigned>(n_rows)), dim3(256), 0, static_cast<cudaStream_t>(stream), rows, n_src,
                static_cast<const uint4*>(a), static_cast<uint4*>(a_out), static_cast<int>(a_bytes / 16),
                static_cast<const uint4*>(b), static_cast<uint4*>(b_out), static_cast<int>(b_bytes / 16), status);
  return launch_status(cudaGetLastError());
}

// ------------------------------------------------------------------------------------------------------- scoring head
namespace ojb {
namespace {
// one block per (candidate, output): out[s, a] = bias[a] + sum_h float(hn[rows[s], h]) * W[a, h]. A handful of outputs of 30 KB of
// reads each: what counts is one round of loads instead of twenty (one warp per output: 10-12 us).
constexpr int kHeadThreads = 320;
__global__ void __launch_bounds__(kHeadThreads)
score_head_kernel(const bf16_t* __restrict__ hn, int64_t n_src, const int64_t* __restrict__ rows, const float* __restrict__ W,
                  const float* __restrict__ bias, float* __restrict__ out, int A, int H, int32_t* status) {
  pdl_begin();
  __shared__ float red[32];
  const int s = blockIdx.x / A, a = blockIdx.x - s * A;
  const int64_t n = rows == nullptr ? s : (n_src > 0 ? row_of_index(rows[s], n_src) : rows[s]);
  if (n < 0) {      // the whole block
    if (threadIdx.x == 0) {
      out[blockIdx.x] = __int_as_float(0x7fffffff);
      report_status(status, OJB_DEV_ROW_INDEX);
    }
    return;
  }
  const bf16_t* x = hn + n * static_cast<int64_t>(H);
  const float* w = W + static_cast<int64_t>(a) * H;
  float acc = 0.f;
#pragma unroll 2
  for (int c = threadIdx.x * 8; c < H; c += kHeadThreads * 8) {
    float f[8];
    unpack8(*reinterpret_cast<const uint4*>(x + c), f);
    const float4 w0 = *reinterpret_cast<const float4*>(w + c), w1 = *reinterpret_cast<const float4*>(w + c + 4);
    acc += f[0] * w0.x + f[1] * w0.y + f[2] * w0.z + f[3] * w0.w + f[4] * w1.x + f[5] * w1.y + f[6] * w1.z + f[7] * w1.w;
  }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) out[blockIdx.x] = acc + (bias ? bias[a] : 0.f);
}
}  // namespace
}  // namespace ojb

static int launch_score_head(const void* hn, int64_t n_src, const int64_t* rows, const float* W, const float* bias, float* out, int64_t S,
                             int64_t A, int64_t H, int32_t* status, ojb_stream_t stream) {
  if (S == 0 || A == 0) return OJB_OK;
  OJB_REQUIRE(hn && W && out && S > 0 && A > 0 && H > 0 && H % 8 == 0);
  OJB_REQUIRE(S * A < (int64_t{1} << 31));
  launch_kernel(ojb::score_head_kernel, dim3(static_cast<unsigned>(S * A)), dim3(ojb::kHeadThreads), 0, static_cast<cudaStream_t>(stream),
      static_cast<const ojb::bf16_t*>(hn), n_src, rows, W, bias, out, static_cast<int>(A), static_cast<int>(H), status);
  return ojb::launch_status(cudaGetLastError());
}

extern "C" int ojb_score_head_rows(const void* hn, int64_t n_src, const int64_t* rows, const float* W, const float* bias, float* out,
                                   int64_t S, int64_t A, int64_t H, int32_t* status, ojb_stream_t stream) {
  OJB_REQUIRE(S == 0 || A == 0 || (n_src > 0 && (rows || S <= n_src)));
  return launch_score_head(hn, n_src, rows, W, bias, out, S, A, H, status, stream);
}

// without the row count of hn (n_src = 0) only a negative index is known to lie outside: none counts from the end
extern "C" int ojb_score_head(const void* hn, const int64_t* rows, const float* W, const float* bias, float* out, int64_t S,
                              int64_t A, int64_t H, ojb_stream_t stream) {
  return launch_score_head(hn, 0, rows, W, bias, out, S, A, H, nullptr, stream);
}

extern "C" int ojb_quantize_rows_e4m3(const void* x, void* q, float* scale, int64_t rows, int64_t K, ojb_stream_t stream) {
  if (rows == 0) return OJB_OK;
  OJB_REQUIRE(x && q && scale && rows > 0 && K > 0 && K % 8 == 0);
  // Smallest block that keeps a row in few registers. us of the loop / 128 x 4 / 256 x 9 (x 6 in its place at K = 6144): 544 rows of 4096
  // 3.2 / 2.4 / 2.9, of 6144 3.9 / 2.7 / 3.1, of 17 408 7.4 / - / 4.4; 4224 rows of 4096 12.6 / 6.3 / 12.5, of 6144 17.5 / 9.0 / 14.8,
  // of 17 408 45.9 / - / 32.3 (512 x 5 34.5, 1024 x 3 46.1); 32 rows of 17 408 3.8 / - / 2.4.
#define OJB_QUANTIZE(kernel, threads, len)                                                                                    \
  launch_kernel(kernel, dim3(static_cast<unsigned>(rows)), dim3(threads), 0, static_cast<cudaStream_t>(stream),              \
                static_cast<const bf16_t*>(x), static_cast<uint8_t*>(q), scale, static_cast<int>(len))
  const int64_t nvec = K / 8;
  if (nvec <= 128 * 4) OJB_QUANTIZE((quantize_held_rows_e4m3_kernel<128, 4>), 128, nvec);
  else if (nvec <= 128 * 6) OJB_QUANTIZE((quantize_held_rows_e4m3_kernel<128, 6>), 128, nvec);
  else if (nvec <= 256 * 9) OJB_QUANTIZE((quantize_held_rows_e4m3_kernel<256, 9>), 256, nvec);
  else OJB_QUANTIZE(quantize_rows_e4m3_kernel, kRowThreads, K);
#undef OJB_QUANTIZE
  return launch_status(cudaGetLastError());
}
