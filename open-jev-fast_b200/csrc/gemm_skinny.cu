// GEMM of few rows (M <= 128), sm_100a: out[M,N] = x[M,K] · w[N,K]^T for a weight that has to come from HBM.
//
// With so few rows the time is that of the weight's bytes, if enough of them are under way: at 6.4 TB/s and about 2 us from request
// to arrival that is 12 MB, 85 KB on every SM. The larger kernels fix the w tile at 128 or 256 rows and carry 128 rows of x (or
// two accumulators) beside it: 97 tiles for 12 352 outputs, 16 for 2048, each SM's share of the link idle on the rest. Here the w
// tile has any multiple of 16 rows up to 128, chosen so that the tiles (times the K ranges) fill the SMs once, and a stage holds
// the rows of x that exist and no more, so that all of the shared memory is weight in flight.
// A stage is several k-blocks, one three-dimensional copy each for x and w: with one k-block per stage the issuing warp's chain of wait,
// MMAs and commit (0.2 us) sets the pace, 21 us for K = 5120 whatever the weight's size, against 12.9 us with four.
//
// One CTA per (w tile, K range), 192 threads: warp 0 asks for the tiles (plain cp.async.bulk.tensor, 128-byte swizzle, mbarrier), one
// lane of warp 1 issues tcgen05.mma, warps 2-5 read the accumulator back and store. The MMA has M = 128 whatever its A operand: that runs on
// behind its own rows into whatever shared memory follows (the other operand, the next k-block, the next stage); a row of the product
// depends on its own row of A alone, and the rows past the operand are never read back. So a k-step costs 128 products for every row
// of the N side, and the narrower of the two operands is the N side: the rows of x (rounded up to 16) under most tiles, the w tile where
// that has fewer rows (2048 outputs: 16). With x always the M side a weight cost 128 products, most of them of other weights taken for
// rows of x, and the products of random operands are what the board's power goes to. x as the M side / the choice, in runs at the 1 kW cap
// (us): 28 rows [12352, 5120] 26.8 / 24.2, [5120, 4096] in two K ranges 11.8 / 11.2, [5120, 17408] in three 35.6 / 32.0; 64 rows 30.5 / 28.9, 12.5 /
// 11.5 and 39.7 / 35.7. In short runs 0 to 25 % faster too, e4m3 up to 33 %. Same bits. With w as the M side the accumulator leaves 16 rows of x at a time,
// loads ahead of the stores: with each load waited for and addresses formed per value it cost 0.3 us for every 16 rows and lost up to 9 %.
#include "gemm_units.cuh"

#include <type_traits>

namespace ojb {
namespace {

constexpr int kSkinnyThreads = 192;
constexpr int kSkinnyMaxStages = 40;
constexpr size_t kSkinnySmem = 227 * 1024;

struct SkinnyArgs {
  int M, N;
  int BN, x_rows;                  // rows of w and of x (a multiple of 16 as the N side, else of 8) in a stage
  int splits, kb_per_split, kb_total;
  int nk;                          // k-blocks per stage
  int stages;
  uint32_t stage_bytes, tmem_cols;
  void* out;
  int64_t ldo, split_stride;
  int32_t* status;
  int wait_ms, drop_copy;
  const float* sx;                 // e4m3 operands: scale per row of x and of w
  const float* sw;
};

// WSIDE: w is the M side, the rows of x the N side.
template <int EPI, bool FP8, bool WSIDE>
__global__ void __launch_bounds__(kSkinnyThreads, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, SkinnyArgs g) {
  pdl_launch_dependents();
  constexpr int kKE = FP8 ? 128 : kBK;      // elements of K per 128-byte k-block
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ __align__(8) uint64_t bars[2 * kSkinnyMaxStages + 1];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag[2];
  const uint32_t tiles0 = smem_u32(smem), full0 = smem_u32(bars), empty0 = full0 + 8 * kSkinnyMaxStages;
  const uint32_t accfull = empty0 + 8 * kSkinnyMaxStages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / g.splits, split = blockIdx.x - tile * g.splits;
  const int kb0 = split * g.kb_per_split, nkb = min(kb0 + g.kb_per_split, g.kb_total) - kb0;
  const int n0 = tile * g.BN;
  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(accfull, 1);
    abort_flag[0] = 0;
    abort_flag[1] = g.wait_ms;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), g.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  pdl_wait();

  const uint32_t x_bytes = static_cast<uint32_t>(g.x_rows) * 128, w_bytes = static_cast<uint32_t>(g.BN) * 128;      // of one k-block
  if (warp == 0) {
    {
      const bool one = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < nkb; kb += g.nk) {
        if (!mbar_wait_warp(empty0 + 8 * stage, phase ^ 1u, abort_flag)) break;
        const uint32_t dst = tiles0 + stage * g.stage_bytes, fb = full0 + 8 * stage;
        if (one) mbar_expect_tx(fb, g.stage_bytes);
        if (!(g.drop_copy && kb == g.nk)) {      // tests only: the announced bytes never arrive
          // (k-blocks past the end of this range are not multiplied; past the end of K they arrive as zeros)
          if (one) tma_load_3d(dst + g.nk * x_bytes, &map_w, fb, 0, n0, kb0 + kb);
          if (one) tma_load_3d(dst, &map_x, fb, 0, 0, kb0 + kb);
        }
        if (++stage == g.stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    {
      const bool one = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      const int n_side = WSIDE ? g.x_rows : g.BN;
      const uint32_t idesc = FP8 ? umma_idesc_e4m3(n_side) : umma_idesc(n_side);
      bool ok = true;
      for (int kb = 0; kb < nkb; kb += g.nk) {
        if (!mbar_wait_warp(full0 + 8 * stage, phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t src = tiles0 + stage * g.stage_bytes;
        for (int j = 0; j < g.nk && kb + j < nkb; ++j) {
          const uint64_t xdesc = smem_desc_sw128(src + j * x_bytes), wdesc = smem_desc_sw128(src + g.nk * x_bytes + j * w_bytes);
          const uint64_t adesc = WSIDE ? wdesc : xdesc, bdesc = WSIDE ? xdesc : wdesc;
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k) {
            const uint32_t accum = (kb + j > 0 || k > 0) ? 1u : 0u;
            if (one) {
              if constexpr (FP8) umma_f8(tmem_base, adesc + 2 * k, bdesc + 2 * k, idesc, accum);
              else umma_bf16(tmem_base, adesc + 2 * k, bdesc + 2 * k, idesc, accum);
            }
          }
        }
        if (one) umma_commit(empty0 + 8 * stage);
        if (++stage == g.stages) { stage = 0; phase ^= 1u; }
      }
      if (ok && one) umma_commit(accfull);
    }
  } else {
    const int quarter = warp & 3, row = quarter * 32 + lane;      // this thread's row of the M side
    if (mbar_wait_warp(accfull, 0, abort_flag)) {
      tc_fence_after();
      const int ncols = min(g.N - n0, g.BN);
      if constexpr (WSIDE) {
        if (quarter * 32 < ncols) {
          const bool col_ok = row < ncols;
          float ws = 1.f;
          if constexpr (FP8) ws = __ldg(g.sw + min(n0 + row, g.N - 1));
          const int64_t off = static_cast<int64_t>(split) * g.split_stride + n0 + row;
          using Out = std::conditional_t<EPI == kEpiPartialF32, float, bf16_t>;
          Out* const out = reinterpret_cast<Out*>(g.out) + off;
          const uint32_t acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
          // neighbouring lanes hold neighbouring columns: whole 128- or 64-byte pieces of a row; TMEM loads run 16 rows ahead of the stores
          auto emit = [&](int m0, const uint32_t (&r)[16]) {
            Out* p = out + static_cast<int64_t>(m0) * g.ldo;
#pragma unroll
            for (int e = 0; e < 16; ++e, p += g.ldo) {
              if (col_ok && m0 + e < g.M) {
                float v = __uint_as_float(r[e]);
                if constexpr (FP8) v *= __ldg(g.sx + m0 + e) * ws;
                if constexpr (EPI == kEpiPartialF32) *p = v;
                else *p = f2bf(v);
              }
            }
            __syncwarp();
          };
          uint32_t ra[16], rb[16];
          tmem_ld16(acc, ra);
          tmem_ld_wait();
#pragma unroll 1
          for (int m0 = 0; m0 < g.M; m0 += 32) {
            if (m0 + 16 < g.M) tmem_ld16(acc + m0 + 16, rb);
            emit(m0, ra);
            tmem_ld_wait();
            if (m0 + 16 < g.M) {
              if (m0 + 32 < g.M) tmem_ld16(acc + m0 + 32, ra);
              emit(m0 + 16, rb);
              tmem_ld_wait();
            }
          }
        }
      } else {
        if (quarter * 32 < g.M) {
          const bool row_ok = row < g.M;
          float rs = 1.f;
          if constexpr (FP8) rs = row_ok ? __ldg(g.sx + row) : 1.f;
          const int64_t off = static_cast<int64_t>(split) * g.split_stride + static_cast<int64_t>(row) * g.ldo + n0;
          const bool vec_ok = (g.ldo & 7) == 0 && (g.split_stride & 3) == 0;      // n0 and the 16-column steps keep the alignment
#pragma unroll 1
          for (int c = 0; c < ncols; c += 16) {
            uint32_t r[16];
            tmem_ld16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c, r);
            tmem_ld_wait();
            if (row_ok) {
              float v[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                v[e] = __uint_as_float(r[e]);
                if constexpr (FP8) v[e] *= rs * __ldg(g.sw + min(n0 + c + e, g.N - 1));
              }
              if constexpr (EPI == kEpiPartialF32) {
                float* o = reinterpret_cast<float*>(g.out) + off + c;
                if (vec_ok && c + 16 <= ncols) {
#pragma unroll
                  for (int e = 0; e < 16; e += 4) *reinterpret_cast<float4*>(o + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
                } else {
#pragma unroll
                  for (int e = 0; e < 16; ++e)
                    if (c + e < ncols) o[e] = v[e];
                }
              } else {
                bf16_t* o = reinterpret_cast<bf16_t*>(g.out) + off + c;
                if (vec_ok && c + 16 <= ncols) {
#pragma unroll
                  for (int e = 0; e < 16; e += 8)
                    *reinterpret_cast<uint4*>(o + e) = make_uint4(pack2(v[e], v[e + 1]), pack2(v[e + 2], v[e + 3]), pack2(v[e + 4], v[e + 5]),
                                                                  pack2(v[e + 6], v[e + 7]));
                } else {
#pragma unroll
                  for (int e = 0; e < 16; ++e)
                    if (c + e < ncols) o[e] = f2bf(v[e]);
                }
              }
            }
            __syncwarp();
          }
        }
      }
      tc_fence_before();
    }
  }

  __syncthreads();
  if (abort_flag[0]) {
    if (threadIdx.x == 0) report_status(g.status, OJB_DEV_WAIT_TIMEOUT);
    for (int i = 0; i < 200; ++i) __nanosleep(1000);      // copies that were already issued land before the CTA leaves
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, g.tmem_cols);
  }
}

template <int EPI, bool FP8, bool WSIDE>
int launch_skinny(int bn, const void* x, const void* w, void* out, int64_t M, int64_t N, int64_t K, int splits, int64_t ldo,
                  int32_t* status, cudaStream_t stream, const float* sx, const float* sw) {
  static int smem_set[kMaxDevices] = {};
  auto kern = gemm_skinny_kernel<EPI, FP8, WSIDE>;
  if (!raise_smem_limit(kern, static_cast<int>(kSkinnySmem - 2048), smem_set)) return OJB_ERR_LAUNCH;      // 2 KB: the static part
  SkinnyArgs g{};
  g.M = static_cast<int>(M);
  g.N = static_cast<int>(N);
  g.BN = bn;
  g.x_rows = static_cast<int>(WSIDE ? ceil_div(M, 16) * 16 : ceil_div(M, 8) * 8);
  g.splits = splits;
  g.kb_total = static_cast<int>(ceil_div(K, FP8 ? 128 : kBK));
  g.kb_per_split = static_cast<int>(ceil_div(g.kb_total, splits));
  if (static_cast<int64_t>(splits - 1) * g.kb_per_split >= g.kb_total) return OJB_ERR_ARG;      // empty K range
  // k-blocks per stage: as many as leave at least six stages, up to four
  const uint32_t kb_bytes = static_cast<uint32_t>(g.x_rows + bn) * 128;
  const uint32_t budget = static_cast<uint32_t>(kSkinnySmem - 2048 - 1024);
  g.nk = 4;
  while (g.nk > 1 && (g.nk * kb_bytes * 6 > budget || g.nk > g.kb_per_split)) --g.nk;
  g.stage_bytes = g.nk * kb_bytes;
  // the A operand of the last k-block may run on behind the last stage
  const uint32_t reach = WSIDE ? g.stage_bytes + (kBM - bn) * 128u : (g.nk - 1) * static_cast<uint32_t>(g.x_rows) * 128 + kBM * 128u;
  const uint32_t over = reach > g.stage_bytes ? reach - g.stage_bytes : 0u;
  g.stages = static_cast<int>((budget - over) / g.stage_bytes);
  if (g.stages > kSkinnyMaxStages) g.stages = kSkinnyMaxStages;
  g.tmem_cols = 32;
  while (static_cast<int>(g.tmem_cols) < (WSIDE ? g.x_rows : bn)) g.tmem_cols *= 2;
  g.out = out;
  g.ldo = ldo;
  g.split_stride = EPI == kEpiPartialF32 ? M * N : 0;
  g.status = status;
  g.wait_ms = gemm_wait_limit_ms();
  g.drop_copy = gemm_drop_copy();
  g.sx = sx;
  g.sw = sw;
  CUtensorMap map_x, map_w;
  int rc = make_kblock_map(&map_x, x, FP8 ? 1 : 2, M, K, g.x_rows, g.nk);
  if (rc == OJB_OK) rc = make_kblock_map(&map_w, w, FP8 ? 1 : 2, N, K, bn, g.nk);
  if (rc != OJB_OK) return rc;
  const size_t smem = 1024 + static_cast<size_t>(g.stages) * g.stage_bytes + over;
  launch_kernel(kern, dim3(static_cast<unsigned>(ceil_div(N, bn) * splits)), dim3(kSkinnyThreads), smem, stream, map_x, map_w, g);
  return launch_status(cudaGetLastError());
}

}  // namespace

// bn = 0: the narrowest multiple of 16 (at most 128) with which the tiles times the K ranges fill the SMs at most once
int gemm_skinny_launch(int epi, int bn, const void* x, const void* w, void* out, int64_t M, int64_t N, int64_t K, int splits,
                       int64_t ldo, int32_t* status, cudaStream_t stream, const float* sx, const float* sw) {
  if (M > kSkinnyRows || K % (sx != nullptr ? 128 : kBK) != 0 || (epi != kEpiBf16 && epi != kEpiPartialF32)) return OJB_ERR_LIMIT;
  if (bn == 0) bn = skinny_bn(N, splits);
  if (bn < 16 || bn > 128 || bn % 16) return OJB_ERR_ARG;
  const bool wside = ceil_div(M, 16) * 16 < bn;
  auto pick = [&](auto fp8, auto side) {
    constexpr bool kFp8 = decltype(fp8)::value, kSide = decltype(side)::value;
    return epi == kEpiBf16 ? launch_skinny<kEpiBf16, kFp8, kSide>(bn, x, w, out, M, N, K, splits, ldo, status, stream, sx, sw)
                           : launch_skinny<kEpiPartialF32, kFp8, kSide>(bn, x, w, out, M, N, K, splits, ldo, status, stream, sx, sw);
  };
  using std::false_type;
  using std::true_type;
  if (sx != nullptr) return wside ? pick(true_type{}, true_type{}) : pick(true_type{}, false_type{});
  return wside ? pick(false_type{}, true_type{}) : pick(false_type{}, false_type{});
}

}  // namespace ojb
