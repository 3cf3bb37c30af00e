// Prefix-tree GQA attention for many rows (head dim 256), tcgen05: one pass over the keys with a running maximum.
//
// tree_attn_tc.cu serves short trees: 16 query rows x all heads of a kv head per CTA, so that a few hundred rows fill the GPU, two
// passes over the keys, any two visible 64-key blocks to a product. On long roots that costs Q K^T twice, a quarter of every
// product's rows (96 of 128) and 192 KB of keys and values per 16 rows. Here a CTA takes 128 operand rows (64 query rows x 2 heads,
// or 128 x 1 where the heads of a kv head are odd in number), 128-key blocks, and goes over them once:
//
//   S = Q K^T       128 x 128 x 256 into one of two 128-column buffers of tensor memory, a block ahead of the softmax
//   softmax         eight warps, two threads per row (64 keys each): block maximum, exchanged with the other thread of the row; the
//                   reference m that the exponents are taken against moves only when the maximum has grown by more than
//                   2^8 since (P = exp2((s - m) scale log2 e) then stays below 256 and the final division is exact either way);
//                   moving it rescales the row of O in tensor memory
//   O += P V        128 x 256 x 128, P as bf16 in tensor memory over the scores it came from: the product reads it there, so it
//                   never passes through shared memory and the softmax waits for no product (except to rescale O)
//
// Shared memory: Q 64 KB and a ring of four 32 KB entries through which K (128 keys x 128 dims at a time) and V (256 dims x 64 keys at a
// time) stream in the order in which the products consume them, K of the next block before V of this one. Each entry costs
// the issuing warp a wait and a commit: seven 16 KB entries and P in shared memory took a third longer. 16 512 rows: 2.5 ms, 1360
// blocks per SM of 1.85 us each, of which the tensor pipe needs 1.1 (48 % of the time busy at 4192 rows); the rest is the arrival of
// K and V and the chain from scores to P.
// Roles: warps 0-7 softmax and epilogue, warp 8 TMA producer, warp 9 MMA issuer; every wait bounded.
#include "tree_attn_rows.cuh"

namespace ojb {
namespace {

constexpr int kLD = 256;                       // head dim
constexpr int kLKeys = 128;                    // keys per block
constexpr int kLThreads = 320;
constexpr int kLSlots = 4;
constexpr uint32_t kLTile = 128 * 128;         // 16 KB: 128 rows of 128 bytes
constexpr uint32_t kLSlot = 2 * kLTile;
constexpr uint32_t kLQ = 4 * kLTile;
constexpr uint32_t kLColO = 0, kLColS = 256;
constexpr int kLPitch = kLD * 2 + 16;          // row of the output staging tile (over Q and the start of the ring)
constexpr int kLMaxBlocks = 1024;              // 131 072 keys
constexpr float kLStale = 8.0f;                // how far (log2) the maximum may run ahead of m
enum { kLBarQ = 0, kLBarFull = 1, kLBarEmpty = kLBarFull + kLSlots, kLBarSFull = kLBarEmpty + kLSlots, kLBarPFull = kLBarSFull + 2,
       kLBarRest, kLBarO, kLBarX, kLNumBars = kLBarX + 4 };
constexpr size_t kLSmem = 1024 + kLQ + kLSlots * kLSlot + kLNumBars * 8 + 16 + (kLMaxBlocks / 32 + 1) * 4 + 2 * 2 * 128 * 4;
static_assert(kLSmem <= 227 * 1024, "shared memory");
static_assert(128 * kLPitch <= static_cast<int>(kLQ + kLSlot), "output staging");

struct LongArgs {
  const bf16_t* gate;
  const int32_t* krange;
  bf16_t* y;
  int32_t* status;
  int N, NQ, HQ, HKV, G, hp, R;      // hp heads x R query rows = 128
  float scale_log2e;
  int wait_ms, drop_copy;
  const int64_t* q_rows;
  int64_t gate_ld;
  int gate_hs;
  const bf16_t *qt, *kt, *vt_t;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// tcgen05.mma with A in tensor memory: row = lane, two bf16 of K per column
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__global__ void __launch_bounds__(kLThreads, 1)
tree_attn_long_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_vt, LongArgs g) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* Qs = smem;
  uint8_t* Rg = Qs + kLQ;
  uint64_t* bars = reinterpret_cast<uint64_t*>(Rg + kLSlots * kLSlot);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kLNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);      // [0] give-up flag, [1] wait limit in ms
  uint32_t* seen = tmem_slot + 4;                                                  // one bit per key block
  float* xch = reinterpret_cast<float*>(seen + kLMaxBlocks / 32 + 1);              // [block parity][half][row]
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * static_cast<uint32_t>(i); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int groups = g.G / g.hp;                                // CTAs per kv head and block of query rows
  const int kvh = blockIdx.x / groups, hq0 = kvh * g.G + (blockIdx.x - kvh * groups) * g.hp;
  const int r0 = (gridDim.y - 1 - blockIdx.y) * g.R;            // the last rows, which see most keys, first
  const int N = g.N;

  if (tid == 0) {
    for (int i = 0; i < kLNumBars; ++i) mbar_init(bar(i), 1);
    mbar_init(bar(kLBarPFull), 8);
    for (int w = 0; w < 4; ++w) mbar_init(bar(kLBarX + w), 2);
    abort_flag[0] = 0;
    abort_flag[1] = g.wait_ms;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_vt) : "memory");
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  const int nblk = (N + kLKeys - 1) / kLKeys, nwords = (nblk + 31) / 32;
  for (int i = tid; i <= nwords; i += kLThreads) seen[i] = 0u;      // (the word behind the last one ends every search)
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp == 8 && lane == 0) {
    mbar_expect_tx(bar(kLBarQ), kLQ);
    for (int w = 0; w < g.hp; ++w)
      for (int c = 0; c < 4; ++c)
        tma_load_2d(smem_u32(Qs) + c * kLTile + w * g.R * 128, &map_q, bar(kLBarQ), c * 64, (hq0 + w) * g.NQ + r0);
  }
  // blocks that at least one of the query rows sees: thread = (row, range)
  for (int i = tid; i < g.R * 3; i += kLThreads) {
    const int r = r0 + i / 3, which = i % 3;
    if (r < g.NQ) {
      const int32_t* q = g.krange + (g.q_rows ? nearest_row(g.q_rows[r], N) : r) * 8;      // (e0, a1, e1, a2, e2, a0)
      const int lo = max(which == 0 ? q[5] : which == 1 ? q[1] : q[3], 0), hi = min(which == 0 ? q[0] : which == 1 ? q[2] : q[4], N);
      if (lo < hi) {
        const int b0 = lo / kLKeys, b1 = (hi - 1) / kLKeys;
        for (int w = b0 >> 5; w <= b1 >> 5; ++w) {
          const uint32_t m = (w == b1 >> 5 ? 0xffffffffu >> (31 - (b1 & 31)) : 0xffffffffu) & (w == b0 >> 5 ? 0xffffffffu << (b0 & 31) : 0xffffffffu);
          if ((seen[w] & m) != m) atomicOr(&seen[w], m);
        }
      }
    }
  }
  __syncthreads();
  int T = 0;
  for (int w = 0; w < nwords; ++w) T += __popc(seen[w]);
  // the first visible block at or after b (b < nblk or none is left)
  auto next_block = [&](int b) {
    int w = b >> 5;
    uint32_t m = seen[w] & (0xffffffffu << (b & 31));
    while (m == 0u && w < nwords) m = seen[++w];
    return w * 32 + __ffs(m) - 1;
  };

  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (T > 0) {
      const bool one = elect_one();
      int use = 0;
      bool ok = true;
      auto slot = [&](uint32_t& dst, uint32_t& fb) {
        const int s = use % kLSlots;
        if (!mbar_wait_warp(bar(kLBarEmpty + s), ((use / kLSlots) & 1) ^ 1, abort_flag)) return false;
        ++use;
        dst = smem_u32(Rg) + s * kLSlot;
        fb = bar(kLBarFull + s);
        if (one) mbar_expect_tx(fb, kLSlot);
        return true;
      };
      auto keys = [&](int kb) {
        for (int c = 0; c < 2 && ok; ++c) {      // 128 dims
          uint32_t dst, fb;
          if (!(ok = slot(dst, fb))) break;
          if (one && !(g.drop_copy && use == 2))      // tests only: the announced bytes of the second entry never arrive
            tma_load_3d(dst, &map_k, fb, 0, kvh * N + kb * kLKeys, 2 * c);
        }
      };
      auto values = [&](int kb) {
        for (int c = 0; c < 2 && ok; ++c) {      // 64 keys
          uint32_t dst, fb;
          if (!(ok = slot(dst, fb))) break;
          if (one) tma_load_2d(dst, &map_vt, fb, kb * kLKeys + c * 64, kvh * kLD);
        }
      };
      int kb = next_block(0);
      keys(kb);
      for (int j = 0; j < T && ok; ++j) {
        int nb = kb;
        if (j + 1 < T) {
          nb = next_block(kb + 1);
          keys(nb);
        }
        values(kb);
        kb = nb;
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    if (T > 0) {
      const bool one = elect_one();
      constexpr uint32_t idesc_s = umma_idesc(kLKeys), idesc_o = umma_idesc(kLD);
      int use = 0;
      bool ok = mbar_wait_warp(bar(kLBarQ), 0, abort_flag);
      // (S of block j goes where S and P of block j - 2 were: its scores have been read, or P V (j - 2) would not have been issued,
      // and the tensor pipe runs the products in the order of their issue)
      auto qk = [&](int j) {
        const uint32_t acc = tmem_base + kLColS + static_cast<uint32_t>(j & 1) * kLKeys;
        for (int c = 0; c < 2; ++c, ++use) {
          const int s = use % kLSlots;
          if (!mbar_wait_warp(bar(kLBarFull + s), (use / kLSlots) & 1, abort_flag)) return false;
          tc_fence_after();
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const uint64_t qd = smem_desc_sw128(smem_u32(Qs) + (2 * c + t) * kLTile), kd = smem_desc_sw128(smem_u32(Rg) + s * kLSlot + t * kLTile);
#pragma unroll
            for (int k = 0; k < 4; ++k) if (one) umma_bf16(acc, qd + 2 * k, kd + 2 * k, idesc_s, (c > 0 || t > 0 || k > 0) ? 1u : 0u);
          }
          if (one) umma_commit(bar(kLBarEmpty + s));
        }
        if (one) umma_commit(bar(kLBarSFull + (j & 1)));
        return true;
      };
      auto pv = [&](int j) {
        if (!mbar_wait_warp(bar(kLBarPFull), j & 1, abort_flag)) return false;
        for (int c = 0; c < 2; ++c, ++use) {
          const int s = use % kLSlots;
          if (!mbar_wait_warp(bar(kLBarFull + s), (use / kLSlots) & 1, abort_flag)) return false;
          tc_fence_after();
          const uint32_t p = tmem_base + kLColS + static_cast<uint32_t>((j & 1) * kLKeys + c * 32);      // two keys per column
          const uint64_t vd = smem_desc_sw128(smem_u32(Rg) + s * kLSlot);
#pragma unroll
          for (int k = 0; k < 4; ++k) if (one) umma_bf16_ts(tmem_base + kLColO, p + 8 * k, vd + 2 * k, idesc_o, (j > 0 || c > 0 || k > 0) ? 1u : 0u);
          if (one) umma_commit(bar(kLBarEmpty + s));
        }
        if (one) umma_commit(bar(kLBarRest));
        return true;
      };
      if (ok) ok = qk(0);
      for (int j = 0; j < T && ok; ++j) {
        if (j + 1 < T) ok = qk(j + 1);
        if (ok) ok = pv(j);
      }
      if (ok && one) umma_commit(bar(kLBarO));
    }
  } else {
    // ------------------------------------------------------------------ softmax: warps w and w + 4 share 32 rows, 64 keys each
    const int half = warp >> 2, quarter = warp & 3, my = quarter * 32 + lane;
    const int qr = r0 + my % g.R;
    int lo0 = 0, hi0 = 0, lo1 = 0, hi1 = 0, lo2 = 0, hi2 = 0;
    if (qr < g.NQ) {
      const int32_t* q = g.krange + (g.q_rows ? nearest_row(g.q_rows[qr], N) : qr) * 8;
      hi0 = q[0]; lo1 = q[1]; hi1 = q[2]; lo2 = q[3]; hi2 = q[4]; lo0 = q[5];
    }
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const float c = g.scale_log2e;
    float m = -INFINITY, l = 0.f;      // reference of the exponents (raw score), sum of this thread's P
    bool ok = true;
    int kb = T > 0 ? next_block(0) : 0;
    for (int j = 0; j < T && ok; ++j) {
      const int sb = j & 1;
      if (!mbar_wait_warp(bar(kLBarSFull + sb), (j >> 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      uint32_t s[2][32];
      const uint32_t ts = tmem_base + lanes + kLColS + static_cast<uint32_t>(sb * kLKeys + half * 64);
      tmem_ld32(ts, s[0]);
      tmem_ld32(ts + 32, s[1]);
      tmem_ld_wait();
      const int k0 = kb * kLKeys + half * 64;
      const bool whole = (lo0 <= k0 && k0 + 64 <= hi0) || (lo1 <= k0 && k0 + 64 <= hi1) || (lo2 <= k0 && k0 + 64 <= hi2);
      if (!__all_sync(0xffffffffu, whole)) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int w = k0 / 32 + i;
          const uint32_t bits = range_bits(lo0, hi0, w) | range_bits(lo1, hi1, w) | range_bits(lo2, hi2, w);
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (!((bits >> e) & 1u)) s[i][e] = 0xff800000u;      // -infinity
        }
      }
      float mx = -INFINITY;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 32; ++e) mx = fmaxf(mx, __uint_as_float(s[i][e]));
      float* x = xch + (j & 1) * 256;
      x[half * 128 + my] = mx;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kLBarX + quarter));
      if (!mbar_wait_warp(bar(kLBarX + quarter), j & 1, abort_flag)) { ok = false; break; }
      mx = fmaxf(mx, x[(half ^ 1) * 128 + my]);
      const bool move = mx > m && (m == -INFINITY || (mx - m) * c > kLStale);
      const float f = move && m != -INFINITY ? exp2f_fast((m - mx) * c) : 1.f;      // (a row that has seen no key has O = 0 and l = 0)
      if (move) m = mx;
      const float mc = m == -INFINITY ? 0.f : m * c;
      l *= f;
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float p0 = exp2f_fast(fmaf(__uint_as_float(s[i][e]), c, -mc));
          const float p1 = exp2f_fast(fmaf(__uint_as_float(s[i][e + 1]), c, -mc));
          l += p0 + p1;
          pk[i * 16 + (e >> 1)] = pack2(p0, p1);
        }
      if (__any_sync(0xffffffffu, f != 1.f)) {
        // P V of the block before has left O at rest, that of this block is not issued before P is there
        if (!mbar_wait_warp(bar(kLBarRest), (j & 1) ^ 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
          uint32_t o[16];
          const uint32_t to = tmem_base + lanes + kLColO + static_cast<uint32_t>(half * 128 + i * 16);
          tmem_ld16(to, o);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
          tmem_st16(to, o);
        }
      }
      // over the scores, which both halves have read (they have exchanged their maxima since)
      tmem_st32(tmem_base + lanes + kLColS + static_cast<uint32_t>(sb * kLKeys + half * 32), pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kLBarPFull));
      if (j + 1 < T) kb = next_block(kb + 1);
    }
    // ---- att = bf16(O / l) into the staging tile (which the Q rows must not be on their way to any more)
    if (T == 0) ok = mbar_wait_warp(bar(kLBarQ), 0, abort_flag);
    if (T > 0 && ok) {
      float* x = xch + (T & 1) * 256;
      x[half * 128 + my] = l;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kLBarX + quarter));
      ok = mbar_wait_warp(bar(kLBarX + quarter), T & 1, abort_flag);
      l += x[(half ^ 1) * 128 + my];
      if (ok) ok = mbar_wait_warp(bar(kLBarO), 0, abort_flag);
    }
    if (ok) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      uint8_t* srow = smem + my * kLPitch;
      float odd = 0.f;                   // not-a-number if a value of O is not finite
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        const int col = half * 4 + i;
        uint32_t o[32];
        if (T > 0) {
          tmem_ld32(tmem_base + lanes + kLColO + col * 32, o);
          tmem_ld_wait();
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          float a[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            a[e] = l > 0.f ? __uint_as_float(o[v * 8 + e]) * inv : 0.f;      // no visible key: zeros
            odd = fmaf(a[e], 0.f, odd);
          }
          *reinterpret_cast<uint4*>(srow + col * 64 + v * 16) = pack8(a);
        }
      }
      for (uint32_t again = __ballot_sync(0xffffffffu, odd != odd); again != 0u; again &= again - 1u) {
        const int src = __ffs(again) - 1, row = quarter * 32 + src;
        auto of = [&](auto x) { return __shfl_sync(0xffffffffu, x, src); };
        const float4 a = row_over_its_keys(
            g.qt + (static_cast<int64_t>(hq0 + row / g.R) * g.NQ + r0 + row % g.R) * kLD, g.kt + static_cast<int64_t>(kvh) * N * kLD,
            g.vt_t + static_cast<int64_t>(kvh) * kLD * N, N, half * 128, of(lo0), of(hi0), of(lo1), of(hi1), of(lo2), of(hi2), c, of(m) * c, of(inv));
        *reinterpret_cast<uint2*>(smem + row * kLPitch + half * 256 + lane * 8) = make_uint2(pack2(a.x, a.y), pack2(a.z, a.w));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // ---- y = bf16(att * sigmoid(gate)), whole 512-byte rows
  if (!abort_flag[0]) {
    for (int i = tid; i < 128 * (kLD / 8); i += kLThreads) {
      const int row = i >> 5, piece = i & 31, r = r0 + row % g.R, h = hq0 + row / g.R;
      if (r < g.NQ) {
        float gv[8], a[8], out[8];
        unpack8(*reinterpret_cast<const uint4*>(g.gate + r * g.gate_ld + static_cast<int64_t>(h) * g.gate_hs + piece * 8), gv);
        unpack8(*reinterpret_cast<const uint4*>(smem + row * kLPitch + piece * 16), a);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float t;
          asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * gv[e]));
          out[e] = a[e] * fmaf(0.5f, t, 0.5f);
        }
        *reinterpret_cast<uint4*>(g.y + (static_cast<int64_t>(r) * g.HQ + h) * kLD + piece * 8) = pack8(out);
      }
    }
  }
  __syncthreads();
  if (abort_flag[0]) {
    if (tid == 0) report_status(g.status, OJB_DEV_WAIT_TIMEOUT);
    for (int i = 0; i < 200; ++i) __nanosleep(1000);       // copies that were already issued land before the CTA leaves
    __syncthreads();
  }
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

int tree_attn_long_launch(const void* qt, int64_t NQ, const int64_t* q_rows, const void* kt, const void* vt_t, int64_t N, const void* gate,
                          int64_t gate_ld, int64_t gate_hs, const int32_t* krange, void* y, int64_t HQ, int64_t HKV, float scale,
                          int32_t* status, cudaStream_t st) {
  LongArgs a{};
  a.G = static_cast<int>(HQ / HKV);
  a.hp = a.G % 2 == 0 ? 2 : 1;
  a.R = 128 / a.hp;
  CUtensorMap map_q, map_k, map_vt;
  int rc = make_map(&map_q, qt, HQ * NQ, kLD, a.R);
  if (rc == OJB_OK) rc = make_kblock_map(&map_k, kt, 2, HKV * N, kLD, kLKeys, 2);
  if (rc == OJB_OK) rc = make_map(&map_vt, vt_t, HKV * kLD, N, kLD);
  if (rc != OJB_OK) return rc;
  static int smem_set[kMaxDevices] = {};
  if (!raise_smem_limit(tree_attn_long_kernel, static_cast<int>(kLSmem), smem_set)) return OJB_ERR_LAUNCH;
  a.gate = static_cast<const bf16_t*>(gate);
  a.krange = krange;
  a.y = static_cast<bf16_t*>(y);
  a.status = status;
  a.N = static_cast<int>(N);
  a.NQ = static_cast<int>(NQ);
  a.HQ = static_cast<int>(HQ);
  a.HKV = static_cast<int>(HKV);
  a.scale_log2e = scale * 1.4426950408889634f;
  a.wait_ms = gemm_wait_limit_ms();
  a.drop_copy = gemm_drop_copy();
  a.q_rows = q_rows;
  a.gate_ld = gate_ld;
  a.gate_hs = static_cast<int>(gate_hs);
  a.qt = static_cast<const bf16_t*>(qt);
  a.kt = static_cast<const bf16_t*>(kt);
  a.vt_t = static_cast<const bf16_t*>(vt_t);
  launch_kernel(tree_attn_long_kernel, dim3(static_cast<unsigned>(HKV * (a.G / a.hp)), static_cast<unsigned>(ceil_div(NQ, a.R))),
                dim3(kLThreads), kLSmem, st, map_q, map_k, map_vt, a);
  return launch_status(cudaGetLastError());
}

}  // namespace ojb
