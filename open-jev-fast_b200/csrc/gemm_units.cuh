// Work decomposition shared by the block GEMM kernels (gemm_block256.cu: one CTA per unit; gemm_pair256.cu: one CTA pair
// per unit): block units of 256 rows of x times BN rows of w, swapped-operand tail units of 256 rows of w times up to 256
// rows of x, optional K ranges, and the order in which the units are dealt out.
#pragma once
// Probe builds (-DOJB_GEMM_PROBES, never the shipped library) can repeat the MMAs of a stage, cap the pipeline depth and
// skip parts of the epilogue to separate tensor-pipe, copy and store costs; in the shipped build these read as constants
// and the code behind them is compiled out.
#ifdef OJB_GEMM_PROBES
#define OJB_PROBE_REPEAT(g) ((g).mma_repeat)
#define OJB_PROBE_DBG(g) ((g).dbg)
#else
#define OJB_PROBE_REPEAT(g) 1
#define OJB_PROBE_DBG(g) 0
#endif
#include "gemm_common.cuh"
#include <cstring>
#include <mutex>

namespace ojb {
namespace {

constexpr int kBlockM = 256;       // rows of x per block unit

struct GemmArgs {
  int M, N, K;
  int BN;          // rows of w per block unit: multiple of 16, <= 256
  int n_xblk;      // 256-row blocks of x served by block units
  int tail_rows;   // rows of x served by tail units, starting at row n_xblk * 256 (0 = none)
  int tail_box;    // rows of x per tail unit: multiple of 16, <= 256 = UMMA N of the tail units
  int n_xchunk;    // tail units per w tile and k-split: the tail rows are cut into n_xchunk chunks of tail_box rows
  int n_wtile;     // ceil(N / BN)
  int n_wtile256;  // ceil(N / 256)
  int splits, kb_per_split, kb_total;   // in k-blocks of 64 columns
  int stages;
  uint32_t stage_bytes;
  void* out;
  int64_t ldo;           // leading dimension of out in elements
  int64_t split_stride;  // elements between split planes (fp32 partials)
  int32_t* status;
  int wait_ms;                 // limit of every mbarrier wait of the kernel, milliseconds
  unsigned long long* trace;   // null, or [0] = record counter followed by records of 4 words (see ojb_gemm_set_trace)
  int trace_cap;
  int tail_sub;                // bytes of a tail sub-stage (128 rows of w + the x rows), 0 = one k-block per stage
  int tma_out;                 // the block epilogue stores through shared-memory tiles and bulk tensor stores
  int pair_rows;               // block kernel, SwiGLU: rows of x below it take their SiLU in pairs (silu2_f), the others by silu_f
  int dbg;                     // probe builds only (see below); 0 otherwise
  int mma_repeat;              // probe builds only; 1 otherwise
  // CTA-pair kernel, swapped-operand units: the tail_box accumulator columns (= rows of x) of a unit are produced by
  // n_chunk MMAs per k-step of chunk_w columns each (the last one narrower), so one pass over 256 rows of w serves up to
  // 512 rows of x; w_split64: the 128 rows of w of a CTA are fetched as rows [64r, 64r+64) and [128+64r, 128+64r+64) of the
  // tile (gate and up rows of the same 64 outputs of a SwiGLU weight interleaved in blocks of 128 rows).
  int n_chunk, chunk_w, w_split64;
  // e4m3 operands (block kernel): fp32 scale per row of x and per row of w, applied to the accumulator in the epilogue
  const float* sx;
  const float* sw;
  int tail_tma;                // block kernel: swapped-operand units store through [16][32] shared-memory tiles and bulk tensor stores
  int band_xblk;               // 0, or the x blocks of a band: all units of a band come before those of the next (see decode_unit)
};

struct Unit {
  bool tail;
  int xb, split, wt, kb0, kb1;
  int xc;   // x chunk of a tail unit
};

// Units are ordered by the w rows they read: w tile j contributes its block units (x-block fastest, then k-split) followed
// by the tail units that start inside it, so a tail unit finds its w rows in L2 instead of streaming them from HBM again.
// group_begin(j) = position of the first unit of tile j; tails_before(j) = tail tiles (256 w rows each) that start before
// row j * BN.
// When x is larger than the L2 keeps (tens of thousands of rows), that order would stream all of x from HBM once per w tile:
// the x blocks are then cut into bands of band_xblk blocks, each band small enough to stay in L2, and the whole order above
// runs band after band (w is streamed once per band instead); the tail units belong to the last band.
__host__ __device__ __forceinline__ int tails_before(const GemmArgs& g, int j, bool tails) {
  if (!tails) return 0;
  const int t = (j * g.BN + 255) / 256;
  return t < g.n_wtile256 ? t : g.n_wtile256;
}
__host__ __device__ __forceinline__ int group_begin(const GemmArgs& g, int j, int nx, bool tails) {
  return (j * nx + tails_before(g, j, tails) * g.n_xchunk) * g.splits;
}

// (also compiled for the host: ojb_gemm_unit_order lists the order for the tests)
__host__ __device__ __forceinline__ Unit decode_unit(const GemmArgs& g, int unit, int total_block) {
  (void)total_block;
  Unit u;
  int xb_base = 0, nx = g.n_xblk;
  bool tails = g.tail_rows > 0;
  if (g.band_xblk > 0) {
    const int full = g.band_xblk * g.n_wtile * g.splits;          // units of a band that is not the last one
    const int n_bands = (g.n_xblk + g.band_xblk - 1) / g.band_xblk;
    int b = unit / full;
    if (b > n_bands - 1) b = n_bands - 1;
    unit -= b * full;
    xb_base = b * g.band_xblk;
    nx = g.band_xblk < g.n_xblk - xb_base ? g.band_xblk : g.n_xblk - xb_base;
    tails = tails && b == n_bands - 1;
  }
  const int nb = nx * g.splits;
  int j = static_cast<int>(unit / (nb + g.splits * g.n_xchunk * (tails ? g.BN / 256.0f : 0.0f) + 1e-6f));
  if (j > g.n_wtile - 1) j = g.n_wtile - 1;
  while (j > 0 && group_begin(g, j, nx, tails) > unit) --j;
  while (j + 1 < g.n_wtile && group_begin(g, j + 1, nx, tails) <= unit) ++j;
  const int off = unit - group_begin(g, j, nx, tails);
  u.tail = off >= nb;
  if (!u.tail) {
    u.xb = xb_base + off % nx;
    u.split = off / nx;
    u.wt = j;
    u.xc = 0;
  } else {
    const int o2 = off - nb;
    u.xb = g.n_xblk;
    u.xc = o2 % g.n_xchunk;                       // x chunk fastest: the chunks of one w tile run side by side
    u.split = (o2 / g.n_xchunk) % g.splits;
    u.wt = tails_before(g, j, tails) + o2 / (g.n_xchunk * g.splits);
  }
  u.kb0 = u.split * g.kb_per_split;
  u.kb1 = u.kb0 + g.kb_per_split < g.kb_total ? u.kb0 + g.kb_per_split : g.kb_total;
  return u;
}

// x blocks per band (0: no bands) for n_xblk blocks of xblk_bytes. x beyond what the L2 keeps beside the streaming weight (64 MB) and
// at least 24 x blocks (with fewer, the CTAs that run at the same time already cover several weight tiles per x block, and x is
// re-read only a few times): bands of about 16 x blocks, equal in size, so that the units under way at any time share both their x
// blocks and their w tiles about twelve times (bands of a fixed 40 MB were 4 blocks at K = 17 408). 16 672 rows, blocks per band
// 8 / 11 / 16 / 22 / 33: gate/up 4345 / 4329 / 4275 / 4412 / 4554 us, [12352, 5120] 1538 / 1520 / 1496 / 1556 / 1593, [5120, 17408]
// 2288 / 2283 / 2319 / 2308 / 2434. For measurements OJB_GEMM_BAND_BLOCKS sets the blocks of a band, OJB_GEMM_BAND_MB its size in MB
// (at least two blocks); 0 switches bands off. With both set the blocks count.
inline int band_blocks(int n_xblk, int64_t xblk_bytes) {
  static const char* const blocks_env = getenv("OJB_GEMM_BAND_BLOCKS");
  static const char* const mb_env = getenv("OJB_GEMM_BAND_MB");
  int64_t per = 16;
  if (blocks_env != nullptr) {
    per = atoi(blocks_env);
  } else if (mb_env != nullptr) {
    const int64_t mb = atoi(mb_env);
    per = mb <= 0 ? 0 : (mb << 20) / xblk_bytes;
    if (mb > 0 && per < 2) per = 2;
  }
  if (per <= 0 || n_xblk < 24 || n_xblk * xblk_bytes <= (64ll << 20)) return 0;
  return static_cast<int>(ceil_div(n_xblk, ceil_div(n_xblk, per)));
}

// ---- Cost model (host). Times are SM clocks; the constants come from unit timelines measured on B200 (ojb_gemm_set_trace):
// the main loops are bound by shared-memory bandwidth (128 bytes per clock per SM shared between the TMA fill of a stage
// and the operand reads of its MMAs), an MMA with M = 128 never takes less than 64 clocks, a k-block of a
// swapped-operand unit takes its wait, commit and eight MMAs at least 600 clocks, and the epilogue of a block unit costs about 19
// (bf16), 33 (fp32) or 40 (SwiGLU) clocks per accumulator column.
// The model as the K ranges of 8-bit products are chosen by (see model_kernel): fp32 partials, every tile width alike.
constexpr int kEpi8BitRanges = 3;

struct UnitCost {
  double block_kb, block_epi, tail_kb, tail_epi;
};
inline UnitCost unit_cost(int bn, int tail_box, int epi) {
  UnitCost c;
  const double smem = 512.0 + 3.0 * bn, mma = 4.0 * bn;
  c.block_kb = smem > mma ? smem : mma;
  // tiles of whole 128-byte pieces leave by bulk stores, others by the threads' own, three times as long (before the model knew,
  // it took 208-wide tiles for fp32 results: [5120, 4096] at 4160 rows 184 us, with 224 149 us)
  const bool bulk = epi == kEpi8BitRanges || bn % (epi == kEpiPartialF32 ? 32 : 64) == 0;
  const bool f32 = epi == kEpiPartialF32 || epi == kEpi8BitRanges;
  c.block_epi = 900.0 + bn * (f32 ? (bulk ? 33.0 : 115.0) : (epi == kEpiSwiglu ? 40.0 : (bulk ? 19.0 : 55.0)));
  const double tsm = 512.0 + 3.0 * tail_box;
  const double floor = epi == kEpi8BitRanges ? 1200.0 : 600.0;
  c.tail_kb = tsm > floor ? tsm : floor;
  c.tail_epi = 3200.0 + 24.0 * tail_box;
  return c;
}

// Never more than block_kernel_clocks of the same arguments: the mean load of the workers. A width search passes over what cannot win by
// this instead of dealing its units out.
inline double block_kernel_floor(int64_t N, int bn, int n_xblk, int tail_box, int n_xchunk, bool has_tail, int splits, int kb_total,
                                 int workers, int epi) {
  const UnitCost c = unit_cost(bn, tail_box, epi);
  const int64_t blocks = n_xblk * ceil_div(N, bn), tails = has_tail ? n_xchunk * ceil_div(N, 256) : 0;      // per K range
  const int64_t units = (blocks + tails) * splits;
  if (units <= 0) return 0.0;
  const double all = static_cast<double>(blocks) * (kb_total * c.block_kb + splits * c.block_epi) +
                     static_cast<double>(tails) * (kb_total * c.tail_kb + splits * c.tail_epi);
  return static_cast<double>(static_cast<int64_t>(all / static_cast<double>(units < workers ? units : workers))) + 5000.0;
}

// Longest per-worker sum when the units of the block kernels (order of decode_unit) are dealt round-robin to `workers`
// CTAs (or CTA pairs). n_xblk == 0: swapped-operand units only.
inline double block_kernel_clocks(int64_t N, int bn, int n_xblk, int tail_box, int n_xchunk, bool has_tail, int splits,
                                  int kb_total, int workers, int epi, int* grid_out = nullptr) {
  const int n_wtile = n_xblk > 0 ? static_cast<int>(ceil_div(N, bn)) : static_cast<int>(ceil_div(N, 256));
  const int n_wtile256 = static_cast<int>(ceil_div(N, 256));
  const int per = static_cast<int>(ceil_div(kb_total, splits));
  const UnitCost c = unit_cost(bn, tail_box, epi);
  const int64_t units = static_cast<int64_t>(n_xblk) * n_wtile * splits + (has_tail ? static_cast<int64_t>(n_wtile256) * splits * n_xchunk : 0);
  int grid = static_cast<int>(units < workers ? units : workers);
  if (units > grid && has_tail && n_xblk > 0) {
    const int group = (n_xblk + n_xchunk) * splits;
    auto gcd = [](int a, int b) { while (b) { const int t = a % b; a = b; b = t; } return a; };
    while (grid > 1 && gcd(grid, group) != 1) --grid;
  }
  if (grid_out) *grid_out = grid;
  if (grid <= 0) return 0.0;
  if (grid > 160) return 1e30;
  // Runs of equal units: units_run[w] holds the difference array of what starts at worker w, `all` what every worker gets. All
  // costs are whole numbers of clocks, so the sums are exact in any order.
  double step[161] = {0.0}, all = 0.0;
  int at = 0;                        // worker of the next unit
  auto run = [&](int64_t n, double cost) {
    all += static_cast<double>(n / grid) * cost;
    const int r = static_cast<int>(n % grid), end = at + r;
    step[at] += cost;
    if (end <= grid) {
      step[end] -= cost;
    } else {
      step[grid] -= cost;
      step[0] += cost;
      step[end - grid] -= cost;
    }
    at = end < grid ? end : end - grid;
  };
  auto kbs = [&](int s) { const int k1 = (s + 1) * per < kb_total ? (s + 1) * per : kb_total; return k1 - s * per; };
  auto tails_before = [&](int j) {
    if (!has_tail) return 0;
    const int t = n_xblk > 0 ? (j * bn + 255) / 256 : j;
    return t < n_wtile256 ? t : n_wtile256;
  };
  const int s_full = kb_total / per < splits ? kb_total / per : splits;      // K ranges of full length; one shorter may follow
  const double block_full = per * c.block_kb + c.block_epi, tail_full = per * c.tail_kb + c.tail_epi;
  for (int j = 0; j < n_wtile; ++j) {
    run(static_cast<int64_t>(s_full) * n_xblk, block_full);
    for (int s = s_full; s < splits; ++s) run(n_xblk, kbs(s) * c.block_kb + c.block_epi);
    const int nt = (j + 1 < n_wtile ? tails_before(j + 1) : (has_tail ? n_wtile256 : 0)) - tails_before(j);
    for (int t = 0; t < nt; ++t) {
      run(static_cast<int64_t>(s_full) * n_xchunk, tail_full);
      for (int s = s_full; s < splits; ++s) run(n_xchunk, kbs(s) * c.tail_kb + c.tail_epi);
    }
  }
  double worst = 0.0, sum = 0.0;
  for (int k = 0; k < grid; ++k) {
    sum += step[k];
    worst = all + sum > worst ? all + sum : worst;
  }
  return worst + 5000.0;      // launch, TMEM allocation, first stages
}

// Answers of the cost model, which depend on nothing but their whole-number arguments: a forward asks for the same handful of
// shapes in every layer. Direct-mapped and of fixed size, shared by all threads under a lock. Measured on the host before /
// after (with the runs above): the K ranges of a [5120, 17408] projection at 400 rows 572 / 0.2 us (0.12 ms when first
// asked), at 16 672 rows 16.7 ms / 0.2 us (0.20 ms).
template <int KEYS, typename Value>
class ModelCache {
 public:
  template <typename Make>
  Value get(const int64_t (&key)[KEYS], Make make) {
    uint64_t hash = 1469598103934665603ull;
    for (int i = 0; i < KEYS; ++i) hash = (hash ^ static_cast<uint64_t>(key[i])) * 1099511628211ull;
    Slot& slot = slots_[(hash ^ (hash >> 32)) % kSlots];
    {
      std::lock_guard<std::mutex> hold(lock_);
      if (slot.used && memcmp(slot.key, key, sizeof(key)) == 0) return slot.value;
    }
    const Value v = make();
    std::lock_guard<std::mutex> hold(lock_);
    memcpy(slot.key, key, sizeof(key));
    slot.value = v;
    slot.used = true;
    return v;
  }

 private:
  static constexpr int kSlots = 1024;
  struct Slot {
    int64_t key[KEYS];
    Value value;
    bool used;
  };
  std::mutex lock_;
  Slot slots_[kSlots] = {};
};

// The few-row kernel (gemm_skinny.cu): what it takes, and the rows of its w tile.
constexpr int kSkinnyRows = 128;
inline bool skinny_serves(int64_t M, int64_t K) { return M <= kSkinnyRows && K % 64 == 0; }
inline int skinny_bn(int64_t N, int splits) {
  const int64_t per = 148 / splits > 0 ? 148 / splits : 1;
  const int64_t bn = ceil_div(ceil_div(N, per), 16) * 16;
  return static_cast<int>(bn < 128 ? bn : 128);
}

// Width of the w tile of the block units: the multiple of 16 with the smallest modelled time, wider tiles preferred.
inline int choose_bn(int64_t N, int n_xblk, int tail_box, int n_xchunk, bool has_tail, int splits, int kb_total, int workers,
                     int epi) {
  if (n_xblk == 0) return 256;
  static ModelCache<9, int> cache;
  const int64_t key[9] = {N, n_xblk, tail_box, n_xchunk, has_tail, splits, kb_total, workers, epi};
  return cache.get(key, [&] {
    int best = 256;
    double best_cost = 1e30;
    for (int bn = 256; bn >= 64; bn -= 16) {
      if (block_kernel_floor(N, bn, n_xblk, tail_box, n_xchunk, has_tail, splits, kb_total, workers, epi) >= best_cost * 0.98) continue;
      const double cost = block_kernel_clocks(N, bn, n_xblk, tail_box, n_xchunk, has_tail, splits, kb_total, workers, epi);
      if (cost < best_cost * 0.98) { best_cost = cost; best = bn; }
    }
    return best;
  });
}

// How the 256-row block kernel takes the rows behind its full blocks, for M > 128 rows.
struct BlockForm {
  int n_xblk;       // 256-row blocks of x in block units
  int tail_rows;    // rows of x in swapped-operand units, in n_xchunk chunks of tail_box (a multiple of 16, at most 256)
  int tail_box, n_xchunk;
};
// Full blocks and a swapped tail of at most 128 rows (a longer remainder as one more, zero-padded block).
inline BlockForm plain_form(int64_t M) {
  BlockForm f{static_cast<int>(M / kBlockM), static_cast<int>(M % kBlockM), 0, 1};
  if (f.tail_rows > kBM) { f.n_xblk += 1; f.tail_rows = 0; }
  f.tail_box = (f.tail_rows + 15) / 16 * 16;
  return f;
}
// `blocks` full blocks and everything else in swapped chunks.
inline BlockForm chunked_form(int64_t M, int64_t blocks) {
  BlockForm f{static_cast<int>(blocks), static_cast<int>(M - blocks * kBlockM), 0, 0};
  f.n_xchunk = static_cast<int>(ceil_div(f.tail_rows, 256));
  f.tail_box = static_cast<int>(ceil_div(ceil_div(f.tail_rows, f.n_xchunk), 16) * 16);
  return f;
}
// All but the last full block in block units, the remaining 257 .. 511 rows in two swapped chunks that fit them (M > 256): no MMA
// runs at the 64-clock floor of a short tail, and none on the zero rows of a padded block.
inline BlockForm hybrid_form(int64_t M) { return chunked_form(M, M / kBlockM - 1); }

inline double form_floor(const BlockForm& f, int64_t N, int splits, int kb_total, int sms, int epi) {
  double least = 1e30;
  for (int bn = 256; bn >= (epi == kEpiSwiglu ? 256 : 64); bn -= 16) {
    const double floor = block_kernel_floor(N, bn, f.n_xblk, f.tail_box, f.n_xchunk, f.tail_rows > 0, splits, kb_total, sms, epi);
    least = floor < least ? floor : least;
  }
  return least;
}
inline double form_clocks(const BlockForm& f, int64_t N, int splits, int kb_total, int sms, int epi) {
  const bool tail = f.tail_rows > 0;
  const int bn = epi == kEpiSwiglu ? 256 : choose_bn(N, f.n_xblk, f.tail_box, f.n_xchunk, tail, splits, kb_total, sms, epi);
  return block_kernel_clocks(N, bn, f.n_xblk, f.tail_box, f.n_xchunk, tail, splits, kb_total, sms, epi);
}
// The cheaper of the two by the model, and its clocks; no result depends on it (GemmArgs::pair_rows). Not for e4m3 operands, whose results
// would move: a block and a swapped unit multiply the two scales in another order. Measured under the power cap, without / with
// the choice: [12352, 5120] at 1066 / 1184 rows 126 / 140 us and 109 / 122, gate/up at 544 / 1984 / 2208 rows 196 / 563 / 624 and 187 / 553 /
// 615, [5120, 17408] in one K range at 1312 rows 210 and 193.
struct FormChoice {
  BlockForm form;
  double clocks;
};
inline FormChoice choose_form(int64_t M, int64_t N, int splits, int kb_total, int sms, int epi) {
  static ModelCache<6, FormChoice> cache;
  const int64_t key[6] = {M, N, splits, kb_total, sms, epi};
  return cache.get(key, [&] {
    const BlockForm plain = plain_form(M);
    FormChoice best{plain, form_clocks(plain, N, splits, kb_total, sms, epi)};
    if (M > kBlockM && M % kBlockM != 0) {
      const BlockForm hybrid = hybrid_form(M);
      if (form_floor(hybrid, N, splits, kb_total, sms, epi) < best.clocks) {
        const double clocks = form_clocks(hybrid, N, splits, kb_total, sms, epi);
        if (clocks < best.clocks) best = FormChoice{hybrid, clocks};
      }
    }
    return best;
  });
}

}  // namespace
}  // namespace ojb
