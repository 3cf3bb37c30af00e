// C entry points of the bf16 GEMM and the choice between its kernels.
//
//   tile128   (gemm_tile128.cu)   128 x 256 (or 128 x 128) output tiles, two TMEM accumulators so that the epilogue of one
//             tile overlaps the MMAs of the next. M is padded to a multiple of 128.
//   block256  (gemm_block256.cu)  256 rows of x share each w tile between two MMAs (one third less shared-memory fill per
//             flop), w-tile width chosen per shape, the last M mod 256 <= 128 rows (or all rows when M <= 2048, on request) run with
//             swapped operands at their true cost.
//   skinny    (gemm_skinny.cu)    up to 128 rows of x against w tiles of any width, every CTA's shared memory full of weight in
//             flight; bf16: the choice up to about 36 to 60 rows (skinny_clocks), e4m3: wherever it serves.
//   pair256   (gemm_pair256.cu)   the same units on CTA pairs with tcgen05.mma.cta_group::2; measured on par with block256
//             (both are bound by shared-memory bandwidth), kept as variants 5 / 6.
// With variant 0 the kernel is the one with the smallest modelled time (plan_kernel): the models replay the round-robin
// deal of units to CTAs with per-unit costs taken from measured unit timelines.
#include "gemm_units.cuh"

using namespace ojb;

namespace {

// variant: 0 = automatic; 1 = tile128 with 128x256 tiles; 2 = tile128 with 128x128 tiles; a multiple of 16 in [16, 256] =
// block256 with that w-tile width; 3 = block256 with full blocks and a swapped tail of at most 128 rows, automatic width; 4 = block256 with
// every row of x in swapped-operand units (M <= 2048).
// 5 = pair256 (CTA pairs, cta_group::2) with automatic width; 6 = pair256 with every row of x in swapped-operand units
// (any M); 512 + a multiple of 16 in [16, 256] = pair256 with that w-tile width; 7 = block256 with the last 257..511 rows of x in
// two swapped-operand chunks and the rows before them in block units; 8 = block256 as 3 or 7, by the model; 1024 = skinny (M <= 128,
// K % 64 == 0, not for SwiGLU; else as 0) with automatic width;
// 1024 + a multiple of 16 in [16, 128] = skinny with that w-tile width.
bool variant_ok(int v) {
  return (v >= 0 && v <= 8) || (v >= 16 && v <= 256 && v % 16 == 0) || (v >= 528 && v <= 768 && v % 16 == 0) ||
         (v >= 1024 && v <= 1152 && v % 16 == 0);
}

// Modelled SM clocks of the 128-row tile kernel: per k-block a CTA fills (128 + BN) rows and its MMAs read them once,
// 128 bytes per clock; the epilogue overlaps the next tile.
double tile128_clocks(int64_t M, int64_t N, int kb_total, int splits, int bn, int sms, bool f32) {
  const int64_t units = ceil_div(M, 128) * ceil_div(N, bn) * splits;
  const int64_t grid = units < sms ? units : sms;
  const int per = static_cast<int>(ceil_div(kb_total, splits));
  // against the power cap; in short runs a k-block takes 740 and 440 clocks, but the second reading of x costs energy: gate/up at 1600
  // rows, chosen by those, ran 405 us in place of the 370 of 256-row blocks, and everything after it slower
  const double kb = bn == 256 ? 900.0 : 600.0;
  return static_cast<double>(ceil_div(units, grid)) * (per * kb + (f32 ? 33.0 * bn : 1500.0)) + 9000.0;
}

// The few-row kernel: a CTA takes in about 30 bytes per clock, and no k-block (its share of a wait, a commit and the MMAs) in less
// than 220 clocks. Measured against the best of the other kernels, each with its best K ranges (us; * = what the models pick), at
// 12 / 32 / 64 / 128 rows: [12352, 5120] 23.7* / 23.9* / 27.1 / 28.2 against 30.1 / 26.7 / 27.2* / 28.2*, [14336, 5120] 26.1* / 26.5* / 28.9 / 30.8
// against 30.7 / 28.9 / 29.7* / 30.4*, [2048, 5120] 15.3* / 15.2* / 16.3* / 18.3* against 21.2 / 21.2 / 21.4 / 21.9, [5120, 4096]
// 10.7* / 11.0* / 11.5 / 15.3 against 11.7 / 12.0 / 13.4* / 15.8*, [5120, 6144] 14.0* / 14.2* / 15.1 / 19.0 against 15.2 / 15.4 / 16.8* / 19.2*,
// [5120, 17408] 31.1* / 31.8 / 33.1 / 38.0 against 32.1 / 33.2* / 35.1* / 38.3*. With many rows the model is too high (30.6 us for
// [2048, 5120] at 128 rows), and the swapped-operand units take over above about 36 rows where this kernel still leads, by 4 to 20 % up to 96 rows
// where there are K ranges: those are chosen by the same figures, and another fit would move results. tune() times both. (Rows are
// counted in eights; a launch with x as the N side loads them in sixteens, at most eight more.)
double skinny_clocks(int64_t M, int64_t N, int kb_total, int splits, int sms) {
  const int bn = skinny_bn(N, splits);
  const double waves = static_cast<double>(ceil_div(ceil_div(N, bn) * splits, sms));
  const double fill = (bn + ceil_div(M, 8) * 8) * 128.0 / 30.0, per = static_cast<double>(ceil_div(kb_total, splits));
  return waves * per * (fill > 220.0 ? fill : 220.0) + 6000.0;
}

struct Plan {
  int variant;
  double clocks;
  int pair_rows = -1;      // see gemm_block256_launch
};

// Cheapest kernel for this shape and number of K ranges according to the cost models (gemm_units.cuh), never below the
// time HBM needs for the weight.
// eight_bit: the ranges of K of an 8-bit product. They regroup its sums, and on e4m3 operands a regrouped sum moves the result of
// a deep model by percents, so that choice stays on the model it was first made with.
// plain_forms: as if the block kernel had its plain form alone, for choices that a result depends on.
Plan model_kernel(int epi, int64_t M, int64_t N, int64_t K, int splits, bool plain_forms, bool eight_bit = false) {
  const int sms = 148;
  const int kb_total = static_cast<int>(ceil_div(K, 64));
  Plan best{3, 1e30};
  const bool f32 = epi == kEpiPartialF32 && !eight_bit;
  const int model_epi = eight_bit ? kEpi8BitRanges : epi;
  auto consider = [&](int variant, double clocks) {
    if (clocks < best.clocks) best = Plan{variant, clocks, -1};
  };
  if (epi != kEpiSwiglu || M > 64) consider(1, tile128_clocks(M, N, kb_total, splits, 256, sms, f32));
  if (epi != kEpiSwiglu) consider(2, tile128_clocks(M, N, kb_total, splits, 128, sms, f32));
  if (plain_form(M).n_xblk > 0) {      // block256
    if (plain_forms) consider(3, form_clocks(plain_form(M), N, splits, kb_total, sms, model_epi));
    else consider(8, choose_form(M, N, splits, kb_total, sms, model_epi).clocks);
  }
  if (M <= 2048) {  // block256 with every row in swapped-operand units
    const BlockForm f = chunked_form(M, 0);
    consider(4, block_kernel_clocks(N, 256, 0, f.tail_box, f.n_xchunk, true, splits, kb_total, sms, model_epi));
  }
  if (epi != kEpiSwiglu && skinny_serves(M, K) && !eight_bit) consider(1024, skinny_clocks(M, N, kb_total, splits, sms));
  const double hbm = (static_cast<double>(N) * K * 2.0) / 3500.0 + 7000.0;     // bytes per clock at 6.3 TB/s and 1.8 GHz
  if (best.clocks < hbm) best.clocks = hbm;
  return best;
}

Plan plan_kernel(int epi, int64_t M, int64_t N, int64_t K, int splits) {
  static ModelCache<5, Plan> cache;
  const int64_t key[5] = {epi, M, N, K, splits};
  return cache.get(key, [&] {
    Plan p = model_kernel(epi, M, N, K, splits, false);
    // SwiGLU: which rows take their SiLU in pairs follows from the kernel that the plain forms would get
    if (epi == kEpiSwiglu && p.variant == 8 && model_kernel(epi, M, N, K, splits, true).variant != 3) p.pair_rows = 0;
    return p;
  });
}

int dispatch(int epi, int variant, const void* x, const void* w, void* out, int64_t M, int64_t N, int64_t K, int splits,
             int64_t ldo, int32_t* status, cudaStream_t st) {
  if (variant == 1024 && (epi == kEpiSwiglu || !skinny_serves(M, K))) variant = 0;
  int pair_rows = -1;
  if (variant == 0) {
    const Plan p = plan_kernel(epi, M, N, K, splits);
    variant = p.variant;
    pair_rows = p.pair_rows;
  }
  if (variant >= 1024) return gemm_skinny_launch(epi, variant - 1024, x, w, out, M, N, K, splits, ldo, status, st);
  if (variant == 5 || variant == 6 || variant >= 512)
    return gemm_pair256_launch(epi, variant == 5 ? 0 : (variant == 6 ? -1 : variant - 512), x, w, out, M, N, K, splits, ldo, status, st);
  if (variant == 1 || variant == 2)
    return gemm_tile128_launch(epi, variant == 1 ? 256 : 128, x, w, out, M, N, K, splits, ldo, status, st);
  return gemm_block256_launch(epi, variant == 8 ? 0 : (variant == 4 ? -1 : (variant == 7 ? -2 : (variant == 3 ? -3 : variant))), x, w, out, M, N, K, splits, ldo, status, st,
                              pair_rows);
}

}  // namespace

extern "C" int ojb_gemm_bf16(const void* x, const void* w, void* out, int64_t M, int64_t N, int64_t K, int variant,
                             int32_t* status, ojb_stream_t stream) {
  OJB_REQUIRE(x && w && out && M > 0 && N > 0 && K > 0 && K % 8 == 0 && variant_ok(variant));
  OJB_REQUIRE(aligned16(x) && aligned16(w) && aligned16(out));
  return dispatch(kEpiBf16, variant, x, w, out, M, N, K, 1, N, status, static_cast<cudaStream_t>(stream));
}

extern "C" int ojb_gemm_bf16_swiglu_v(const void* x, const void* w_blk, void* out, int64_t M, int64_t N, int64_t K, int variant,
                                      int32_t* status, ojb_stream_t stream) {
  OJB_REQUIRE(x && w_blk && out && M > 0 && N > 0 && K > 0 && K % 8 == 0 && N % 256 == 0);
  OJB_REQUIRE(aligned16(x) && aligned16(w_blk) && aligned16(out) && (variant == 0 || variant == 1 || variant == 3 || variant == 4 || variant == 5 || variant == 6 || variant == 7 || variant == 8 || variant == 1024));
  return dispatch(kEpiSwiglu, variant, x, w_blk, out, M, N, K, 1, N / 2, status, static_cast<cudaStream_t>(stream));
}

extern "C" int ojb_gemm_bf16_swiglu(const void* x, const void* w_blk, void* out, int64_t M, int64_t N, int64_t K,
                                    int32_t* status, ojb_stream_t stream) {
  return ojb_gemm_bf16_swiglu_v(x, w_blk, out, M, N, K, 0, status, stream);
}

extern "C" int ojb_gemm_bf16_splitk(const void* x, const void* w, float* parts, int64_t M, int64_t N, int64_t K,
                                    int splits, int variant, int32_t* status, ojb_stream_t stream) {
  OJB_REQUIRE(x && w && parts && M > 0 && N > 0 && K > 0 && K % 8 == 0 && splits >= 1 && splits <= 16 && variant_ok(variant));
  OJB_REQUIRE(aligned16(x) && aligned16(w) && aligned16(parts));
  return dispatch(kEpiPartialF32, variant, x, w, parts, M, N, K, splits, N, status, static_cast<cudaStream_t>(stream));
}

extern "C" int ojb_gemm_bf16_add(const void* x, const void* w, float* h, int64_t M, int64_t N, int64_t K, int variant, int32_t* status,
                                 ojb_stream_t stream) {
  OJB_REQUIRE(x && w && h && M > 0 && N > 0 && K > 0 && K % 8 == 0 && N % 32 == 0 && (variant == 0 || variant == 3 || variant == 4));
  OJB_REQUIRE(aligned16(x) && aligned16(w) && aligned16(h));
  return gemm_block256_add_launch(variant == 4 ? -1 : (variant == 3 ? -3 : 0), x, w, h, M, N, K, status, static_cast<cudaStream_t>(stream));
}

namespace ojb {
namespace { int g_wait_ms = kDefaultWaitMs, g_drop_copy = 0; }
int gemm_wait_limit_ms() { return g_wait_ms; }
int gemm_drop_copy() { return g_drop_copy; }
}  // namespace ojb

extern "C" int ojb_gemm_set_wait_limit_ms(int32_t ms) {
  OJB_REQUIRE(ms >= 0 && ms <= 60000);
  ojb::g_wait_ms = ms == 0 ? ojb::kDefaultWaitMs : ms;
  return OJB_OK;
}

extern "C" int ojb_gemm_test_drop_copy(int32_t on) {
  ojb::g_drop_copy = on ? 1 : 0;
  return OJB_OK;
}

extern "C" int ojb_gemm_set_trace(uint64_t* records, int32_t capacity) {
  OJB_REQUIRE(capacity >= 0);
  gemm_block256_set_trace(reinterpret_cast<unsigned long long*>(records), capacity);
  gemm_pair256_set_trace(reinterpret_cast<unsigned long long*>(records), capacity);
  return OJB_OK;
}

#ifdef OJB_GEMM_PROBES
// Probe builds only (not declared in the public header): MMA repeat count and pipeline / epilogue knobs.
extern "C" int ojb_gemm_set_probe(int32_t mma_repeat, int32_t knob) {
  OJB_REQUIRE(mma_repeat >= 0 && mma_repeat <= 64 && (knob == 0 || (knob >= 2 && knob <= 12) || knob == 100 || knob == 101 || knob == 102));
  gemm_block256_set_probe(mma_repeat, knob);
  gemm_pair256_set_probe(mma_repeat, knob);
  return OJB_OK;
}
#endif

extern "C" int ojb_gemm_band_blocks(int32_t n_xblk, int64_t K, int32_t elt) {
  return n_xblk > 0 && K > 0 && (elt == 1 || elt == 2) ? band_blocks(n_xblk, 256 * K * elt) : 0;
}

extern "C" int ojb_gemm_plan(int64_t M, int64_t N, int64_t K, int32_t kind, int32_t max_splits, int32_t* variant, int32_t* splits,
                             float* microseconds) {
  OJB_REQUIRE(M > 0 && N > 0 && K > 0 && kind >= 0 && kind <= 3 && max_splits >= 1 && max_splits <= 16 && variant && splits);
  struct Ranges {
    Plan plan;
    int splits;
  };
  static ModelCache<5, Ranges> cache;
  const int64_t key[5] = {M, N, K, kind, max_splits};
  const Ranges r = cache.get(key, [&] {
    const int kb_total = static_cast<int>(ceil_div(K, 64));
    const bool eight_bit = kind == 3, parts = kind >= 2;
    Plan best{0, 1e30};
    int best_s = 1;
    for (int s = 1; s <= (parts ? max_splits : 1); ++s) {
      const int per = static_cast<int>(ceil_div(kb_total, s));
      if (static_cast<int64_t>(s - 1) * per >= kb_total) continue;
      // (K ranges regroup the sums, so they are chosen over the plain forms: another form of the block kernel changes no result)
      Plan p = model_kernel(eight_bit ? kEpiPartialF32 : kind, M, N, K, s, parts, eight_bit);
      // the kernel that sums the partial planes reads S * M * N floats (mostly from L2)
      if (parts) p.clocks += (s - 1) * static_cast<double>(M) * N * 4.0 / 5000.0;
      if (p.clocks < best.clocks * 0.97) { best = p; best_s = s; }
    }
    if (kind == 2) {
      best = model_kernel(kind, M, N, K, best_s, false);
      best.clocks += (best_s - 1) * static_cast<double>(M) * N * 4.0 / 5000.0;
    }
    return Ranges{best, best_s};
  });
  *variant = r.plan.variant == 8 ? 3 : r.plan.variant;      // (the block kernel, whatever its form)
  *splits = r.splits;
  if (microseconds) *microseconds = static_cast<float>(r.plan.clocks / 1800.0);
  return OJB_OK;
}

extern "C" int ojb_gemm_e4m3(const void* xq, const float* sx, const void* wq, const float* sw, void* out, int64_t M, int64_t N,
                             int64_t K, int32_t kind, int32_t splits, int32_t* status, ojb_stream_t stream) {
  if (M == 0 || N == 0) return OJB_OK;
  OJB_REQUIRE(xq && sx && wq && sw && out && M > 0 && N > 0 && K > 0 && K % 16 == 0 && kind >= 0 && kind <= 3);
  OJB_REQUIRE(aligned16(xq) && aligned16(wq) && aligned16(out));
  OJB_REQUIRE(kind == 2 ? (splits >= 1 && splits <= 16) : splits == 1);
  OJB_REQUIRE(kind != 1 || N % 256 == 0);
  OJB_REQUIRE(kind != 3 || N % 64 == 0);
  const int epi = kind == 0 ? kEpiBf16 : (kind == 1 ? kEpiSwiglu : kEpiPartialF32);
  if (kind == 3)
    return gemm_block256_launch_e4m3(epi, xq, sx, wq, sw, out, M, N, K, 1, N, status, static_cast<cudaStream_t>(stream), true);
  if (M <= kSkinnyRows && K % 128 == 0 && epi != kEpiSwiglu)
    return gemm_skinny_launch(epi, 0, xq, wq, out, M, N, K, splits, N, status, static_cast<cudaStream_t>(stream), sx, sw);
  return gemm_block256_launch_e4m3(epi, xq, sx, wq, sw, out, M, N, K, splits, kind == 1 ? N / 2 : N, status,
                                   static_cast<cudaStream_t>(stream));
}
