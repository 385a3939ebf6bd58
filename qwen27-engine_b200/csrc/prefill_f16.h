// Launcher of the f16-cache prefill kernel (prefill_f16.cu), called by q27b_attn_prefill* when the
// cache is f16.
#pragma once
#include "host.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace q27b {

// How the CTAs of a prefill call (one CTA per SM at a time) split their positions: tiles [0, ts) are split ns ways
// (partials + merge), tiles >= ts are not.
struct SplitPlan {
  int ts, ns;
};
// Q27_ATTN_SPLIT=<n> of the reference (src/attn.cu:952): every tile in n pieces.
inline bool forced_plan(int tiles, bool must_merge, SplitPlan* plan) {
  const char* e = getenv("Q27_ATTN_SPLIT");
  const int f = e ? atoi(e) : 0;
  if (f <= 0) return false;
  *plan = {f > 1 || must_merge ? tiles : 0, std::max(std::min(f, 64), must_merge ? 2 : 1)};
  return true;
}

// The query rows of a KV head are its M * 6 (token, head) pairs, token-major; a CTA takes 128 of them.
constexpr int PF_ROWS = 128, PF_GQA = 6;
__host__ __device__ inline int row_tiles(int M) { return (int)(((int64_t)M * PF_GQA + PF_ROWS - 1) / PF_ROWS); }
// Tokens of the first ts row tiles. Three tiles are 64 tokens; a plan that splits some tiles and not others cuts there.
inline int split_tokens(int M, int ts) { return ts >= row_tiles(M) ? M : ts / 3 * 64; }

// The plan of a prefill call: the first ts row tiles of every KV head are cut into ns pieces over their positions.
// A model of the launch in units of one 64-position tile of a CTA (one CTA per SM at a time): a CTA costs its tiles and
// C0 more (Q tile, pipeline fill, epilogue), a piece CP on top of that (its partials are written), a merge M0 (launch)
// and MROW + MPART * pieces for each row. Three forms compete:
//  * nothing is split;
//  * every tile is split. Few rows behind a long prefix leave most SMs idle otherwise, and a second, partly filled
//    round of CTAs costs as much as a full one: 131 tokens behind 30,011 are 28 tiles, 5 pieces each fill one round of
//    148 SMs (235 us a pass; 4 pieces 276, 6 pieces 359, 10 pieces 249). The other end: 1,000 tokens of one KV head
//    behind 100, 47 tiles of 17 position tiles, 64 us unsplit and 86 in 3 pieces: the merge of 6,000 rows costs more
//    than the idle SMs.
//  * tail split: more CTAs than SMs on a deep prefix. The unsplit CTAs are launched first; only the earliest ts tiles,
//    as many CTAs as the last round would hold, are cut, and their pieces fill the machine evenly at the end. 2048
//    tokens behind 32,768 / 148,000: 3,105 / 13,279 us unsplit, 2,874 / 11,774 with 5 pieces, 2,896 / 11,798 with 8.
// On a short prefix the tiles differ in length (the causal part): longest first, no split once there is a CTA per SM.
// The constants were fitted to an earlier form of the int8 kernel, whose position tile took a seventh longer. Checked with
// the present kernels against forced pieces on fifty shapes (16 to 2,048 tokens behind 100 to 148,000; the times above are
// of the int8 kernel): mostly within 2 % of the best. Known misses: up to some 150 tokens behind 200 to 800, left unsplit
// where three pieces take 15 to 30 % less (16 behind 382, int8: 41.6 us and 31.2), and more than 48 pieces, which the
// merge takes in two turns (39 of one KV head behind 9,071: 33.5 us with 55 pieces, 30.7 with 48).
// f16_qk: the f16-QK kernel, whose position tile takes 1.0 to 1.2 us against 2.0: a merged row costs that many more tiles
// (1,115 tokens of one KV head behind 2,906, 6,690 rows: 86 us unsplit on an f16 cache and 107 in two pieces, 100 and 113
// with f16 Q K^T on a q8_0 cache; the int8 kernel 151 and 139. 600 of two KV heads behind 2,000, f16 cache: 66 and 101).
inline SplitPlan plan_prefill_rows(int M, int nkvh, int n_sm, int depth_hint, bool must_merge, bool f16_qk) {
  constexpr double C0 = 3.0, CP = 4.0, M0 = 2.0;
  const double MROW = f16_qk ? 4.5e-3 : 1.2e-3, MPART = f16_qk ? 3.0e-4 : 2.0e-4;
  const int rt = row_tiles(M), ctas = rt * nkvh;
  SplitPlan plan;
  if (forced_plan(rt, must_merge, &plan)) return plan;
  if (depth_hint < 0) return must_merge ? SplitPlan{rt, 2} : SplitPlan{0, 1};
  const bool deep = depth_hint >= M;
  if (!must_merge && !deep && ctas > n_sm) return {0, 1};
  const double N = ((double)depth_hint + M) / 64, rows = (double)M * nkvh * PF_GQA;
  const int ns_max = std::max(2, std::min(64, (int)(N / 2)));  // two position tiles a piece at least
  auto rounds = [&](double n) { return std::ceil(n / n_sm - 1e-9); };
  plan = must_merge ? SplitPlan{rt, 2} : SplitPlan{0, 1};
  double best = must_merge ? 1e300 : rounds(ctas) * (N + C0);
  for (int k = 2; k <= ns_max && (k == 2 || (int64_t)ctas * (k - 1) < 4 * n_sm); k++) {
    const double t = rounds((double)ctas * k) * (N / k + C0 + CP) + M0 + rows * (MROW + MPART * k);
    if (t < best) best = t, plan = {rt, k};
  }
  const char* tail = getenv("Q27B_PREFILL_TAIL_SPLIT");
  if (must_merge || (tail && tail[0] == '0') || ctas <= n_sm || ctas % n_sm == 0) return plan;
  const int ts = ((ctas % n_sm + nkvh - 1) / nkvh + 2) / 3 * 3;  // whole tokens: see split_tokens
  if (ts >= rt) return plan;
  const int U = ctas - ts * nkvh, b = U % n_sm;
  const int forced = tail ? std::min({atoi(tail), ns_max, 8}) : 0;  // tuning: Q27B_PREFILL_TAIL_SPLIT=<pieces>
  for (int k = 2; k <= std::min(ns_max, 8); k++) {
    const double piece = N / k + C0 + CP;
    // pieces that run beside the last, partly filled round of unsplit CTAs; a tenth of a round more than a whole
    // number does not start another one (the unsplit CTAs do not end all at once)
    const double left = std::max(0.0, (double)ts * nkvh * k - (b ? (n_sm - b) * std::floor((N + C0) / piece) : 0.0));
    const double t = rounds(U) * (N + C0) + rounds(std::max(0.0, left - 0.1 * n_sm)) * piece + M0 +
                     rows * split_tokens(M, ts) / M * (MROW + MPART * k);
    if (forced > 1 ? k == forced : t < best) best = t, plan = {ts, k};
  }
  return plan;
}

// The f16-QK kernel: on an f16 cache (q8 = false), or on a q8_0 cache whose K and V it dequantises to
// f16 on the way (q8 = true; the reference's Q27_ATTN_I8=0 path). o (f32) or xq/xd (q8_1, written by
// the merge kernel of the split path). Same contract as q27b_attn_prefill.
int launch_prefill_f16(DeviceCtx* ctx, const float* qn, const float* qg, const void* kcache, const void* vcache, float* o,
                       int8_t* xq, float* xd, const int* pos0, int M, float kq_scale, int nqh, int nkvh, int n_ctx, bool q8,
                       int depth_hint, cudaStream_t s);

}  // namespace q27b
