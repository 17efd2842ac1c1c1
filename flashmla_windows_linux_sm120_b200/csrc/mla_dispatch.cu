// Which kernel runs an MLA attention call: the CTA pair (mla_pair.cu) where 128 heads share a kv head, or the 64 heads of two
// query tokens -- its two CTAs read every cached token once for all of them.  Otherwise one CTA per 64 heads (mla_tile64.cu) for
// the sparse prefill and where several such tiles of a dense decode read the same pages, or per at most 64 query rows
// (mla_few_rows.cu).
#include "kernels.h"

#include <algorithm>
#include <cstdlib>

namespace fmla {

// FMLA_DISABLE_PAIR=1 in the environment keeps the one-CTA kernels for every shape (A/B runs)
static bool pair_kernel_enabled() {
  static const bool on = [] {
    const char* v = getenv("FMLA_DISABLE_PAIR");
    return !(v && v[0] == '1');
  }();
  return on;
}

bool decode_dense_merges_in_kernel(const DecodeKernelParams& p) {
  return p.topk < 0 && decode_dense_pair_applies(p) && pair_kernel_enabled() && p.arrival_counters != nullptr && !p.force_partial;
}

// Whether the schedule of requests of `topk` indices each lets sub_splits (mla_work.cuh) share out its rows; costs, pitch and cuts as
// in csrc/scheduler.cu.  Another schedule of the same sizes is served as well, without sharing or by what the kernels find in it.
static bool uniform_schedule_shares_rows(int b, int topk, int parts) {
  const int64_t cost = topk / 64 + 5, total = b * cost, pitch = (total + parts - 1) / parts + 5;      // b < parts
  const int64_t cuts = (total - 1) / pitch;
  if (cuts <= b || cuts + 1 > parts / 2) return false;
  int64_t slots = b;
  for (int64_t i = 1; i <= cuts; ++i) slots += i * pitch % cost > 5;
  return slots > 2 * b && 2 * slots <= b + parts;
}

// Whether a call takes the form of the kernels that looks for rows to share.  The kernel for at most 64 rows only; not where the
// partials leave the GPU, and not where the caller says that there are none.  Looking costs a call that shares nothing 0.1 to 0.5 us
// (32 heads, 32 x 500 tokens 21.9 -> 22.2 us, 16 heads, 40 x 4 000 47.2 -> 47.6), so it is left out where it is known to find nothing.
bool decode_splits_rows_further(const DecodeKernelParams& p) {
  if (p.force_partial || p.no_split_hint) return false;
  if (3 * static_cast<int64_t>(p.b) + 2 > p.num_sm_parts) return false;      // twice 2 b + 1 slots are more than the b + num_sm_parts there are
  if (p.topk >= 0) return !(decode_sparse_pair_applies(p) && pair_kernel_enabled()) && uniform_schedule_shares_rows(p.b, p.topk, p.num_sm_parts);
  // The most blocks that a request can have, as far as the stride of the block table tells: a row of the schedule has six or more,
  // so that requests of seven are cut once at most.
  if (p.block_table_stride_b > 0 && p.block_table_stride_b < 8) return false;
  return !(decode_dense_pair_applies(p) && pair_kernel_enabled()) && !decode_dense_tile64_applies(p);
}

cudaError_t launch_decode_dense_tc(const DecodeKernelParams& p, cudaStream_t stream) {
  if (decode_dense_pair_applies(p) && pair_kernel_enabled()) return launch_decode_dense_pair(p, stream);
  if (decode_dense_tile64_applies(p)) return launch_decode_dense_tile64(p, stream);
  return launch_decode_few_rows(p, stream);
}

cudaError_t launch_decode_sparse_tc(const DecodeKernelParams& p, cudaStream_t stream) {
  if (decode_sparse_pair_applies(p) && pair_kernel_enabled()) return launch_decode_sparse_pair(p, stream);
  return launch_decode_sparse_few_rows(p, stream);
}

// The tokens of a last round that leaves half of the units or more idle (with few query tokens, that is all of them) are cut,
// in stretches of at least two blocks, where the blocks saved are worth more than the merge.  Both sides in us, from 72 shapes of 1 to 333
// tokens, 64 and 128 heads, top-k 384 to 2048: a block takes a pair 1.06 and a CTA 1.66; the merge kernel and the partials
// 4 and 0.04 for every partial of 64 rows, 3 more where a pair has whole tokens in front (a token boundary) and 3 % of those (the
// kernel with both kinds of stores spills).
// Whole -> cut: 128 heads, top-k 2048, 1 / 12 / 37 / 100 tokens 44.7 -> 16.8, 45.2 -> 26.8, 46.5 -> 38.3, 91.4 -> 80.7 us; top-k 1024, 24 / 37
// tokens 27.1 -> 26.4, 27.8 -> 28.5; 64 heads, top-k 2048, 1 / 37 / 333 tokens 63.2 -> 16.4, 63.5 -> 30.7, 183 -> 154; top-k 512, 1 / 37
// tokens 20.5 -> 14.3, 20.5 -> 20.5.  (All blocks on one line, cut anywhere: 60 tokens, 128 heads, top-k 2048 53.7 -> 61.3.)
// At its line the rule takes what is worth nothing either way.  64 heads, top-k 512, one round of whole tokens in front, whole -> cut: 37 left
// over (four parts of two blocks, taken) 37.0 -> 34.5; 38, 44, 50, 62 and 74 (three and two parts, refused) 37.0 -> 36.8, 36.8 -> 37.0, 36.8 ->
// 36.9, 37.0 -> 36.9, 37.4 -> 37.7; two rounds in front 37: 53.7 -> 53.2, 50: 53.3 -> 54.9.  Top-k 1024, 38 to 74 (taken) 65.8 -> 56.4 to 59.6.  128 heads, top-k
// 1024, 74 in front, 18 (refused) 50.7 -> 47.1, 25: 50.9 -> 50.8, 31: 51.0 -> 51.2.
// With the kernels as they are now a block takes a CTA 1.39 and the merge and its partials some 2 to 3; over 100 shapes of up to one round in
// front the constants still choose within 0.8 us of the better side, but for pairs with one round in front, where less is lost than
// assumed (refused: 92 tokens, top-k 1024 47.1 -> 43.5, 111, top-k 1536 64.6 -> 60.4; two rounds 1 to 6 us of it, three all of it).  They stay
// because they also say which calls need scratch, and a caller of the C entry may bring none where none was needed.
void plan_sparse_prefill(SparsePrefillKernelParams& sp, int sms, bool can_split) {
  const int cap = std::max(1, sms / (sp.h_q / 64)), nblk = sp.topk / 64;      // pairs for 128 heads, CTAs per 64-head tile otherwise
  sp.units = std::min(sp.s_q, cap);
  sp.whole = sp.s_q;
  sp.pitch = nblk;
  sp.per = 1;
  const int rest = sp.s_q % cap;
  if (!can_split || rest == 0) return;
  const int pitch = std::max((nblk + cap / rest - 1) / (cap / rest), 2), per = (nblk + pitch - 1) / pitch;
  const bool pair = sparse_prefill_pair_applies(sp) && pair_kernel_enabled();
  const float saved = (nblk - pitch) * (pair ? 1.06f : 1.66f);
  float cost = 4.f + 0.04f * rest * per * (sp.h_q / 64);
  if (pair && sp.s_q > rest) cost += 3.f + 0.03f * 1.06f * nblk * (sp.s_q / cap);
  if (saved <= cost) return;
  sp.whole = sp.s_q - rest;
  sp.pitch = pitch;
  sp.per = per;
  sp.units = sp.whole > 0 ? cap : rest * per;
}

cudaError_t launch_sparse_prefill_tc(const SparsePrefillKernelParams& sp, cudaStream_t stream) {
  const cudaError_t e = sparse_prefill_pair_applies(sp) && pair_kernel_enabled() ? launch_sparse_prefill_pair(sp, stream) : launch_sparse_prefill_64(sp, stream);
  return e == cudaSuccess && sp.per > 1 ? launch_sparse_prefill_combine(sp, stream) : e;
}

}  // namespace fmla
