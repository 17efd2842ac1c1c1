// Work decomposition of the CTA-pair MLA attention kernel (mla_pair.cu; the modes also of mla_few_rows.cu): which tile of heads and
// which stretch of the split-KV schedule a CTA owns, and the requests / query tokens it walks.
// The kernel is resident while the one that writes the schedule may still run, so schedule and lengths are read with plain
// loads, after pdl_wait(): __ldg is undefined for memory written meanwhile and may be moved above the wait.
#pragma once

#include "kernels.h"

namespace fmla {

enum TcMode { kDense = 0, kSparseDecode = 1, kSparsePrefill = 2, kSparsePrefillCut = 3 };      // the last: with query tokens that are cut

struct TcParams {
  DecodeKernelParams d;          // decode modes
  SparsePrefillKernelParams sp;  // prefill mode
};

// One unit of work of a CTA: a request (decode) or a query token (prefill) and the range of
// 64-token blocks of its key list that this CTA covers.
struct Work {
  int batch;                 // request index (decode) / query token (prefill)
  int blk_lo, blk_hi;
  int seqlen, border;        // dense: cached tokens, first masked token
  int split_slot;
  bool no_split;
  const int* idx;            // sparse: the index list of this (request, query token)
};

// Which tile and which stretch of the schedule a CTA owns.
struct Tile {
  int sq, hb, kh, head0;
  int begin_idx, end_idx, begin_block, end_block, begin_split;
  int n_work;
};

template <int MODE>
__device__ __forceinline__ Tile make_tile(const TcParams& P) {
  Tile t;
  if constexpr (MODE == kSparsePrefill || MODE == kSparsePrefillCut) {
    // persistent over query tokens: this CTA takes tokens blockIdx.y, blockIdx.y + gridDim.y, ... so that the
    // Q load and the output stores of one token overlap with the blocks of its neighbours; kSparsePrefillCut: then a stretch of a
    // token that is cut (SparsePrefillKernelParams)
    t.hb = blockIdx.x; t.sq = blockIdx.y; t.kh = 0;
    t.head0 = t.hb * 64;
    t.begin_idx = t.end_idx = 0; t.begin_block = 0; t.end_block = P.sp.topk / 64; t.begin_split = 0;
    const int whole = MODE == kSparsePrefill ? P.sp.s_q : P.sp.whole;
    t.end_idx = max(0, whole - t.sq + static_cast<int>(gridDim.y) - 1) / static_cast<int>(gridDim.y);      // whole tokens of this unit
    t.n_work = t.end_idx + (MODE == kSparsePrefillCut && t.sq < (P.sp.s_q - whole) * P.sp.per ? 1 : 0);
  } else {
    const DecodeKernelParams& p = P.d;
    int part;
    if constexpr (MODE == kDense) {
      const int n_hb = (p.hq_per_hk + 63) >> 6;
      t.sq = blockIdx.x / n_hb; t.hb = blockIdx.x % n_hb; t.kh = blockIdx.y; part = blockIdx.z;
    } else {
      t.hb = blockIdx.x; t.sq = blockIdx.y; t.kh = 0; part = blockIdx.z;
    }
    t.head0 = t.kh * p.hq_per_hk + t.hb * 64;
    const int4 md = *reinterpret_cast<const int4*>(p.tile_scheduler_metadata + part * 8);
    t.begin_idx = md.x; t.begin_block = md.y; t.end_idx = md.z; t.end_block = md.w;
    t.begin_split = p.tile_scheduler_metadata[part * 8 + 4];
    t.n_work = t.begin_idx >= p.b ? 0 : t.end_idx - t.begin_idx + 1;
  }
  return t;
}

template <int MODE>
__device__ __forceinline__ Work get_work(const TcParams& P, const Tile& t, int i) {
  Work w;
  if constexpr (MODE == kSparsePrefill || MODE == kSparsePrefillCut) {
    w.batch = t.sq + i * static_cast<int>(gridDim.y);          // the query token
    w.blk_lo = 0; w.blk_hi = P.sp.topk / 64;
    w.seqlen = P.sp.topk; w.border = P.sp.topk;
    w.split_slot = t.sq; w.no_split = true;
    if (MODE == kSparsePrefillCut && i >= t.end_idx) {
      w.batch = P.sp.whole + t.sq / P.sp.per;
      w.blk_lo = t.sq % P.sp.per * P.sp.pitch;
      w.blk_hi = min(w.blk_lo + P.sp.pitch, w.blk_hi);
      w.no_split = false;
    }
    w.idx = P.sp.indices + (int64_t)w.batch * P.sp.indices_stride_s;
  } else {
    const DecodeKernelParams& p = P.d;
    const int batch = t.begin_idx + i;
    w.batch = batch;
    int nblk_total, nblk_visible;
    if constexpr (MODE == kDense) {
      w.seqlen = p.seqlens_k[batch];
      nblk_total = (w.seqlen + 63) >> 6;
      w.border = p.is_causal ? w.seqlen - (p.s_q - 1 - t.sq) : w.seqlen;
      // with 64 heads the two CTAs of a pair hold consecutive query tokens and walk the blocks that the later one sees
      const int seen = p.is_causal && p.hq_per_hk == 64 ? w.seqlen - (p.s_q - 1 - (t.sq | 1)) : w.border;
      nblk_visible = seen > 0 ? (seen + 63) >> 6 : 0;
      w.idx = nullptr;
    } else {
      w.seqlen = p.topk; w.border = p.topk;
      nblk_total = nblk_visible = p.topk >> 6;
      w.idx = p.indices + batch * p.indices_stride_b + t.sq * p.indices_stride_s;
    }
    w.blk_lo = batch == t.begin_idx ? t.begin_block : 0;
    w.blk_hi = min(min(batch == t.end_idx ? t.end_block : nblk_total, nblk_total), nblk_visible);
    if (w.blk_hi < w.blk_lo) w.blk_hi = w.blk_lo;
    const int lo = p.num_splits[batch];
    w.no_split = !p.force_partial && p.num_splits[batch + 1] - lo == 1;
    w.split_slot = lo + (batch == t.begin_idx ? t.begin_split : 0);
  }
  return w;
}

// CTAs per row of the schedule.  With no more requests than rows the schedule takes at least six blocks per row (the slack that lets
// equal requests fall one per row), so a small batch leaves most rows empty: 7 requests of 2 000 tokens occupy 34 of 148.  Each
// row is then shared by as many CTAs as there are empty rows for (the rows in use come first), as far as the partials fit the
// b + num_sm_parts slots; slot i of num_splits becomes the slots k i .. k i + k - 1.  Only where the schedule has more than two parts per
// request on average: the merge is then paid for (from more than three on 16 x 1 000 tokens, 16 heads, stay at 20.2 us instead of 15.3; from
// more than one on 64 heads, 30 x top-k 512 would take 21.8 instead of 28.9, but one request of 100 tokens 11.4 instead of 9.7).
// Attention and merge kernel find the same k from the schedule alone.
// Unshared -> shared: 16 heads, 4 x 1 024 tokens 16.1 -> 13.5 us, 16 x 1 000 19.8 -> 15.2; 64 heads, 1 x 8 000 25.0 -> 22.0, 24 x 1 500 29.6 ->
// 24.3; sparse, 64 heads, top-k 2048, 1 request 24.5 -> 17.5, 5 of two tokens, top-k 512, 24.2 -> 16.6.
// Seven would take a schedule of at most a seventh of the rows, and the rows of that have six blocks.
constexpr int kMaxSubSplits = 6;
constexpr int kMaxPartsPerRequest = 64;      // on average: 1 x 8 000 tokens, 64 heads: 21.3 us with 44 parts, 26.3 with 132
// AT_ONCE: everything is asked for at once; otherwise first what rules most schedules out.  The words are the same for all CTAs, and as
// soon as many warps ask for them they queue up: one thread of each attention CTA reads them at once, the warps of the merge
// one after the other (all of them at once: 32 x 500 tokens, 32 heads, 22.2 -> 22.8 us, past the L1 cache 23.9).
template <bool AT_ONCE>
__device__ __forceinline__ int sub_splits(const DecodeKernelParams& p) {
  const int slots = p.num_splits[p.b], room = min(p.b + p.num_sm_parts, kMaxPartsPerRequest * p.b);
  int first[kMaxSubSplits + 1];      // the request of the first row that has to be empty for k = i
  first[2] = p.tile_scheduler_metadata[p.num_sm_parts / 2 * 8];
  if (!AT_ONCE && (slots <= 2 * p.b || first[2] < p.b)) return 1;
#pragma unroll
  for (int i = 3; i <= kMaxSubSplits; ++i) first[i] = p.tile_scheduler_metadata[p.num_sm_parts / i * 8];
  int k = 1;
#pragma unroll
  for (int i = 2; i <= kMaxSubSplits; ++i)
    if (first[i] >= p.b && i * slots <= room) k = i;
  return slots > 2 * p.b ? k : 1;
}

}  // namespace fmla
