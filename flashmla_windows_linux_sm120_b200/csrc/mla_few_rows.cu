// Split-KV MLA decode for at most 64 query rows per CTA on sm_100a -- dense (heads x query tokens of one kv head) and
// sparse FP8 (heads of one query token): the products are computed transposed, with the cached tokens as the rows of the
// accumulator and the query rows as its columns.
//   S^T[64 tokens x N] = K Q^T       36 x tcgen05.mma m64nNk16    A = the page as TMA lands it, B = Q
//   O^T[512 x N]      += V^T P^T     16 x tcgen05.mma m128nNk16   A = the same page read MN-major, B = P
// with N = 16, 32 or 64, the smallest that holds the tile's rows.  What bounds the path is the cache stream (1152 bytes
// per token against 2 * 1088 * rows FLOP), so the layout serves the loads in flight:
//   * Q takes N x 1152 bytes of shared memory instead of 72 KB: the rest is a ring of 8 KB slots (64 tokens x 64
//     columns) filled slot by slot behind the pages that P V has finished with -- 22 + 3 slots for N = 16 (2.8 pages in flight), 20 + 2 for N = 32,
//     16 + 2 for N = 64.  Two whole-page stages, each held from the start of its load to the end of its P V, left the
//     memory idle half of the time (61 requests x 6000 tokens, 16 heads: 117 us against 63 us at the copy bandwidth).
//   * several query tokens share a CTA and with it the page (s_q * heads <= 64: the cache is read once per step, not
//     once per query token).
//   * an output column lives in one TMEM lane: a warp's store to a partial covers 32 consecutive columns of a row (64 rows of
//     2 KB leave the SM in 5 200 clk; with one row per lane they took 10 000).  Rows of whole requests are transposed on the
//     way out (stmatrix) and leave in 16-byte pieces: 4 600 clk for 64 of them.
// 64-head tiles that read the same pages belong to the CTA pair (two of them, mla_pair.cu) or to mla_tile64.cu instead.  The next page is read into L2
// ahead of its loads, as one piece (kPrefetchBlocks); in tiles and six pages ahead that was slower throughout.
// Warps: 0-3 softmax and epilogue, 4 TMA, 5 MMA, 6-13 gather (sparse), which read the 656-byte records of a 64-index block
// into registers one block ahead, de-quantise (bf16(fp32(e4m3) * scale)) and store them into the slots in the layout TMA
// produces.  An invalid index leaves a zero row and a cleared validity bit.
//   softmax : S^T by 16x256b loads (lane = token row t/4 and t/4 + 8 of the warp's 16 tokens, columns 2(t%4) + 8k + {0,1}).
//             The running reference m_used of a column moves only when a logit exceeds it by more than 2^8, which one
//             barrier-with-reduction per block decides for all 128 threads; only then the column maxima are formed
//             (shuffles + shared memory) and O^T is rescaled.  P goes out as bf16 / fp16 through stmatrix.trans into the
//             K-major operand tile [N x 64 tokens].
// TMEM: O^T value columns [128 m, 128 m + 128) = columns [m N, m N + N); S^T buffers at 256 and 256 + N.
// Semantics follow the reference kernels: decode borders / split outputs / LSE conventions
// csrc/sm90/decode/dense/splitkv_mla.cu:948-957, 1022-1042, 1237-1269; sparse decode
// csrc/sm100/decode/sparse_fp8/splitkv_mla.cu:168-186, 217-256; FP8 record README.md:162-170 with de-quantisation as tests/quant.py:60-63.
// Every wait is bounded; on expiry the CTA drains and frees its tensor memory.
#include "kernels.h"
#include "launch.cuh"
#include "mla_work.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

#include <cuda.h>
#include <cuda_fp8.h>
#include <type_traits>

namespace fmla {

// What a CTA works on where the rows of the schedule are shared (share_of_row), laid out as a row is.
struct alignas(16) RowShare {
  int4 row;                    // first request and block, last request and block
  int split;                   // first split of the first request
  int share;                   // k, and part v of c of the request's blocks: k | v << 8 | c << 16
};

namespace frt {
constexpr int kSlot = 64 * 128;                   // 64 tokens x 64 columns of 16 bits
constexpr int kPageBytes = 9 * kSlot;
constexpr int kPageBars = 4;                      // pages that can have slots in the ring at the same time
constexpr int kGather = 8;                        // gather warps, eight rows of a block each
// Stretches of a request from this many pages on ask for the next page in L2.  16 heads, 61 x 6000 tokens 88.8 -> 81.5 us (5.2 ->
// 5.7 TB/s), 128 x 2000 72.7 -> 67.0; 32 heads, 20 x 9000 57.4 -> 54.3; 64 heads, 32 x 9000 95 -> 88, 100 x 1000 (16 pages) 55.9 -> 52.9.  Shorter ones lose:
// 16 heads, 60 x 700, two tokens (11 pages) 28.9 -> 29.2, 128 x 300 24.2 -> 24.5, 1 x 30 000 (4 pages a CTA) 26.6 -> 27.3.  Two pages ahead 84.0 us
// in the first case, three 88.1.
constexpr int kPrefetchBlocks = 12;
constexpr int threads(int mode) { return (6 + (mode == kDense ? 0 : kGather)) * 32; }
template <int N>
struct Layout {
  static constexpr int kQChunk = N * 128;
  static constexpr int Q_OFF = 0;
  static constexpr int kVSlots = N == 16 ? 22 : N == 32 ? 20 : 16;      // even: the pair (2m, 2m+1) of a page never wraps
  static constexpr int kRopeSlots = N == 16 ? 3 : 2;
  static constexpr int kPBufs = N == 64 ? 1 : 2;
  static constexpr int V_OFF = ((9 * kQChunk + 1023) / 1024) * 1024;
  static constexpr int R_OFF = V_OFF + kVSlots * kSlot;
  static constexpr int P_OFF = R_OFF + kRopeSlots * kSlot;
  static constexpr int BAR_OFF = P_OFF + kPBufs * N * 128;
  static constexpr int X_OFF = BAR_OFF + 256;              // float [4][N]: column maxima / sums of the four warps
  static constexpr int M_OFF = X_OFF + 4 * N * 4;          // float [N]: rescale factors, then 1 / l
  static constexpr int MISC_OFF = M_OFF + N * 4;
  static constexpr int VALID_OFF = MISC_OFF + 32;          // sparse modes: 64 validity bits per page in flight
  static constexpr int ROW_OFF = VALID_OFF + kPageBars * 8;        // int64 [N]: element offset of a row within a request's output
  static constexpr int SHARE_OFF = ROW_OFF + N * 8;
  static constexpr int SMEM_BYTES = SHARE_OFF + sizeof(RowShare);
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared memory limit per CTA");
  static_assert(kPBufs * N * 128 >= 4 * N * (N == 64 ? 16 : 32) * 2, "the P buffers stage the output rows of the four softmax warps");
  static_assert(kVSlots % 2 == 0 && kVSlots >= 16 && kVSlots <= 8 * (kPageBars - 1) + 1, "ring sizes");
};
enum Bar { Q_FULL = 0, Q_EMPTY, KV_FULL0, KV_EMPTY0 = KV_FULL0 + kPageBars, ROPE_EMPTY0 = KV_EMPTY0 + kPageBars, S_FULL0 = ROPE_EMPTY0 + 3, S_FULL1,
           P_FULL0, P_FULL1, O_FULL, NUM_BARS };
static_assert(NUM_BARS * 8 <= 256, "barrier area too small");
constexpr int TMEM_O = 0, TMEM_S = 256;
constexpr float kRescaleThreshold = 8.0f;         // log2 units; below it O keeps its stale scale
}  // namespace frt

__device__ int g_decode_few_status = 0;

struct FewParams {
  DecodeKernelParams d;
  int tokens_per_tile;         // > 0: a tile holds this many query tokens with all heads of the kv head; 0: 64 heads of one token
};

// 16 TMEM lanes x 8*K columns: registers 4k + {0,1} = row t/4, columns 8k + 2(t%4) + {0,1}; 4k + {2,3} = row t/4 + 8
template <int R>
__device__ __forceinline__ void tmem_ld_16x256b(uint32_t taddr, uint32_t (&v)[R]) {
  static_assert(R == 8 || R == 16 || R == 32, "x2, x4 or x8");
  if constexpr (R == 8) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
  } else if constexpr (R == 16) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                   "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
  } else {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
  }
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
// four 8x8 matrices of 16-bit elements, each stored transposed; lane i gives the address of row i % 8 of matrix i / 8
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}
// barrier over the 128 softmax threads that also tells whether any of them passed true
__device__ __forceinline__ bool bar_any(int id, bool x) {
  uint32_t r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %2, 0;\nbarrier.cta.red.or.aligned.pred q, %1, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
               : "=r"(r)
               : "r"(id), "r"(static_cast<uint32_t>(x))
               : "memory");
  return r != 0;
}

// What this CTA works on with k > 1 CTAs to a row of the schedule.  A CTA works on one request of the row: each request gets CTAs in
// proportion to its blocks, one at least; where there are more requests than CTAs the first takes them all.
__device__ __noinline__ void share_of_row(const DecodeKernelParams& p, int k, int lag_last, RowShare* out) {
  const int* md = p.tile_scheduler_metadata + blockIdx.z / k * 8;
  RowShare s = {*reinterpret_cast<const int4*>(md), md[4], k | 1 << 16};
  const int u = blockIdx.z % k, n = s.row.z - s.row.x + 1;
  if (s.row.x >= p.b || n > k) {
    if (u > 0) s.row.x = p.b;
    *out = s;
    return;
  }
  struct Blocks { int lo, hi; };
  auto blocks = [&](int i) {       // as `request` in the kernel
    const int batch = s.row.x + i, len = p.topk >= 0 ? p.topk : p.seqlens_k[batch], total = (len + 63) >> 6, seen = len - lag_last;
    Blocks r = {i == 0 ? s.row.y : 0, min(i == n - 1 ? min(s.row.w, total) : total, seen > 0 ? (seen + 63) >> 6 : 0)};
    r.hi = max(r.hi, r.lo);
    return r;
  };
  const Blocks r0 = blocks(0), r1 = blocks(n - 1);       // (their lengths are on the way together)
  auto of = [&](int i) { return i == 0 ? r0 : i == n - 1 ? r1 : blocks(i); };
  int total = 0, seen = 0, first = 0, w = 0, next = 0;
  for (int i = 0; i < n; ++i) { const Blocks r = of(i); total += r.hi - r.lo; }
  Blocks r;
  for (;; ++w) {
    r = of(w);
    seen += r.hi - r.lo;
    next = w == n - 1 ? k : min(max(total > 0 ? (k * seen + total / 2) / total : 0, first + 1), k - (n - 1 - w));
    if (u < next) break;
    first = next;
  }
  const int v = u - first, c = next - first, len = r.hi - r.lo;
  s.row = make_int4(s.row.x + w, r.lo + len * v / c, s.row.x + w, r.lo + len * (v + 1) / c);
  if (w > 0) s.split = 0;
  s.share = k | v << 8 | c << 16;
  *out = s;
}

// grid (row tiles, h_k, parts).  SHARED: rows of the schedule may be shared, which the schedule tells.  Calls in which none can be take the
// other form: with one for all they were 0.7 to 2 us slower (64 heads, top-k 2048, 30 requests 42.4 -> 44.2, 140 x 1 000 tokens 63.8 ->
// 65.4).
template <int MODE, int N, bool F16, bool SHARED>
__global__ void __launch_bounds__(frt::threads(MODE), 1)
mla_few_rows_kernel(const __grid_constant__ FewParams P, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv) {
  using namespace frt;
  using L = Layout<N>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  auto bar = [&](int i) { return sbase + L::BAR_OFF + i * 8; };
  float* sX = reinterpret_cast<float*>(smem + L::X_OFF);
  float* sM = reinterpret_cast<float*>(smem + L::M_OFF);
  int64_t* sRow = reinterpret_cast<int64_t*>(smem + L::ROW_OFF);
  volatile uint32_t* sTmem = reinterpret_cast<volatile uint32_t*>(smem + L::MISC_OFF);
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + L::MISC_OFF + 8);   // set by a softmax thread whose wait expired
  RowShare* sShare = reinterpret_cast<RowShare*>(smem + L::SHARE_OFF);
  int* status = &g_decode_few_status;
  const DecodeKernelParams& p = P.d;
  constexpr bool SPARSE = MODE == kSparseDecode;
  const float scale_log2 = p.scale_log2;
  volatile uint32_t* sValid = reinterpret_cast<volatile uint32_t*>(smem + L::VALID_OFF);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    // a page has landed: with its bytes (TMA), or when every gather warp has stored its rows
    constexpr int kFull = SPARSE ? kGather : 1;
    for (int i = 0; i < NUM_BARS; ++i)
      tc::mbar_init(bar(i), i == P_FULL0 || i == P_FULL1 ? 4                             // one arrival per softmax warp
                            : (i >= KV_FULL0 && i < KV_EMPTY0)              ? kFull : 1);
    tc::fence_mbar_init();
    *sAbort = 0;
  }
  if (warp == 5) tc::tmem_alloc(sbase + L::MISC_OFF, 512);
  if (warp == 4 && tc::elect_one()) {
    tc::prefetch_tensormap(&tmap_q);
    if constexpr (!SPARSE) tc::prefetch_tensormap(&tmap_kv);
  }
  // query rows that no TMA copy fills (a tile with fewer than N rows) stay zero
  for (int i = tid; i < 9 * L::kQChunk / 16; i += threads(MODE)) reinterpret_cast<uint4*>(smem + L::Q_OFF)[i] = make_uint4(0, 0, 0, 0);
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  // The schedule, the queries and the cache may come from the kernel in front of this one.  From here on plain loads (not
  // __ldg, which the compiler may move above the wait and whose path is undefined for memory that is written while this
  // kernel is resident) read the schedule, the lengths, the block table and the indices; the FP8 records hang on those.
  pdl_wait();
  pdl_allow_dependents();       // the merge kernel may become resident now
  const uint32_t tmem = *sTmem;

  // ---- the tile and the stretch of the schedule this CTA owns -----------------------------------
  const int hq = p.hq_per_hk, kh = blockIdx.y;
  int sq0 = 0, ntok = 1, hb = 0;
  if (P.tokens_per_tile > 0) {
    sq0 = blockIdx.x * P.tokens_per_tile;
    ntok = min(P.tokens_per_tile, p.s_q - sq0);
  } else {
    const int n_hb = (hq + 63) >> 6;
    sq0 = blockIdx.x / n_hb;
    hb = blockIdx.x % n_hb;
  }
  const int tile_heads = min(hq - hb * 64, 64), nrows = ntok * tile_heads, head0 = kh * hq + hb * 64;
  // dense: query token t of the sequence sees keys below seqlen - (s_q - 1 - t)
  const int lag_first = MODE == kDense && p.is_causal ? p.s_q - 1 - sq0 : 0, lag_last = MODE == kDense && p.is_causal ? p.s_q - sq0 - ntok : 0;
  const int* md_row = p.tile_scheduler_metadata + blockIdx.z * 8;
  if constexpr (SHARED) {
    if (tid == 0) {
      const int4 own = *reinterpret_cast<const int4*>(md_row);      // on the way together with what tells k
      const int split = md_row[4], k = sub_splits<true>(p);
      if (k == 1) *sShare = {own, split, 1 | 1 << 16};
      else share_of_row(p, k, lag_last, sShare);
    }
    __syncthreads();
    // One load for either case, from an address that is the same for all threads: where the row came out of a branch, or out of the
    // loops of share_of_row, the compiler took the loops of every role for divergent (32 heads, 7 x 22 000 tokens 47.7 -> 49.7 us).
    md_row = reinterpret_cast<const int*>(sShare);
  }
  const int4 md = *reinterpret_cast<const int4*>(md_row);
  const int begin_split = md_row[4];
  const int begin_idx = md.x, begin_block = md.y, end_idx = md.z, end_block = md.w;
  const int n_work = begin_idx >= p.b ? 0 : end_idx - begin_idx + 1;
  struct Req { int batch, seqlen, blk_lo, blk_hi; const int* idx; };
  auto request = [&](int wi) {
    Req r;
    r.batch = begin_idx + wi;
    r.seqlen = SPARSE ? p.topk : p.seqlens_k[r.batch];
    const int total = (r.seqlen + 63) >> 6, seen = r.seqlen - lag_last;
    r.blk_lo = r.batch == begin_idx ? begin_block : 0;
    r.blk_hi = min(r.batch == end_idx ? min(end_block, total) : total, seen > 0 ? (seen + 63) >> 6 : 0);
    if (r.blk_hi < r.blk_lo) r.blk_hi = r.blk_lo;
    r.idx = SPARSE ? p.indices + r.batch * p.indices_stride_b + sq0 * p.indices_stride_s : nullptr;
    return r;
  };
  const bool misaligned = (sbase & 1023u) != 0;      // the swizzled tiles need a 1024-byte aligned base
  if (misaligned && tid == 0) tc::report_status(status, 30);

  if (n_work == 0 || misaligned) {
    // nothing to do
  } else if (warp == 4) {
    // ================================ TMA producer =====================================
    if (tc::elect_one()) {
      int g = 0, req = 0, freed = 0, slot = 0;     // pages loaded, requests, pages whose slots are known to be free again, next slot
      bool alive = true;
      for (int wi = 0; wi < n_work && alive; ++wi) {
        const Req r = request(wi);
        if (r.blk_hi == r.blk_lo) continue;
        const int* bt = SPARSE ? nullptr : p.block_table + (int64_t)r.batch * p.block_table_stride_b;
        int page_next = SPARSE ? 0 : bt[r.blk_lo];      // on the way while the queries are asked for
        alive = tc::mbar_wait(bar(Q_EMPTY), (req & 1) ^ 1, status, 201);
        if (!alive) break;
        // the box of the map covers all rows of one token (rows past the tensor read as zero); 64-column chunks
        const int box_rows = P.tokens_per_tile > 0 ? hq : N;
        tc::mbar_arrive_expect_tx(bar(Q_FULL), ntok * box_rows * 1152);
        for (int t = 0; t < ntok; ++t)
#pragma unroll
          for (int c = 0; c < 9; ++c)
            tc::tma_load_4d(sbase + L::Q_OFF + c * L::kQChunk + t * hq * 128, &tmap_q, c * 64, head0, sq0 + t, r.batch, bar(Q_FULL));
        ++req;
        if constexpr (SPARSE) continue;
        const bool ahead = r.blk_hi - r.blk_lo >= kPrefetchBlocks && p.k_stride_row == 576;
        const char* kv_head = reinterpret_cast<const char*>(p.kcache) + kh * p.k_stride_head * 2;
        for (int blk = r.blk_lo; blk < r.blk_hi && alive; ++blk, ++g) {
          const int page = page_next, full = bar(KV_FULL0 + g % kPageBars);
          if (blk + 1 < r.blk_hi) page_next = bt[blk + 1];
          alive = tc::mbar_wait(bar(ROPE_EMPTY0 + g % L::kRopeSlots), ((g / L::kRopeSlots) & 1) ^ 1, status, 202);
          if (!alive) break;
          // (page g - 4 has left the ring before page g starts to enter it, so its full barrier has turned over)
          tc::mbar_arrive_expect_tx(full, kPageBytes);
          tc::tma_load_4d(sbase + L::R_OFF + (g % L::kRopeSlots) * kSlot, &tmap_kv, 512, kh, 0, page, full);
          // the next page, as one piece: the tiles read it 128 bytes of a row at a time, and their slots are only free a page later
          // (an entry of the block table that is no page: the loads read zeros there, a bare address would be one past the cache)
          if (ahead && blk + 1 < r.blk_hi && static_cast<unsigned>(page_next) < static_cast<unsigned>(p.num_blocks))
            prefetch_l2(kv_head + page_next * p.k_stride_block * 2, kPageBytes);
#pragma unroll 1
          for (int c = 0; c < 8 && alive; ++c) {
            const int n = g * 8 + c;               // chunk n takes the slot of chunk n - kVSlots, i.e. of page (n - kVSlots) / 8
            while (alive && freed * 8 <= n - L::kVSlots) {
              alive = tc::mbar_wait(bar(KV_EMPTY0 + freed % kPageBars), (freed / kPageBars) & 1, status, 203);
              ++freed;
            }
            if (alive) tc::tma_load_4d(sbase + L::V_OFF + slot * kSlot, &tmap_kv, c * 64, kh, 0, page, full);
            if (++slot == L::kVSlots) slot = 0;
          }
        }
      }
    }
  } else if (SPARSE && warp >= 6) {
    // ================================ gather producers =================================
    // Page g takes its slots when P V of page g - 2 has completed (the ring holds at least two pages).
    const int gw = warp - 6;
    auto page_free = [&](int g) {
      return g < 2 || __all_sync(0xffffffffu, tc::mbar_wait(bar(KV_EMPTY0 + (g - 2) % kPageBars), ((g - 2) / kPageBars) & 1, status, 204));
    };
    auto slot_of = [&](int g, int chunk) {      // shared memory address of 64-column chunk `chunk` of page g
      return sbase + (chunk < 8 ? L::V_OFF + ((g * 8 + chunk) % L::kVSlots) * kSlot : L::R_OFF + (g % L::kRopeSlots) * kSlot);
    };
    if constexpr (SPARSE) {
      // Eight records per warp and block: the 32 lanes read the 32 pieces of e4m3 values, their tile's scale, and 8 lanes
      // the bf16 rope part.  The records of a block are read one block ahead and its indices two blocks ahead of the
      // stores: a warp executes in order, and looking at an index right after its load costs a memory latency.
      const unsigned char* cache = reinterpret_cast<const unsigned char*>(p.kcache);
      uint4 nope[8], rope[8];
      float scl[8];
      auto to_slot = [&](int v, int batch) {
        if (p.indices_logical) {       // token position of the request -> physical slot through its block table
          const int pos = v;
          v = -1;
          if (pos >= 0 && pos < p.seqlens_k[batch]) v = p.block_table[batch * p.block_table_stride_b + (pos >> 6)] * 64 + (pos & 63);
        }
        return (v < 0 || v >= p.num_blocks * 64) ? -1 : v;
      };
      int c_wi = 0, c_blk = 0;         // position of the index reader in the block list of this CTA
      Req c_r = request(0);
      auto skip = [&] {
        while (c_wi < n_work && c_blk >= c_r.blk_hi) {
          ++c_wi;
          if (c_wi < n_work) { c_r = request(c_wi); c_blk = c_r.blk_lo; }
        }
      };
      c_blk = c_r.blk_lo;
      skip();
      int raw = -1, raw_batch = 0;
      auto read_indices = [&] {        // lanes 0..7: row 8 gw + lane of the next unread block
        if (c_wi >= n_work) return false;
        raw = c_r.idx[c_blk * 64 + gw * 8 + (lane & 7)];
        raw_batch = c_r.batch;
        ++c_blk;
        skip();
        return true;
      };
      uint32_t valid = 0;
      auto read_records = [&] {
        const int my_slot = to_slot(raw, raw_batch);
        valid = __ballot_sync(0xffffffffu, my_slot >= 0) & 0xffu;
#pragma unroll
        for (int rr = 0; rr < 8; ++rr) {
          const int slot = __shfl_sync(0xffffffffu, my_slot, rr);
          nope[rr] = make_uint4(0, 0, 0, 0);
          rope[rr] = make_uint4(0, 0, 0, 0);
          scl[rr] = 0.f;
          if (slot >= 0) {
            const unsigned char* rec = cache + (int64_t)(slot >> 6) * p.k_stride_block + (slot & 63) * p.k_stride_row;
            nope[rr] = __ldg(reinterpret_cast<const uint4*>(rec) + lane);
            scl[rr] = __ldg(reinterpret_cast<const float*>(rec + 512) + (lane >> 3));
            if (lane < 8) rope[rr] = __ldg(reinterpret_cast<const uint4*>(rec + 528) + lane);
          }
        }
      };
      int g = 0;
      bool alive = true, have = read_indices();
      if (have) read_records();
      bool have_next = have && read_indices();
      while (have && alive) {
        alive = page_free(g);
        if (!alive) break;
        const uint32_t nbase = slot_of(g, lane >> 2), rbase = slot_of(g, 8);
#pragma unroll
        for (int rr = 0; rr < 8; ++rr) {
          const int row = gw * 8 + rr;
          const float scale = scl[rr];
          const uint32_t w[4] = {nope[rr].x, nope[rr].y, nope[rr].z, nope[rr].w};
          uint32_t o[8];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            // 4 e4m3 bytes -> 4 floats (exact), * scale in fp32, round to bf16
            const __half2_raw h01 = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w[k] & 0xffffu), __NV_E4M3);
            const __half2_raw h23 = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w[k] >> 16), __NV_E4M3);
            const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&h01));
            const float2 f23 = __half22float2(*reinterpret_cast<const __half2*>(&h23));
            o[k * 2] = pack_bf16x2(f01.x * scale, f01.y * scale);
            o[k * 2 + 1] = pack_bf16x2(f23.x * scale, f23.y * scale);
          }
          // pieces 2 lane and 2 lane + 1 of the row: chunk lane / 4, places 2 (lane % 4) and the next one, swizzled by row % 8 == rr
          st_shared_v4(nbase + row * 128 + ((((lane & 3) * 2) ^ rr) << 4), make_uint4(o[0], o[1], o[2], o[3]));
          st_shared_v4(nbase + row * 128 + ((((lane & 3) * 2 + 1) ^ rr) << 4), make_uint4(o[4], o[5], o[6], o[7]));
          if (lane < 8) st_shared_v4(rbase + row * 128 + ((lane ^ rr) << 4), rope[rr]);
        }
        if (lane == 0) reinterpret_cast<volatile uint8_t*>(sValid)[(g % kPageBars) * 8 + gw] = static_cast<uint8_t>(valid);
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(KV_FULL0 + g % kPageBars));
        ++g;
        have = have_next;
        if (have) {
          read_records();
          have_next = read_indices();
        }
      }
    }
  } else if (warp == 5) {
    // ================================ MMA issuer =======================================
    // One thread.  As a warp with a vote on every wait: 16 heads, 61 x 6 000 tokens 78.6 us, 75.9 now, 60 x 300 17.6 -> 15.5, 32 heads,
    // 32 x 500 21.8 -> 20.4, 64 heads, 8 x 3 000 22.7 -> 22.2, sparse, 64 heads, 30 x top-k 2 048 40.7 -> 39.9, 2 x 512 14.65 -> 14.8.
    if (tc::elect_one()) {
      constexpr uint32_t idesc_s = tc::idesc_bf16_f32(64, N, 0, 0, F16);
      constexpr uint32_t idesc_o = tc::idesc_bf16_f32(128, N, 1, 0, F16);
      const uint64_t desc_q = tc::smem_desc_sw128(sbase + L::Q_OFF, 16, 1024);        // B of S^T: K-major
      const uint64_t desc_k = tc::smem_desc_sw128(sbase + L::V_OFF, 16, 1024);        // A of S^T: K-major (slot 0)
      const uint64_t desc_r = tc::smem_desc_sw128(sbase + L::R_OFF, 16, 1024);        // the same, rope slot 0
      const uint64_t desc_v = tc::smem_desc_sw128(sbase + L::V_OFF, kSlot, 1024);     // A of O^T: MN-major, 64-wide column groups 8 KB apart
      const uint64_t desc_p = tc::smem_desc_sw128(sbase + L::P_OFF, 16, 1024);        // B of O^T: K-major
      int g = 0, req = 0;
      int slot_s = 0, slot_p = 0;      // first slot of the page of the next S^T / O^T (running: a division would cost more than the MMAs of a chunk)
      auto next_page = [](int slot) { return slot + 8 >= L::kVSlots ? slot + 8 - L::kVSlots : slot + 8; };
      auto wrap = [](int slot) { return slot >= L::kVSlots ? slot - L::kVSlots : slot; };
      bool alive = true;
      for (int wi = 0; wi < n_work && alive; ++wi) {
        const Req r = request(wi);
        const int nblk = r.blk_hi - r.blk_lo;
        if (nblk == 0) continue;
        alive = tc::mbar_wait(bar(Q_FULL), req & 1, status, 205);
        // S^T runs one block ahead of O^T; where both could be next, whichever has its inputs first is issued, O^T first: it
        // releases slots of the ring.  S^T(js) overwrites S^T(js - 2), and O^T(0) what the request before left: the softmax
        // warps had read both before they arrived on a P_FULL that has been waited for here (P_FULL(js - 2), P_FULL(0)).
        int js = 0, jp = 0, idle = 0;
        while (jp < nblk && alive) {
          const int gs = g + js, gp = g + jp;
          const bool want_s = js < nblk && js <= jp + 1, want_p = jp < js;
          const uint32_t p_full = bar(P_FULL0 + gp % L::kPBufs), kv_full = bar(KV_FULL0 + gs % kPageBars);
          const uint32_t p_ph = (gp / L::kPBufs) & 1, kv_ph = (gs / kPageBars) & 1;
          bool go_p = false, go_s = false;
          if (want_s && want_p) {
            go_p = tc::mbar_test_wait(p_full, p_ph);
            if (!go_p) go_s = tc::mbar_test_wait(kv_full, kv_ph);
          } else if (want_p) {
            go_p = alive = tc::mbar_wait(p_full, p_ph, status, 207);
          } else {
            go_s = alive = tc::mbar_wait(kv_full, kv_ph, status, 212);
          }
          if (go_p) {
            tc::tc_fence_after();
            const uint64_t dp = tc::desc_advance(desc_p, (gp % L::kPBufs) * N * 128);
#pragma unroll
            for (int mb = 0; mb < 4; ++mb) {
              const uint64_t dv = tc::desc_advance(desc_v, wrap(slot_p + mb * 2) * kSlot);
#pragma unroll
              for (int s = 0; s < 4; ++s)
                tc::mma_ss(tmem + TMEM_O + mb * N, tc::desc_advance(dv, s * 2048), tc::desc_advance(dp, s * 32), idesc_o, (jp == 0 && s == 0) ? 0u : 1u);
            }
            tc::tc_commit(bar(KV_EMPTY0 + gp % kPageBars));
            slot_p = next_page(slot_p);
            ++jp;
            idle = 0;
          } else if (go_s) {
            tc::tc_fence_after();
            const uint32_t d = tmem + TMEM_S + (gs & 1) * N;
#pragma unroll
            for (int c = 0; c < 9; ++c) {
              const uint64_t da = c < 8 ? tc::desc_advance(desc_k, wrap(slot_s + c) * kSlot)
                                        : tc::desc_advance(desc_r, (gs % L::kRopeSlots) * kSlot);
#pragma unroll
              for (int s = 0; s < 4; ++s)
                tc::mma_ss(d, tc::desc_advance(da, s * 32), tc::desc_advance(desc_q, c * L::kQChunk + s * 32), idesc_s, (c | s) ? 1u : 0u);
            }
            tc::tc_commit(bar(S_FULL0 + (gs & 1)));
            tc::tc_commit(bar(ROPE_EMPTY0 + gs % L::kRopeSlots));
            if (js == nblk - 1) tc::tc_commit(bar(Q_EMPTY));
            slot_s = next_page(slot_s);
            ++js;
            idle = 0;
          } else if (alive && ++idle > tc::kSpinLimit) {
            tc::report_status(status, 206);
            alive = false;
          }
        }
        g += nblk;
        if (alive) tc::tc_commit(bar(O_FULL));
        ++req;
      }
    }
  } else {
    // ================================ softmax / epilogue ================================
    constexpr int K8 = N / 8;                            // groups of 8 columns
    const uint32_t lane_addr = static_cast<uint32_t>(warp * 32) << 16;
    const int t4 = lane & 3, tr = lane >> 2;
    // Where row `tid` of the tile goes: one division per row and CTA (it is read after the barriers of an epilogue).
    const int my_tok = sq0 + tid / tile_heads, my_head = head0 + tid % tile_heads;
    if (tid < N) sRow[tid] = my_tok * p.o_stride_s + my_head * p.o_stride_h;
    int g = 0, req = 0;
    bool aborted = false;        // uniform over the 128 softmax threads: only read right after a barrier
    for (int wi = 0; wi < n_work; ++wi) {
      const Req r = request(wi);
      const int nblk = r.blk_hi - r.blk_lo;
      const int lo = p.num_splits[r.batch], hi = p.num_splits[r.batch + 1];      // here: their latency hides behind the blocks
      // per column of this thread: the scale O^T and l carry (-inf: no visible key yet), and its share of the row sum
      float m_used[K8][2], l_part[K8][2];
#pragma unroll
      for (int k = 0; k < K8; ++k) { m_used[k][0] = m_used[k][1] = neg_inf(); l_part[k][0] = l_part[k][1] = 0.f; }
      for (int j = 0; j < nblk; ++j, ++g) {
        uint32_t sv[4 * K8];
        if (tc::mbar_wait(bar(S_FULL0 + (g & 1)), (g >> 1) & 1, status, 208)) {
          __syncwarp();
          tc::tc_fence_after();
          tmem_ld_16x256b(tmem + lane_addr + TMEM_S + (g & 1) * N, sv);
          tc::tmem_wait_ld();
          tc::tc_fence_before();
        } else {
          *sAbort = 1;
#pragma unroll
          for (int i = 0; i < 4 * K8; ++i) sv[i] = 0u;
        }
        // logits of hidden tokens become -inf (a select: they may hold anything)
        const int blk0 = (r.blk_lo + j) * 64, tok0 = blk0 + warp * 16 + tr;
        if constexpr (SPARSE) {
          const uint32_t v = sValid[(g % kPageBars) * 2 + (warp >> 1)] >> ((warp & 1) * 16);      // this warp's 16 tokens
          if ((v & 0xffffu) != 0xffffu) {
#pragma unroll
            for (int k = 0; k < K8; ++k)
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                if (!((v >> tr) & 1u)) sv[4 * k + c] = 0xff800000u;
                if (!((v >> (tr + 8)) & 1u)) sv[4 * k + 2 + c] = 0xff800000u;
              }
          }
        } else if (blk0 + 64 > r.seqlen - lag_first) {
          // rows of the last page beyond the sequence may hold anything (NaN included): zeroed, now that S^T has read them, so that
          // 0 * garbage cannot reach O^T
          const int rows_valid = r.seqlen - blk0;
          for (int i = tid; i < (64 - rows_valid) * 64; i += 128) {
            const int row = rows_valid + (i >> 6), c = (i >> 3) & 7, piece = i & 7;
            *reinterpret_cast<uint4*>(smem + L::V_OFF + (g * 8 + c) % L::kVSlots * kSlot + row * 128 + piece * 16) = make_uint4(0, 0, 0, 0);
          }
#pragma unroll
          for (int k = 0; k < K8; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int row = 8 * k + 2 * t4 + c;
              const int border = r.seqlen - (p.is_causal ? max(lag_first - row / hq, 0) : 0);   // row / hq: the token within the tile
              if (tok0 >= border) sv[4 * k + c] = 0xff800000u;
              if (tok0 + 8 >= border) sv[4 * k + 2 + c] = 0xff800000u;
            }
        }
        bool need = false;
#pragma unroll
        for (int k = 0; k < K8; ++k)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const float mx = fmaxf(__uint_as_float(sv[4 * k + c]), __uint_as_float(sv[4 * k + 2 + c])) * scale_log2;
            need |= mx > m_used[k][c] + kRescaleThreshold;
          }
        const bool any_need = bar_any(1, need);
        if (*sAbort) { aborted = true; break; }            // every wait that can expire lies before the barrier or one block back
        if (any_need) {
          // maxima of the block per column: over the 8 row pairs of the warp, then over the four warps
#pragma unroll
          for (int k = 0; k < K8; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              float mx = fmaxf(__uint_as_float(sv[4 * k + c]), __uint_as_float(sv[4 * k + 2 + c])) * scale_log2;
#pragma unroll
              for (int off = 4; off <= 16; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
              if (lane < 4) sX[warp * N + 8 * k + 2 * t4 + c] = mx;
            }
          bar_sync(1, 128);
          bool moved = false;
#pragma unroll
          for (int k = 0; k < K8; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int col = 8 * k + 2 * t4 + c;
              const float mx = fmaxf(fmaxf(sX[col], sX[N + col]), fmaxf(sX[2 * N + col], sX[3 * N + col]));
              const bool up = mx > m_used[k][c] + kRescaleThreshold;
              // the first visible key sets the scale: O^T and l are exactly zero so far
              const float alpha = (up && m_used[k][c] != neg_inf()) ? exp2f(m_used[k][c] - mx) : 1.f;
              moved |= alpha != 1.f;
              l_part[k][c] *= alpha;
              if (up) m_used[k][c] = mx;
              if (warp == 0 && lane < 4) sM[col] = alpha;
            }
          if (bar_any(1, moved)) {
            // every earlier O^T product must be complete (they complete in order)
            const int gl = g - 1;
            if (!tc::mbar_wait(bar(KV_EMPTY0 + gl % kPageBars), (gl / kPageBars) & 1, status, 209)) *sAbort = 1;
            __syncwarp();
            tc::tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 4 * N; c += 16) {
              uint32_t ov[16];
              tc::tmem_ld16(tmem + lane_addr + TMEM_O + c, ov);
              tc::tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * sM[(c % N) + i]);
              tc::tmem_st16(tmem + lane_addr + TMEM_O + c, ov);
            }
            tc::tmem_wait_st();
            tc::tc_fence_before();
          }
        }
        uint32_t pk[2 * K8];      // [2k]: tokens tr, [2k + 1]: tokens tr + 8, columns 8k + 2 t4 + {0,1}
#pragma unroll
        for (int k = 0; k < K8; ++k) {
          const float m0 = m_used[k][0] == neg_inf() ? 0.f : m_used[k][0], m1 = m_used[k][1] == neg_inf() ? 0.f : m_used[k][1];
          const float p00 = exp2f(fmaf(__uint_as_float(sv[4 * k]), scale_log2, -m0));
          const float p01 = exp2f(fmaf(__uint_as_float(sv[4 * k + 1]), scale_log2, -m1));
          const float p10 = exp2f(fmaf(__uint_as_float(sv[4 * k + 2]), scale_log2, -m0));
          const float p11 = exp2f(fmaf(__uint_as_float(sv[4 * k + 3]), scale_log2, -m1));
          l_part[k][0] += p00 + p10;
          l_part[k][1] += p01 + p11;
          pk[2 * k] = pack_16x2<F16>(p00, p01);
          pk[2 * k + 1] = pack_16x2<F16>(p10, p11);
        }
        // the P buffer is free: O^T of the block that had it is complete
        if (const int gb = g - L::kPBufs; gb >= 0 && !tc::mbar_wait(bar(KV_EMPTY0 + gb % kPageBars), (gb / kPageBars) & 1, status, 210)) *sAbort = 1;
        __syncwarp();
        // P[column][token] as the K-major 128B-swizzled B operand: 16-byte chunk (2 warp + half) ^ (column & 7) of row `column`
        const uint32_t pbase = sbase + L::P_OFF + (g % L::kPBufs) * N * 128;
        const int mrow = lane & 7, mat = lane >> 3;         // this lane's matrix: token half mat & 1, column group + (mat >> 1)
#pragma unroll
        for (int k = 0; k < K8; k += 2)
          stmatrix_x4_trans(pbase + ((k + (mat >> 1)) * 8 + mrow) * 128 + (((warp * 2 + (mat & 1)) ^ mrow) << 4), pk[2 * k], pk[2 * k + 1],
                            pk[2 * k + 2], pk[2 * k + 3]);
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(P_FULL0 + g % L::kPBufs));
      }

      // ---- epilogue of this work item ---------------------------------------------------
      bar_sync(1, 128);
      int k = 1, share = 0, given = 1;
      if constexpr (SHARED) { k = sShare->share & 0xff; share = sShare->share >> 8 & 0xff; given = sShare->share >> 16; }
      const bool no_split = !p.force_partial && hi - lo == 1 && k == 1;
      const int64_t slot = static_cast<int64_t>(lo + (r.batch == begin_idx ? begin_split : 0)) * k + share;
      const int64_t part_row = (slot * p.h_k + kh) * (int64_t)p.s_q * hq + sq0 * hq + hb * 64;      // row 0 of the tile in its partial slot
      if (*sAbort) aborted = true;
      if (aborted) break;
#pragma unroll
      for (int k = 0; k < K8; ++k)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float s = l_part[k][c];
#pragma unroll
          for (int off = 4; off <= 16; off <<= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
          if (lane < 4) sX[warp * N + 8 * k + 2 * t4 + c] = s;
          if (lane < 4 && warp == 0) sM[8 * k + 2 * t4 + c] = m_used[k][c];
        }
      bar_sync(1, 128);
      float l = 0.f, m = 0.f;
      if (tid < N) {
        l = (sX[tid] + sX[N + tid]) + (sX[2 * N + tid] + sX[3 * N + tid]);
        m = sM[tid];
      }
      bar_sync(1, 128);
      if (tid < N) {
        sM[tid] = (l == 0.f || nblk == 0) ? 0.f : 1.f / l;
        if (tid < nrows) {
          if (no_split) {
            p.softmax_lse[((int64_t)r.batch * p.h_q + my_head) * p.s_q + my_tok] = l == 0.f ? pos_inf() : (log2f(l) + m) * kLn2;
          } else {
            p.lse_accum[part_row + tid] = l == 0.f ? neg_inf() : log2f(l) + m;
            if (SHARED && share == 0)                      // slots of this request that no CTA has been given
              for (int i = given; i < k; ++i) p.lse_accum[part_row + (int64_t)i * p.h_k * p.s_q * hq + tid] = neg_inf();
            if (p.no_split_hint && tid == 0) tc::report_status(status, 41);     // a split request although the caller ruled it out
          }
        }
      }
      bool have_o = nblk > 0;
      if (have_o) {
        if (!tc::mbar_wait(bar(O_FULL), req & 1, status, 211)) { *sAbort = 1; have_o = false; }
        __syncwarp();
        tc::tc_fence_after();
      }
      bar_sync(1, 128);
      if (*sAbort) { aborted = true; break; }
      if (no_split) {
        // 16-bit rows, through the P buffers (free: every P V of the request has completed).  A warp transposes W of its 32 value
        // columns at a time with stmatrix and stores rows in 16-byte pieces, a full 32-byte sector or two per row.
        // Scattered from the lanes' columns 4 bytes at a time, 64 unsplit rows took 13 000 clk, against 4 600 now.
        constexpr int W = N == 64 ? 16 : 32, kPieces = W / 8;
        const uint32_t stage = sbase + L::P_OFF + warp * (N * W * 2);
        auto piece_at = [&](int row, int piece) {      // swizzled so that eight rows of one piece fall into different banks
          return stage + row * (W * 2) + ((piece ^ (W == 16 ? (row >> 2) & 1 : (row >> 1) & 3)) << 4);
        };
        float2 inv[K8];
#pragma unroll
        for (int k = 0; k < K8; ++k) inv[k] = *reinterpret_cast<const float2*>(sM + 8 * k + 2 * t4);
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + r.batch * p.o_stride_b + warp * 32;
#pragma unroll 1
        for (int c = 0; c < 512 / 4 / W; ++c) {          // 128 mb + 32 warp + W part
          const int mb = c / (32 / W), part = c % (32 / W);
#pragma unroll
          for (int h = 0; h < W / 16; ++h) {
            uint32_t ov[4 * K8];
            if (have_o) {
              tmem_ld_16x256b(tmem + lane_addr + (static_cast<uint32_t>(part * W + h * 16) << 16) + TMEM_O + mb * N, ov);
              tc::tmem_wait_ld();
            } else {
#pragma unroll
              for (int i = 0; i < 4 * K8; ++i) ov[i] = 0u;
            }
            uint32_t pk[2 * K8];
#pragma unroll
            for (int k = 0; k < K8; ++k) {
              pk[2 * k] = pack_16x2<F16>(__uint_as_float(ov[4 * k]) * inv[k].x, __uint_as_float(ov[4 * k + 1]) * inv[k].y);
              pk[2 * k + 1] = pack_16x2<F16>(__uint_as_float(ov[4 * k + 2]) * inv[k].x, __uint_as_float(ov[4 * k + 3]) * inv[k].y);
            }
            const int mrow = lane & 7, mat = lane >> 3;
#pragma unroll
            for (int k = 0; k < K8; k += 2)
              stmatrix_x4_trans(piece_at((k + (mat >> 1)) * 8 + mrow, h * 2 + (mat & 1)), pk[2 * k], pk[2 * k + 1], pk[2 * k + 2], pk[2 * k + 3]);
          }
          __syncwarp();
          constexpr int kEach = N * kPieces / 32;
          uint4 v[kEach];
          int64_t at[kEach];
#pragma unroll
          for (int i = 0; i < kEach; ++i) {
            const int row = (i * 32 + lane) / kPieces, piece = lane % kPieces;
            v[i] = ld_shared_v4(piece_at(row, piece));
            at[i] = sRow[row] + mb * 128 + part * W + piece * 8;
          }
#pragma unroll
          for (int i = 0; i < kEach; ++i)
            if ((i * 32 + lane) / kPieces < nrows) *reinterpret_cast<uint4*>(out + at[i]) = v[i];
          __syncwarp();
        }
      } else {
        // fp32 partial: lane = value column 128 mb + 32 warp + lane, registers = query rows
#pragma unroll 1
        for (int c = 0; c < 4 * N; c += 16) {
          const int mb = c / N, row0 = c % N;
          if (row0 >= nrows) continue;
          uint32_t ov[16];
          if (have_o) {
            tc::tmem_ld16(tmem + lane_addr + TMEM_O + c, ov);
            tc::tmem_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) ov[i] = 0u;
          }
          // the factors are read before the first store: the compiler keeps a load behind the stores in front of it, and each
          // store then cost the latency of one (64 rows: 8 700 clk, now 5 200)
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 f = *reinterpret_cast<const float4*>(sM + row0 + i);
            ov[i] = __float_as_uint(__uint_as_float(ov[i]) * f.x);
            ov[i + 1] = __float_as_uint(__uint_as_float(ov[i + 1]) * f.y);
            ov[i + 2] = __float_as_uint(__uint_as_float(ov[i + 2]) * f.z);
            ov[i + 3] = __float_as_uint(__uint_as_float(ov[i + 3]) * f.w);
          }
          float* dst = p.o_accum + (part_row + row0) * 512 + mb * 128 + warp * 32 + lane;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (row0 + i < nrows) dst[i * 512] = __uint_as_float(ov[i]);
        }
      }
      if (nblk > 0) {
        tc::tc_fence_before();
        ++req;
      }
      bar_sync(1, 128);          // sM and sX are reused by the next request
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if (warp == 5) tc::tmem_dealloc(tmem, 512);
}

// ---- host side ----------------------------------------------------------------------------------
template <int MODE, int N, bool F16 = false>
static cudaError_t launch_few(const FewParams& P, const CUtensorMap& tq, const CUtensorMap& tkv, dim3 grid, cudaStream_t stream) {
  auto launch = [&](auto shared) {
    constexpr auto kern = mla_few_rows_kernel<MODE, N, F16, decltype(shared)::value>;
    if (cudaError_t e = allow_smem<kern>(frt::Layout<N>::SMEM_BYTES); e != cudaSuccess) return e;
    return launch_dependent(kern, grid, frt::threads(MODE), frt::Layout<N>::SMEM_BYTES, stream, P, tq, tkv);
  };
  return P.d.sub_split ? launch(std::true_type{}) : launch(std::false_type{});
}

cudaError_t launch_decode_few_rows(const DecodeKernelParams& p, cudaStream_t stream) {
  FewParams P = {};
  P.d = p;
  // whole query tokens share a tile when their heads fill whole 8-row groups of the swizzled operand tile
  const bool fold = p.hq_per_hk < 64 && p.hq_per_hk % 8 == 0;
  P.tokens_per_tile = fold ? 64 / p.hq_per_hk : 0;
  const int tile_tokens = fold ? (p.s_q < P.tokens_per_tile ? p.s_q : P.tokens_per_tile) : 1;
  const int rows = fold ? tile_tokens * p.hq_per_hk : (p.hq_per_hk < 64 ? p.hq_per_hk : 64);
  const int tiles = fold ? (p.s_q + P.tokens_per_tile - 1) / P.tokens_per_tile : p.s_q * ((p.hq_per_hk + 63) / 64);
  const int n = rows <= 16 ? 16 : rows <= 32 ? 32 : 64;
  CUtensorMap tq, tkv;
  // q [b][s_q][h_q][576]; cache [num_blocks][64][h_k][576] as (col, head, row in page, page), one map type for bf16 and fp16
  if (!tmah::make_map_4d(&tq, p.q, p.h_q, p.s_q, p.b, p.q_stride_h, p.q_stride_s, p.q_stride_b, fold ? p.hq_per_hk : n, 1)) return cudaErrorInvalidValue;
  if (!tmah::make_map_4d(&tkv, p.kcache, p.h_k, 64, p.num_blocks, p.k_stride_head, p.k_stride_row, p.k_stride_block, 1, 64)) return cudaErrorInvalidValue;
  const dim3 grid(tiles, p.h_k, p.num_sm_parts);
  if (p.is_f16) {
    if (n == 16) return launch_few<kDense, 16, true>(P, tq, tkv, grid, stream);
    if (n == 32) return launch_few<kDense, 32, true>(P, tq, tkv, grid, stream);
    return launch_few<kDense, 64, true>(P, tq, tkv, grid, stream);
  }
  if (n == 16) return launch_few<kDense, 16>(P, tq, tkv, grid, stream);
  if (n == 32) return launch_few<kDense, 32>(P, tq, tkv, grid, stream);
  return launch_few<kDense, 64>(P, tq, tkv, grid, stream);
}

cudaError_t launch_decode_sparse_few_rows(const DecodeKernelParams& p, cudaStream_t stream) {
  FewParams P = {};
  P.d = p;
  const int rows = p.hq_per_hk < 64 ? p.hq_per_hk : 64, n = rows <= 16 ? 16 : rows <= 32 ? 32 : 64;
  CUtensorMap tq;
  if (!tmah::make_map_4d(&tq, p.q, p.h_q, p.s_q, p.b, p.q_stride_h, p.q_stride_s, p.q_stride_b, n, 1)) return cudaErrorInvalidValue;
  const dim3 grid(p.s_q * ((p.hq_per_hk + 63) / 64), 1, p.num_sm_parts);
  if (n == 16) return launch_few<kSparseDecode, 16>(P, tq, tq, grid, stream);      // the cache is not read through a map
  if (n == 32) return launch_few<kSparseDecode, 32>(P, tq, tq, grid, stream);
  return launch_few<kSparseDecode, 64>(P, tq, tq, grid, stream);
}

cudaError_t set_status_mirror_few_rows(int* mapped_host_word) { return tc::set_status_mirror(mapped_host_word); }

cudaError_t read_decode_few_rows_status(int* host_status, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(host_status, g_decode_few_status, sizeof(int));
  if (e != cudaSuccess) return e;
  if (reset && *host_status != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_decode_few_status, &zero, sizeof(int));
  }
  return e;
}

}  // namespace fmla
