// MLA attention for 64 query rows per CTA on sm_100a (tcgen05 / TMA / tensor memory), the rows being the rows of an M = 64 tile:
//   kSparsePrefillCut sparse prefill forward with 64 heads: top-k row indices into kv[s_kv, 576], rows gathered with cp.async by
//                  eight producer warps.  128 heads take the CTA pair (mla_pair.cu).
//   kDense         dense split-KV decode where several 64-row tiles read the same pages and no pair takes them: three or more
//                  query tokens of 64 heads, 96 or 192 heads.  Whichever tile is first pulls a page into L2 (six ahead), the others
//                  find it there.
//
// One CTA = the 64-head tile of one query token (at a time).
//   warps 0-3 softmax : TMEM S -> registers, mask, running max / sum (base 2), P (16 bits) -> shared
//                       memory, lazy rescale of O in TMEM, final 1/l normalisation and stores
//   warp 4   TMA      : Q tile (9 boxes of 64 rows x 64 cols); kDense also the pages
//   warp 5   MMA      : one thread: S = Q K^T (36 x tcgen05.mma.ws m64n64k16, 24 of them with A in tensor memory) -> TMEM S[block & 1]
//                       O += P V   ( 8 x tcgen05.mma.ws m64n256k16) -> TMEM O
//                       V is the first 512 columns of the same K tile, read MN-major
//   warps 6-13 gather : kSparsePrefillCut; write K rows in the layout TMA produces (64-column chunks of 128-byte rows, 128-byte
//                       swizzle)
// A block goes through shared memory in halves: columns 0..255 and 256..511 in a ring of five 32 KB stages, the last 64 in three slots
// of their own.  That there is room for two and a half blocks beside the P buffers is due to Q: its chunks 0..5 live in the 192
// columns of tensor memory that O and S leave idle, and pass through two stages on their way there.  S starts on the first half while
// the second is gathered, and P V releases half by half.
// What bounds it: the chain of a block (with trace points: gather 1 500 to 2 000 clk, of which 1 150 are the 64 bytes a clock that an SM
// takes from L2; S 1 050; softmax 1 500; P V 650) over two and a half blocks in flight: 2 560 clk a block (148 tokens, top-k 2048, one time
// stamp per block), against 1 700 of tensor pipe.  With two whole pages as stages and a polling issuer it was 3 300.  333 tokens, top-k 512 51.3 -> 45.3 us, 4096, top-k 2048 1 765 -> 1 456; dense,
// 64 heads x 3 tokens, 16 x 3 000 53.8 -> 45.4; a call of one or two blocks is up to 0.4 us slower than with whole pages (one token, top-k
// 128, 8.9 -> 9.3), for the copy of Q.
// The transposed products of mla_few_rows.cu were measured slower in the prefill (333 query tokens, top-k 512: 105 us against 64 us then).
// TMEM map (512 columns allocated): O = [0,256) (two N=256 halves of 128 columns), S[0] = [256,288), S[1] = [288,320), Q chunks 0..5 =
// [320,512).  In the M=64 weight-stationary layout element
// (row r, col c) of an N-wide result sits in lane r + 64*(c >= N/2), column c % (N/2).
//
// Semantics follow the reference kernels: sparse prefill csrc/sm100/prefill/sparse/fwd.cu:399-417, 438-445, 677-679; decode
// borders / split outputs / LSE conventions csrc/sm90/decode/dense/splitkv_mla.cu:948-957, 1022-1042, 1237-1269.
// Every mbarrier wait is bounded (tc_common.cuh); a pipeline fault sets a status word and lets the
// CTA drain and free its tensor memory.
#include "kernels.h"
#include "launch.cuh"
#include "mla_work.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

#include <cuda.h>

namespace fmla {

namespace dtc {
constexpr int kChunkBytes = 64 * 128;             // [64 rows x 64 bf16], 128-byte rows
constexpr int kQTmemChunks = 6;                   // column chunks 0..5 of Q are kept in tensor memory, 6..8 in shared memory
constexpr int kHalfBytes = 4 * kChunkBytes;       // 64 rows x 256 value columns
constexpr int kStages = 5;                        // ring of halves: a block takes two, so does Q on its way to tensor memory
constexpr int kRopes = 3;                         // columns 512..575, block g in slot g % 3
constexpr int Q_OFF = 0;                          // chunks 6..8
constexpr int KV_OFF = Q_OFF + (9 - kQTmemChunks) * kChunkBytes;
constexpr int R_OFF = KV_OFF + kStages * kHalfBytes;
constexpr int P_OFF = R_OFF + kRopes * kChunkBytes;      // 2 x [64 x 64]
constexpr int BAR_OFF = P_OFF + 2 * kChunkBytes;  // mbarriers
constexpr int MX_OFF = BAR_OFF + 192;             // float [3][128] exchange (2 for row maxima, 1 for row sums)
constexpr int MISC_OFF = MX_OFF + 1536;           // tmem base, abort flag, token validity masks
constexpr int SMEM_BYTES = MISC_OFF + 64;         // misc words
enum Bar { Q_FULL = 0, Q_EMPTY, FULL0, EMPTY0 = FULL0 + kStages, S_FULL0 = EMPTY0 + kStages, S_FULL1, P_FULL0, P_FULL1, O_FULL, O_EMPTY, NUM_BARS };
constexpr int TMEM_O = 0, TMEM_S = 256, TMEM_Q = 320;
static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared memory limit per CTA");
static_assert(NUM_BARS * 8 <= 192, "barrier area too small");
constexpr float kRescaleThreshold = 8.0f;         // log2 units; below it O keeps its stale scale
constexpr int kGatherThreads = 256;               // 8 gather warps
constexpr int threads(int mode) { return 192 + (mode == kDense ? 0 : kGatherThreads); }
constexpr int kPrefetchDist = 6;                  // cache pages pulled into L2 ahead of the stage loads
}  // namespace dtc

__device__ int g_tile64_status = 0;

// Optional timeline of the first blocks of CTA (0,0,0), compiled in with -DFMLA_TRACE only.
#ifdef FMLA_TRACE
__device__ long long g_tile64_trace[64 * 16];
#define FMLA_TRACE_AT(blk, slot)                                                          \
  do {                                                                                     \
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && (blk) < 64) g_tile64_trace[(blk) * 16 + (slot)] = clock64(); \
  } while (0)
#else
#define FMLA_TRACE_AT(blk, slot) do {} while (0)
#endif

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
using Ring = tc::RingPos<dtc::kStages>;

// S = Q K^T of one block, as straight-line code whose descriptors are a base plus an immediate: the products with the first
// half of its columns (four chunks), and those with the second half and the last 64.
__device__ __forceinline__ void s_first(uint32_t tmem_s, uint32_t tmem_q, uint64_t desc_h, uint32_t idesc) {
  using namespace dtc;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int s = 0; s < 4; ++s)
      tc::mma_ws_ts(tmem_s, tmem_q + c * 32 + s * 8, tc::desc_advance(desc_h, c * kChunkBytes + s * 32), idesc, (c | s) ? 1u : 0u);
}
__device__ __forceinline__ void s_second(uint32_t tmem_s, uint32_t tmem_q, uint64_t desc_q, uint64_t desc_h, uint64_t desc_r, uint32_t idesc) {
  using namespace dtc;
#pragma unroll
  for (int c = 4; c < 9; ++c)
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint64_t db = c < 8 ? tc::desc_advance(desc_h, (c - 4) * kChunkBytes + s * 32) : tc::desc_advance(desc_r, s * 32);
      if (c < kQTmemChunks) tc::mma_ws_ts(tmem_s, tmem_q + c * 32 + s * 8, db, idesc, 1u);
      else tc::mma_ws_ss(tmem_s, tc::desc_advance(desc_q, (c - kQTmemChunks) * kChunkBytes + s * 32), db, idesc, 1u);
    }
}
// O += P V for one half of the value columns
__device__ __forceinline__ void pv_half(uint32_t tmem_o, uint64_t desc_p, uint64_t desc_v, uint32_t idesc, bool first) {
#pragma unroll
  for (int s = 0; s < 4; ++s)
    tc::mma_ws_ss(tmem_o, tc::desc_advance(desc_p, s * 32), tc::desc_advance(desc_v, s * 2048), idesc, (first && s == 0) ? 0u : 1u);
}

// kDense: grid (s_q * ceil(hq_per_hk / 64), h_k, parts); kSparsePrefillCut: grid (h_q / 64, units), persistent over query
// tokens (SparsePrefillKernelParams)
template <int MODE, bool F16>
__global__ void __launch_bounds__(dtc::threads(MODE), 1)
mla_tile64_kernel(const __grid_constant__ TcParams P, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv) {
  using namespace dtc;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + Q_OFF, sKV = sbase + KV_OFF, sR = sbase + R_OFF, sP = sbase + P_OFF;
  auto bar = [&](int i) { return sbase + BAR_OFF + i * 8; };
  float* sMx = reinterpret_cast<float*>(smem + MX_OFF);
  volatile uint32_t* sTmem = reinterpret_cast<volatile uint32_t*>(smem + MISC_OFF);
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + MISC_OFF + 8);   // set by a softmax thread whose wait expired
  volatile uint32_t* sValid = reinterpret_cast<volatile uint32_t*>(smem + MISC_OFF + 16);   // [block % 3][token half]: 32 validity bits
  int* status = &g_tile64_status;

  const DecodeKernelParams& p = P.d;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool misaligned = (sbase & 1023u) != 0;      // the swizzled tiles need a 1024-byte aligned base
  if (misaligned && tid == 0) tc::report_status(status, 30);
  const float scale_log2 = MODE == kSparsePrefillCut ? P.sp.scale_log2 : p.scale_log2;
  // arrivals per filled stage: one (with a byte count) from the TMA thread, or one per gather thread (by hardware) and one
  // per gather warp
  constexpr int kKvFullCount = MODE == kDense ? 1 : kGatherThreads + kGatherThreads / 32;

  if (tid == 0) {
    tc::mbar_init(bar(Q_FULL), 1);
    tc::mbar_init(bar(Q_EMPTY), 1);
    for (int i = 0; i < kStages; ++i) {
      tc::mbar_init(bar(FULL0 + i), kKvFullCount);
      tc::mbar_init(bar(EMPTY0 + i), 1);
    }
    tc::mbar_init(bar(S_FULL0), 1);
    tc::mbar_init(bar(S_FULL1), 1);
    tc::mbar_init(bar(P_FULL0), 4);         // one arrival per softmax warp
    tc::mbar_init(bar(P_FULL1), 4);
    tc::mbar_init(bar(O_FULL), 1);
    tc::mbar_init(bar(O_EMPTY), 4);
    tc::fence_mbar_init();
    *sAbort = 0;
  }
  if (warp == 5) tc::tmem_alloc(sbase + MISC_OFF, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *sTmem;
  if constexpr (MODE == kDense) pdl_wait();     // the schedule, the queries and the cache may come from the kernel in front of this one (loads: mla_work.cuh)
  pdl_allow_dependents();       // the merge kernel may become resident now
  const Tile tile = make_tile<MODE>(P);

  if (misaligned || tile.n_work == 0) {
    // nothing to do
  } else if (warp == 4) {
    // ================================ TMA producer =====================================
    if (tc::elect_one()) {
      tc::prefetch_tensormap(&tmap_q);
      if constexpr (MODE == kDense) tc::prefetch_tensormap(&tmap_kv);
      int g = 0, req = 0;
      Ring at = {0, 0u};
      bool alive = true;
      for (int wi = 0; wi < tile.n_work && alive; ++wi) {
        const Work r = get_work<MODE>(P, tile, wi);
        if (r.blk_hi == r.blk_lo) continue;
        // Q: chunks 6..8 to their place, 0..5 through two stages of the ring into tensor memory (MMA thread).  Every S of the request
        // before has been formed.
        alive = tc::mbar_wait(bar(Q_EMPTY), (req & 1) ^ 1, status, 1);
        Ring second = at;
        second.step(1);
        if (alive) alive = tc::mbar_wait(bar(EMPTY0 + at.st), at.ph ^ 1, status, 2);
        if (alive) alive = tc::mbar_wait(bar(EMPTY0 + second.st), second.ph ^ 1, status, 2);
        if (!alive) break;
        tc::mbar_arrive_expect_tx(bar(Q_FULL), 9 * kChunkBytes);
#pragma unroll
        for (int c = 0; c < 9; ++c)
          tc::tma_load_4d(c < 4 ? sKV + at.st * kHalfBytes + c * kChunkBytes : c < kQTmemChunks ? sKV + second.st * kHalfBytes + (c - 4) * kChunkBytes : sQ + (c - kQTmemChunks) * kChunkBytes,
                          &tmap_q, c * 64, tile.head0, MODE == kDense ? tile.sq : r.batch, MODE == kDense ? r.batch : 0, bar(Q_FULL));
        ++req;
        if constexpr (MODE == kDense) {
          tc::mbar_arrive(bar(FULL0 + at.st));
          tc::mbar_arrive(bar(FULL0 + second.st));
          at.step(2);
          const int* bt = p.block_table + r.batch * p.block_table_stride_b;
          // pages kPrefetchDist steps ahead are pulled into L2 while the shared-memory stages are busy, so that the load
          // that later fills a stage sees L2 latency instead of HBM latency
          auto prefetch = [&](int blk) {
            const int pg = bt[blk];
#pragma unroll
            for (int c = 0; c < 9; ++c) tc::tma_prefetch_l2_4d(&tmap_kv, c * 64, tile.kh, 0, pg);
          };
          for (int blk = r.blk_lo; blk < min(r.blk_lo + kPrefetchDist, r.blk_hi); ++blk) prefetch(blk);
          int page_next = bt[r.blk_lo];
          for (int blk = r.blk_lo; blk < r.blk_hi && alive; ++blk, ++g) {
            const int page = page_next;
            if (blk + 1 < r.blk_hi) page_next = bt[blk + 1];
            if (blk + kPrefetchDist < r.blk_hi) prefetch(blk + kPrefetchDist);
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              alive = tc::mbar_wait(bar(EMPTY0 + at.st), at.ph ^ 1, status, 2);
              if (!alive) break;
              tc::mbar_arrive_expect_tx(bar(FULL0 + at.st), kHalfBytes + h * kChunkBytes);
#pragma unroll
              for (int c = 0; c < 4; ++c)
                tc::tma_load_4d(sKV + at.st * kHalfBytes + c * kChunkBytes, &tmap_kv, (h * 4 + c) * 64, tile.kh, 0, page, bar(FULL0 + at.st));
              // (the slot's last block, three before, is done with: the stage of this block's first half was free after it)
              if (h == 1) tc::tma_load_4d(sR + g % kRopes * kChunkBytes, &tmap_kv, 512, tile.kh, 0, page, bar(FULL0 + at.st));
              at.step(1);
            }
          }
        } else {
          at.step(2 + 2 * (r.blk_hi - r.blk_lo));
        }
      }
    }
  } else if (warp >= 6) {
    // ================================ gather producers =================================
    if constexpr (MODE == kSparsePrefillCut) {
      // Eight gather warps, eight rows each, all on the same block: the first 256 columns of their rows into one stage, then the last 64
      // and the second 256 into the next (a gather is bound by the 64 bytes a clock that an SM takes from L2, some 1 150 clk a block and
      // as much again for latency: S starts on the first half while the second is under way).  For each row and half the 32 lanes
      // copy consecutive 16-byte pieces: coalesced cp.async with a handful of address instructions per row.
      const int gw = warp - 6;
      const char* kv = reinterpret_cast<const char*>(P.sp.kv);
      const int64_t row_bytes = P.sp.kv_stride_s * 2;
      const uint32_t lane_base = static_cast<uint32_t>((lane >> 3) * kChunkBytes + gw * 8 * 128);
      const int sw = lane & 7;
      // No thread waits for its own copies: the stage barrier counts one arrival per gather thread that the
      // hardware performs when that thread's copies have landed, so the warp goes on to the next half at once
      // and the L2 round trips of several blocks overlap.  Lane 0 adds one ordinary arrival after its store of
      // the validity bits.  The issuing thread makes the landed data visible to the tensor pipe (proxy fence).
      auto arrive = [&](int st) {
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar(FULL0 + st)) : "memory");
        if (lane == 0) tc::mbar_arrive(bar(FULL0 + st));
      };
      int g = 0;
      Ring at = {0, 0u};
      bool alive = true;
      auto stage_free = [&] { return __all_sync(0xffffffffu, tc::mbar_wait(bar(EMPTY0 + at.st), at.ph ^ 1, status, 11)); };
      for (int wi = 0; wi < tile.n_work && alive; ++wi) {
        const Work r = get_work<MODE>(P, tile, wi);
        if (r.blk_hi == r.blk_lo) continue;
        int my_idx = __ldg(r.idx + r.blk_lo * 64 + gw * 8 + (lane & 7));
        for (int i = 0; i < 2 && alive; ++i) {           // the stages that Q passes through
          alive = stage_free();
          if (alive) arrive(at.st);
          at.step(1);
        }
        for (int blk = r.blk_lo; blk < r.blk_hi && alive; ++blk, ++g) {
          int idx_next = -1;
          if (blk + 1 < r.blk_hi) idx_next = __ldg(r.idx + (blk + 1) * 64 + gw * 8 + (lane & 7));
          if (my_idx < 0 || my_idx >= P.sp.s_kv) my_idx = -1;
          const uint32_t bal = __ballot_sync(0xffffffffu, my_idx >= 0) & 0xffu;
          auto gather_half = [&](int h) {
            const uint32_t stage = sKV + at.st * kHalfBytes + lane_base;
#pragma unroll
            for (int rr = 0; rr < 8; ++rr) {
              const int idx = __shfl_sync(0xffffffffu, my_idx, rr);
              const bool ok = idx >= 0;
              const char* src = kv + (ok ? (int64_t)idx * row_bytes + h * 512 + lane * 16 : 0);
              cp_async16(stage + rr * 128 + ((sw ^ rr) << 4), src, ok);
            }
          };
          alive = stage_free();
          if (!alive) break;
          if (lane == 0 && gw == 0) FMLA_TRACE_AT(g, 0);
          if (lane == 0) reinterpret_cast<volatile uint8_t*>(sValid)[g % 3 * 8 + gw] = static_cast<uint8_t>(bal);   // tokens 8*gw ..
          gather_half(0);
          arrive(at.st);
          at.step(1);
          // the last 64 columns, four rows at a time (the slot's last block, three before, is done with: the stage of this block's
          // first half was free after it)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int row = i * 4 + (lane >> 3);
            const int idx = __shfl_sync(0xffffffffu, my_idx, row);
            const bool ok = idx >= 0;
            cp_async16(sR + g % kRopes * kChunkBytes + (gw * 8 + row) * 128 + ((sw ^ row) << 4), kv + (ok ? (int64_t)idx * row_bytes + 1024 + sw * 16 : 0), ok);
          }
          alive = stage_free();
          if (!alive) break;
          gather_half(1);
          arrive(at.st);
          at.step(1);
          if (lane == 0 && gw == 0) FMLA_TRACE_AT(g, 1);
          my_idx = idx_next;
        }
      }
    }
  } else if (warp == 5) {
    // ================================ MMA issuer =======================================
    // One thread.  A warp that polled four barriers, shared the outcome by a vote and slept between polls took 8 % longer, and with
    // it went the arrivals of 128 threads on each of S_EMPTY, P_FULL and O_EMPTY (one per warp now, or none): 333 tokens, top-k 512, 50.4 ->
    // 47.7 us, 4096, top-k 2048, 1717 -> 1605; dense, 64 heads x 3 tokens, 16 x 16 000 156.5 -> 143.9.
    if (tc::elect_one()) {
      constexpr uint32_t idesc_s = tc::idesc_bf16_f32(64, 64, 0, 0, F16);
      constexpr uint32_t idesc_o = tc::idesc_bf16_f32(64, 256, 0, 1, F16);
      const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);             // A of S, chunks 6..8: K-major
      const uint64_t desc_k = tc::smem_desc_sw128(sKV, 16, 1024);            // B of S: K-major (stage 0); also Q's chunks 0..5 on their way
      const uint64_t desc_r = tc::smem_desc_sw128(sR, 16, 1024);             // the same for the last 64 columns (slot 0)
      const uint64_t desc_p = tc::smem_desc_sw128(sP, 16, 1024);             // A of PV: K-major
      const uint64_t desc_v = tc::smem_desc_sw128(sKV, kChunkBytes, 1024);   // B of PV: MN-major, 64-wide column groups 8 KB apart (stage 0)
      int g = 0, req = 0;
      Ring at_s = {0, 0u}, at_p = {0, 0u};
      bool alive = true;
      for (int wi = 0; wi < tile.n_work && alive; ++wi) {
        const Work r = get_work<MODE>(P, tile, wi);
        const int nblk = r.blk_hi - r.blk_lo;
        if (nblk == 0) continue;
        alive = tc::mbar_wait(bar(Q_FULL), req & 1, status, 5);
        if (!alive) break;
        // Q chunks 0..5: shared memory -> tensor memory (8 copies of 64 rows x 16 bytes per chunk)
        tc::tc_fence_after();
#pragma unroll
        for (int c = 0; c < kQTmemChunks; ++c) {
          if (c == 4) at_s.step(1);
#pragma unroll
          for (int sub = 0; sub < 8; ++sub)
            tc::tmem_cp_64x128b(tmem + TMEM_Q + c * 32 + sub * 4, tc::desc_advance(desc_k, at_s.st * kHalfBytes + (c & 3) * kChunkBytes + sub * 16));
          // a stage is given back only when everybody who fills it has arrived for this round, too
          if (c == 3 || c == kQTmemChunks - 1) {
            alive = alive && tc::mbar_wait(bar(FULL0 + at_s.st), at_s.ph, status, 5);
            tc::tc_commit(bar(EMPTY0 + at_s.st));
          }
        }
        at_s.step(1);
        at_p.step(2);
        // S of block js, half by half, and P V of block jp < js are issued in whichever order their inputs become ready; P V goes first
        // when both are possible: it releases stages and the next loads depend on that.  S of block js may follow when P V of block
        // js - 2 has been issued: that block's S has been read then, and the S buffer is free.
        int js = 0, jp = 0, idle = 0;
        bool half = false;
        while (jp < nblk && alive) {
          const int gs = g + js, gp = g + jp;
          if (jp < js && tc::mbar_test_wait(bar(P_FULL0 + (gp & 1)), (gp >> 1) & 1)) {
            if (jp == 0) alive = tc::mbar_wait(bar(O_EMPTY), (req & 1) ^ 1, status, 6);
            if (!alive) break;
            tc::tc_fence_after();
            FMLA_TRACE_AT(gp, 4);
            const uint64_t dp = tc::desc_advance(desc_p, (gp & 1) * kChunkBytes);
            pv_half(tmem + TMEM_O, dp, tc::desc_advance(desc_v, at_p.st * kHalfBytes), idesc_o, jp == 0);
            tc::tc_commit(bar(EMPTY0 + at_p.st));
            at_p.step(1);
            pv_half(tmem + TMEM_O + 128, dp, tc::desc_advance(desc_v, at_p.st * kHalfBytes), idesc_o, jp == 0);
            tc::tc_commit(bar(EMPTY0 + at_p.st));
            at_p.step(1);
            FMLA_TRACE_AT(gp, 5);
            ++jp;
            idle = 0;
          } else if (js < nblk && js - jp < 2 && tc::mbar_test_wait(bar(FULL0 + at_s.st), at_s.ph)) {
            if constexpr (MODE == kSparsePrefillCut) tc::fence_proxy_async_smem();   // rows written by cp.async -> tensor pipe
            tc::tc_fence_after();
            const uint32_t tmem_s = tmem + TMEM_S + (gs & 1) * 32;
            const uint64_t dh = tc::desc_advance(desc_k, at_s.st * kHalfBytes);
            if (!half) {
              FMLA_TRACE_AT(gs, 2);
              s_first(tmem_s, tmem + TMEM_Q, dh, idesc_s);
            } else {
              FMLA_TRACE_AT(gs, 12);
              s_second(tmem_s, tmem + TMEM_Q, desc_q, dh, tc::desc_advance(desc_r, gs % kRopes * kChunkBytes), idesc_s);
              tc::tc_commit(bar(S_FULL0 + (gs & 1)));
              FMLA_TRACE_AT(gs, 3);
              if (js == nblk - 1) tc::tc_commit(bar(Q_EMPTY));
              ++js;
            }
            half = !half;
            at_s.step(1);
            idle = 0;
          } else if (++idle > tc::kSpinLimit) {
            tc::report_status(status, 6);
            alive = false;
          }
        }
        g += nblk;
        if (alive) tc::tc_commit(bar(O_FULL));
        ++req;
      }
    }
  } else if (warp < 4) {
    // ================================ softmax / epilogue ================================
    const int r_row = tid & 63, th = tid >> 6;           // TMEM lane tid: row tid%64, token/column half tid/64
    const uint32_t lane_addr = static_cast<uint32_t>(warp * 32) << 16;
    int g = 0, req = 0;
    Ring at = {0, 0u}, before = {0, 0u};      // first stage of this block; second stage of the one before
    bool aborted = false;        // uniform over the 128 softmax threads: only read right after a bar_sync
    for (int wi = 0; wi < tile.n_work; ++wi) {
      const Work r = get_work<MODE>(P, tile, wi);
      const int nblk = r.blk_hi - r.blk_lo;
      if (nblk > 0) at.step(2);    // Q
      float m_run = neg_inf();     // running maximum (base-2 scaled logits)
      float m_used = 0.f;          // the maximum O and l are currently scaled with
      float l_part = 0.f;          // this thread's share of the row sum
      for (int j = 0; j < nblk && !aborted; ++j, ++g) {
        const int st = g & 1;
        uint32_t sv[32];
        uint32_t vbits = 0xffffffffu;
        if (tc::mbar_wait(bar(S_FULL0 + st), (g >> 1) & 1, status, 8)) {
          if (tid == 0) FMLA_TRACE_AT(g, 6);
          tc::tc_fence_after();
          tc::tmem_ld32(tmem + lane_addr + TMEM_S + st * 32, sv);
          if constexpr (MODE == kSparsePrefillCut) vbits = sValid[g % 3 * 2 + th];
          tc::tmem_wait_ld();
          tc::tc_fence_before();
        } else {
          *sAbort = 1;
#pragma unroll
          for (int i = 0; i < 32; ++i) sv[i] = 0u;
        }
        if (tid == 0) FMLA_TRACE_AT(g, 7);

        if constexpr (MODE == kDense) {
          // Rows of the last page beyond the sequence may hold anything (NaN included) and 0 * NaN must not reach O.  Their logits,
          // which S has been formed with by now, are masked.
          const int rows_valid = r.seqlen - (r.blk_lo + j) * 64;
          for (int i = tid; i < (64 - rows_valid) * 64; i += 128) {
            const int row = rows_valid + (i >> 6), c16 = i & 63;
            *reinterpret_cast<uint4*>(smem + KV_OFF + (c16 < 32 ? at.st : (at.st + 1) % kStages) * kHalfBytes + (c16 >> 3 & 3) * kChunkBytes + row * 128 + (c16 & 7) * 16) =
                make_uint4(0, 0, 0, 0);
          }
          const int tok0 = (r.blk_lo + j) * 64 + th * 32;
          if (tok0 + 32 > r.border) vbits = tok0 >= r.border ? 0u : (0xffffffffu >> (32 - (r.border - tok0)));
        }
        // masked logits become -inf (a select: they may hold anything); the maximum is taken over the raw
        // logits in four independent chains and scaled once (the scale is positive)
        if (vbits != 0xffffffffu) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (!((vbits >> i) & 1u)) sv[i] = 0xff800000u;
        }
        float mx4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          mx4[c] = fmaxf(__uint_as_float(sv[c * 8]), __uint_as_float(sv[c * 8 + 1]));
#pragma unroll
          for (int i = 2; i < 8; i += 2) mx4[c] = max3(mx4[c], __uint_as_float(sv[c * 8 + i]), __uint_as_float(sv[c * 8 + i + 1]));
        }
        float mx = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * scale_log2;
        float* xch = sMx + (j & 1) * 128;
        xch[tid] = mx;
        bar_sync(1, 128);
        const bool stop = *sAbort != 0;      // (looked at later: nothing here waits for the load)
        if (tid == 0) FMLA_TRACE_AT(g, 8);
        mx = fmaxf(mx, xch[tid ^ 64]);
        const float m_new = fmaxf(m_run, mx);

        // O and l carry the scale 2^-m_used; it is moved only when the maximum grew by more than the
        // threshold (or when the first real value arrives after fully masked blocks)
        bool need = false;
        if (j == 0 || (m_run == neg_inf() && m_new != neg_inf())) {
          // first block, or the first visible key after fully masked blocks: O and l are exactly zero, so the
          // reference scale is simply set (multiplying 0 by 2^(0 - m_new) would give NaN for m_new < -128)
          m_used = (m_new == neg_inf()) ? 0.f : m_new;
        } else {
          need = (m_new - m_used) > kRescaleThreshold;
        }
        m_run = m_new;
        const bool any_need = __any_sync(0xffffffffu, need);
        if (any_need) {
          if (!tc::mbar_wait(bar(EMPTY0 + before.st), before.ph, status, 9)) *sAbort = 1;      // every P V so far is complete
          const float m_next = need ? m_new : m_used;
          const float alpha = exp2f(m_used - m_next);
          m_used = m_next;
          l_part *= alpha;
          tc::tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 8; ++c) {
            uint32_t ov[32];
            tc::tmem_ld32(tmem + lane_addr + TMEM_O + c * 32, ov);
            tc::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
            tc::tmem_st32(tmem + lane_addr + TMEM_O + c * 32, ov);
          }
          tc::tmem_wait_st();
          tc::tc_fence_before();
        }
        if (tid == 0) FMLA_TRACE_AT(g, 10);
        F2 sum[2] = {f2(0.f), f2(0.f)};
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          F2 x = f2_fma(F2{__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])}, f2(scale_log2), f2(-m_used));
          x.lo = exp2f(x.lo);
          x.hi = exp2f(x.hi);
          sum[i & 1] = f2_add(sum[i & 1], x);
          pk[i] = pack_16x2<F16>(x.lo, x.hi);
        }
        sum[0] = f2_add(sum[0], sum[1]);
        l_part += sum[0].lo + sum[0].hi;
        if (stop) { aborted = true; break; }
        // P has two buffers.  P V of block g - 2 was issued before the last products of S of block g, whose commit tells of both: it is
        // complete.  (Its stages do not tell: where a request has one block, Q of the next but one has passed through them since.)
        if (tid == 0) FMLA_TRACE_AT(g, 9);
        // P[row][th*32 .. +32) -> K-major 128B-swizzled A operand: 16-byte chunk (th*4 + q) ^ (row & 7)
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)
          st_shared_v4(sP + st * kChunkBytes + r_row * 128 + ((((th * 4 + q4) ^ (r_row & 7))) << 4),
                       make_uint4(pk[q4 * 4], pk[q4 * 4 + 1], pk[q4 * 4 + 2], pk[q4 * 4 + 3]));
        tc::fence_proxy_async_smem();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(P_FULL0 + st));
        if (tid == 0) FMLA_TRACE_AT(g, 11);
        before = at;
        before.step(1);
        at.step(2);
      }

      // ---- epilogue of this work item ---------------------------------------------------
      float* xch = sMx + 256;
      bar_sync(1, 128);
      xch[tid] = l_part;
      bar_sync(1, 128);
      if (*sAbort) aborted = true;
      if (aborted) break;
      const float l = l_part + xch[tid ^ 64];
      const int head = tile.head0 + r_row;
      const float inv = (l == 0.f || nblk == 0) ? 0.f : 1.f / l;
      bool have_o = nblk > 0;
      if (have_o) {
        if (!tc::mbar_wait(bar(O_FULL), req & 1, status, 10)) { *sAbort = 1; have_o = false; }
        tc::tc_fence_after();
      }
      // Every store is one full 32-byte sector (each thread writes its own row: 16-byte stores made the load/store unit handle
      // twice as many half-filled ones).
      const bool row_ok = MODE == kSparsePrefillCut || r_row < p.hq_per_hk - tile.hb * 64;
      const int q_seq_per_hk = MODE == kSparsePrefillCut ? 0 : p.s_q * p.hq_per_hk;
      // row of the partial slot of a split request: (kv head, query token, head)
      const int64_t part_row = MODE == kSparsePrefillCut ? (int64_t)r.split_slot * P.sp.h_q + head : ((int64_t)r.split_slot * p.h_k + tile.kh) * q_seq_per_hk + tile.sq * p.hq_per_hk + tile.hb * 64 + r_row;
      __nv_bfloat16* o_row = MODE == kSparsePrefillCut
          ? reinterpret_cast<__nv_bfloat16*>(P.sp.out) + ((int64_t)r.batch * P.sp.h_q + head) * 512
          : reinterpret_cast<__nv_bfloat16*>(p.out) + r.batch * p.o_stride_b + tile.sq * p.o_stride_s + head * p.o_stride_h;
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        uint32_t cur[32];
        if (have_o) {
          tc::tmem_ld32(tmem + lane_addr + TMEM_O + c * 32, cur);
          tc::tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) cur[i] = 0u;
        }
        const int col = (c >> 2) * 256 + th * 128 + (c & 3) * 32;
        if (!row_ok) continue;
        if (r.no_split) {
#pragma unroll
          for (int q8 = 0; q8 < 2; ++q8) {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
              w[i] = pack_16x2<F16>(__uint_as_float(cur[q8 * 16 + 2 * i]) * inv, __uint_as_float(cur[q8 * 16 + 2 * i + 1]) * inv);
            st_global_32B(o_row + col + q8 * 16, w);
          }
        } else {
#pragma unroll
          for (int q8 = 0; q8 < 4; ++q8) {
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = __float_as_uint(__uint_as_float(cur[q8 * 8 + i]) * inv);
            st_global_32B((MODE == kSparsePrefillCut ? P.sp.o_accum : p.o_accum) + part_row * 512 + col + q8 * 8, w);
          }
        }
      }
      if (nblk > 0) {
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(O_EMPTY));
        ++req;
      }
      if (th == 0 && row_ok) {
        if constexpr (MODE == kSparsePrefillCut) {
          const int64_t o = r.no_split ? (int64_t)r.batch * P.sp.h_q + head : part_row;
          (r.no_split ? P.sp.max_logits : P.sp.max_accum)[o] = inv == 0.f ? neg_inf() : m_run;
          (r.no_split ? P.sp.lse : P.sp.lse_accum)[o] = inv == 0.f ? neg_inf() : log2f(l) + m_used;
        } else if (r.no_split) {
          p.softmax_lse[((int64_t)r.batch * p.h_q + head) * p.s_q + tile.sq] = inv == 0.f ? pos_inf() : (log2f(l) + m_used) * kLn2;
        } else {
          p.lse_accum[part_row] = inv == 0.f ? neg_inf() : log2f(l) + m_used;
          if (p.no_split_hint && tid == 0) tc::report_status(status, 41);     // a split request although the caller ruled it out
        }
      }
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if (warp == 5) tc::tmem_dealloc(tmem, 512);
}

// ---- host side ----------------------------------------------------------------------------------
cudaError_t launch_sparse_prefill_64(const SparsePrefillKernelParams& sp, cudaStream_t stream) {
  TcParams P = {};
  P.sp = sp;
  CUtensorMap tq;
  // q [s_q][h_q][576] as (col, head, token, 1)
  if (!tmah::make_map_4d(&tq, sp.q, sp.h_q, sp.s_q, 1, sp.q_stride_h, sp.q_stride_s, sp.q_stride_s * sp.s_q, 64, 1)) return cudaErrorInvalidValue;
  constexpr auto kern = mla_tile64_kernel<kSparsePrefillCut, false>;
  if (cudaError_t e = allow_smem<kern>(dtc::SMEM_BYTES); e != cudaSuccess) return e;
  kern<<<dim3(sp.h_q / 64, sp.units, 1), dtc::threads(kSparsePrefillCut), dtc::SMEM_BYTES, stream>>>(P, tq, tq);      // no page is read through a map
  return cudaGetLastError();
}

template <bool F16>
static cudaError_t launch_dense_tile64(const TcParams& P, const CUtensorMap& tq, const CUtensorMap& tkv, dim3 grid, cudaStream_t stream) {
  constexpr auto kern = mla_tile64_kernel<kDense, F16>;
  if (cudaError_t e = allow_smem<kern>(dtc::SMEM_BYTES); e != cudaSuccess) return e;
  return launch_dependent(kern, grid, dtc::threads(kDense), dtc::SMEM_BYTES, stream, P, tq, tkv);
}

// Several 64-row tiles read the same pages (and the pair does not apply, mla_dispatch.cu).  Device time, mla_few_rows.cu -> this kernel:
// 64 heads x 3 tokens, 16 requests of 16 000 tokens 163 -> 135 us, 64 of 4 000 160 -> 138, 128 of 1 000 103 -> 90, 16 of 1 000 31.3 -> 30.7, 4 of 500
// 22.0 -> 21.3; 96 heads, 16 of 3 000 38.9 -> 35.2, two tokens 50.6 -> 45.0; 192 heads, 16 of 3 000 51.6 -> 44.3.  The other way where that
// kernel shares the rows of the schedule (one request of 1 000 14.3 -> 19.6, 96 heads, 4 of 500 14.6 -> 18.9).  The lengths are on the
// device, so the line is drawn for the larger calls.
bool decode_dense_tile64_applies(const DecodeKernelParams& p) { return p.hq_per_hk >= 64 && p.s_q * ((p.hq_per_hk + 63) / 64) > 1; }

cudaError_t launch_decode_dense_tile64(const DecodeKernelParams& p, cudaStream_t stream) {
  TcParams P = {};
  P.d = p;
  CUtensorMap tq, tkv;
  // q [b][s_q][h_q][576], box of 64 heads (heads past h_q read as zero); cache [num_blocks][64][h_k][576] as (col, head, row in page, page)
  if (!tmah::make_map_4d(&tq, p.q, p.h_q, p.s_q, p.b, p.q_stride_h, p.q_stride_s, p.q_stride_b, 64, 1)) return cudaErrorInvalidValue;
  if (!tmah::make_map_4d(&tkv, p.kcache, p.h_k, 64, p.num_blocks, p.k_stride_head, p.k_stride_row, p.k_stride_block, 1, 64)) return cudaErrorInvalidValue;
  const dim3 grid(p.s_q * ((p.hq_per_hk + 63) / 64), p.h_k, p.num_sm_parts);
  return p.is_f16 ? launch_dense_tile64<true>(P, tq, tkv, grid, stream) : launch_dense_tile64<false>(P, tq, tkv, grid, stream);
}

#ifdef FMLA_TRACE
extern "C" int fmla_debug_read_trace(long long* host, int n) {
  return (int)cudaMemcpyFromSymbol(host, g_tile64_trace, sizeof(long long) * n);
}
#endif

cudaError_t set_status_mirror_tile64(int* mapped_host_word) { return tc::set_status_mirror(mapped_host_word); }

cudaError_t read_tile64_status(int* host_status, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(host_status, g_tile64_status, sizeof(int));
  if (e != cudaSuccess) return e;
  if (reset && *host_status != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_tile64_status, &zero, sizeof(int));
  }
  return e;
}

}  // namespace fmla
