// Dense variable-length MHA forward (bf16, head dims 192/128 and 128/128) for sm_100a on
// tcgen05 / TMA / tensor memory.
//
// One CTA = 256 query rows (two tiles of 128) of one (sequence, head) at a time; keys are walked in blocks of 128.
//   warps 0-3  softmax of tile 0, warps 4-7 softmax of tile 1: one thread per query row (TMEM lane = row): largest logit, then in two
//              halves of 64 keys S -> registers, P (bf16) written back over the columns S came from, row sums; at the end 1/l
//              normalisation and stores
//   warp 8     TMA: both Q tiles once; K and V blocks in the order of their use through one ring of 32 KB stages (64-column chunks of
//              [128 rows x 128 bytes], 128-byte swizzle); columns 128 to 191 of K into two slots of their own
//   warp 9     MMA, one thread: S_t = Q_t K^T (tcgen05.mma m128n128k16, both operands from shared memory),
//              O_t += P_t V (m128n128k16, P from tensor memory, V from shared memory MN-major), in the
//              order  P V of tile 0, S of tile 0 for the next block, P V of tile 1, S of tile 1 for the
//              next block: while the softmax of one tile runs, the tensor pipe works for the other tile.  P V starts on the first 64
//              keys of a block while the softmax of the others runs.
//   warp 10    in large grids: takes over CTAs that have not been started (clusterlaunchcontrol), one after the other
// What bounds it: a tile's chain S -> softmax -> P V -> S (P lies over S, and tensor memory has no room for a second S), of
// which the tensor pipe can hide the part that is as long as the other tile's two GEMMs (1280 clk at 192/128, 1024 at
// 128/128), and in long runs the power limit.  A block of a CTA (two tiles) took 4 240 clk at 192/128 and 3 850 at 128/128 with two
// threads per row, single V stages at 192/128 (700 clk waiting for V) and issue and waits by a whole warp; it takes 3 295 and 3 220
// now (two sequences of 4 096, no mask, one time stamp per block; 3 890 -> 3 235 and 3 560 -> 3 055 with 2 000), at a clock that falls from 1.84 to
// 1.65 GHz at 128/128 in a burst of four calls and from 1.60 to 1.44 in a loop.  What shortened it: one ring for K and V; the maximum first,
// so that a warp decides alone whether the scale moves and P can be handed over in halves; part of the exponentials off the special
// function unit; and little code: the warps of both tiles and the issuing thread share an instruction cache, and the block's body
// rolled up to 64 logits, with masked blocks rewritten in place first, is 6 % faster than unrolled to 128.
// The scale m_used of a row moves only when one of its logits exceeds it by more than 2^8; only then O is rescaled.
// TMEM map (all 512 columns): S/P of tile 0 = [0,128), of tile 1 = [128,256), O of tile 0 = [256,384),
// of tile 1 = [384,512).  For M = 128 element (row r, col c) of a result sits in lane r, column c;
// the bf16 A operand in tensor memory holds k values (2c, 2c+1) of row r in the 32-bit column c of lane r.
//
// Semantics of the reference forward (csrc/sm100/prefill/dense/fmha_cutlass_fwd_sm100.cu:67-119
// and its mainloop): packed varlen q/k/v with cu_seqlens; GQA maps q head h to kv head
// h / (h_q/h_k); causal masking is bottom-right aligned (query i sees keys j <= i + s_k - s_q,
// collective/fmha_fusion.hpp:266-274); LSE is the natural log of the row sum; rows with no
// visible key give O = 0, LSE = -inf.
// Every mbarrier wait is bounded (tc_common.cuh); a pipeline fault sets a status word and lets the
// CTA drain and free its tensor memory.
#include "kernels.h"
#include "launch.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

#include <algorithm>
#include <type_traits>

namespace fmla {

namespace dft {
constexpr int kChunkBytes = 128 * 128;            // [128 rows x 64 bf16], 128-byte rows
constexpr int kVBytes = 2 * kChunkBytes;          // 128 x 128 bf16
constexpr int kSoftmaxWarps = 8;
constexpr int threads(bool take_over) { return (kSoftmaxWarps + 2 + take_over) * 32; }
constexpr int kMaxStages = 5;
enum Bar { Q_FULL = 0, Q_EMPTY, FULL0, EMPTY0 = FULL0 + kMaxStages, S_FULL0 = EMPTY0 + kMaxStages, S_FULL1, P_HEAD0, P_HEAD1, P_FULL0,
           P_FULL1, O_DONE0, O_DONE1, CLAIMED, TILE_FULL, TILE_EMPTY, NUM_BARS };
constexpr int TMEM_S = 0, TMEM_O = 256;
// One pair of logits in so many is exponentiated on the multiply-add pipe (the special function unit does 16 a clock and SM: 1024 clk
// for a tile's block, as long as its two products).  4 x 1000 tokens, 8 heads, 128/128, causal: none 23.3, one in eight 20.9, in four
// 20.4, in three 19.9, in two 21.3 us.
constexpr int kPolyPeriod = 3;
constexpr float kRescaleThreshold = 8.0f;         // log2 units; below it O keeps its stale scale
// A row's exponents are as exact as its scale's last place: with a scale below this, half a place is at most 2^7 and so are they.
constexpr float kWideScale = 0x1p32f;
template <int D_QK>
struct Layout {
  static constexpr int NCH = D_QK / 64;           // 64-column chunks of Q and K
  static constexpr int kTileBytes = NCH * kChunkBytes;    // one Q tile / one K block
  static constexpr int Q_OFF = 0;                 // 2 tiles
  static constexpr int RING_OFF = 2 * kTileBytes;
  static constexpr int kStages = D_QK == 192 ? 3 : 5;
  static constexpr int REST_OFF = RING_OFF + kStages * kVBytes;      // columns 128 to 191 of K: two slots, block c in slot c & 1
  static constexpr int kRestSlots = D_QK == 192 ? 2 : 0;
  static constexpr int BAR_OFF = REST_OFF + kRestSlots * kChunkBytes;
  static constexpr int MISC_OFF = BAR_OFF + 192;
  static constexpr int CLAIM_OFF = MISC_OFF + 16; // answer of a claim
  static constexpr int TILE_OFF = CLAIM_OFF + 16; // int [2][8]: the tile that is worked on and the next one
  static constexpr int SMEM_BYTES = TILE_OFF + 64;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared memory limit per CTA");
};
static_assert(NUM_BARS * 8 <= 192, "barrier area too small");
}  // namespace dft

__device__ int g_dense_tc_status = 0;

// The S = Q K^T instructions of a tile and key block.  One copy of the code serves every (tile, K stage): the bases come in at
// run time (warp-uniform) and the unrolled code adds immediates; with a copy for each, every copy's first instruction
// waited for its fetch.
template <int D_QK>
__device__ __forceinline__ void dense_s_block(uint32_t tmem_s, uint64_t desc_q, uint64_t desc_k, uint64_t desc_rest, uint32_t idesc) {
  using L = dft::Layout<D_QK>;
#pragma unroll
  for (int c = 0; c < L::NCH; ++c)
#pragma unroll
    for (int s = 0; s < 4; ++s)
      tc::mma_ss(tmem_s, tc::desc_advance(desc_q, c * dft::kChunkBytes + s * 32), c < 2 ? tc::desc_advance(desc_k, c * dft::kChunkBytes + s * 32) : tc::desc_advance(desc_rest, s * 32), idesc,
                 (c | s) ? 1u : 0u);
}
// O += P V of one tile and key block, the 16-key steps [kFirst, kEnd): P from the first 64 of the S columns (8 a step).
template <int kFirst, int kEnd>
__device__ __forceinline__ void dense_pv_steps(uint32_t tmem_o, uint32_t tmem_p, uint64_t desc_v, uint32_t idesc, bool first) {
#pragma unroll
  for (int s = kFirst; s < kEnd; ++s)
    tc::mma_ts(tmem_o, tmem_p + s * 8, tc::desc_advance(desc_v, s * 2048), idesc, (first && s == 0) ? 0u : 1u);
}
// the largest of three; NaN if one of them is
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// What a CTA works on: 256 query rows of one head of one sequence.
struct DenseTile {
  int q0, lq, k0, lk, m_base, head;
  bool valid;                  // false: nothing is left to do
};
__device__ __forceinline__ DenseTile dense_tile(const DenseKernelParams& p, int index) {
  // with a causal mask the last tiles have the most keys: they are started first
  const int n_tiles = (p.max_seqlen_q + 255) / 256, n_heads = p.h_q * p.batch;
  const int tile_rank = p.tiles_outer ? index / n_heads : index % n_tiles;
  const int bh = p.tiles_outer ? index % n_heads : index / n_tiles;
  const int b = bh / p.h_q;
  DenseTile t;
  t.head = bh % p.h_q;
  t.q0 = __ldg(p.cu_q + b);
  t.lq = __ldg(p.cu_q + b + 1) - t.q0;
  t.k0 = __ldg(p.cu_k + b);
  t.lk = __ldg(p.cu_k + b + 1) - t.k0;
  t.m_base = (n_tiles - 1 - tile_rank) * 256;
  t.valid = true;
  return t;
}
// blocks of 128 keys that 128-row tile `t` needs: those its last row sees; none for a tile without rows.  n1 >= n0, or n1 == 0
__device__ __forceinline__ int dense_blocks(const DenseKernelParams& p, const DenseTile& w, int t) {
  const int first = w.m_base + t * 128;
  if (first >= w.lq) return 0;
  const int all = (w.lk + 127) >> 7;
  if (!p.is_causal) return all;
  const int last_key = min(first + 127, w.lq - 1) + (w.lk - w.lq);   // inclusive
  return last_key < 0 ? 0 : min(all, (last_key >> 7) + 1);
}

// prefetch of one tile into L2
__device__ __forceinline__ void tma_prefetch_l2_3d(const void* tmap, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];\n" ::"l"(tmap), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

// Asks for the next CTA of the grid that has not been started (it then never is); the answer arrives as 16 bytes at `answer`,
// counted on `bar`.
__device__ __forceinline__ void claim_next_cta(uint32_t answer, uint32_t bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n" ::"r"(answer), "r"(bar) : "memory");
}
// its blockIdx.x, or -1 when every CTA has been started
__device__ __forceinline__ int claimed_cta(uint32_t answer) {
  int x;
  asm volatile(
      "{\n.reg .b128 r;\n.reg .pred p;\n.reg .b64 lo, hi;\nld.shared.v2.b64 {lo, hi}, [%1];\nmov.b128 r, {lo, hi};\n"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\nmov.b32 %0, -1;\n"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, r;\n}\n"
      : "=r"(x)
      : "r"(answer)
      : "memory");
  return x;
}

// grid: ceil(max_seqlen_q/256) * h_q * batch CTAs in the order `p.tiles_outer` selects.  kTakeOver: a CTA that is running takes over
// CTAs that have not been started (warp 10), so that the loads and first products of its next tile overlap the last softmax,
// the read of O and the stores of the present one; barriers, tensor memory and tensor maps are set up once.
template <int D_QK, bool kTakeOver>
__global__ void __launch_bounds__(dft::threads(kTakeOver), 1)
dense_fwd_tc_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_q,
                    const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v) {
  using namespace dft;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + L::Q_OFF, sRing = sbase + L::RING_OFF, sRest = sbase + L::REST_OFF;
  auto bar = [&](int i) { return sbase + L::BAR_OFF + i * 8; };
  volatile uint32_t* sTmem = reinterpret_cast<volatile uint32_t*>(smem + L::MISC_OFF);
  volatile int* sTile = reinterpret_cast<volatile int*>(smem + L::TILE_OFF);
  int* status = &g_dense_tc_status;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = p.h_q / p.h_k;
  DenseTile w = dense_tile(p, blockIdx.x);
  if (w.m_base >= w.lq) return;
  if ((sbase & 1023u) != 0) {   // the swizzled tiles need a 1024-byte aligned base
    if (tid == 0) tc::report_status(status, 30);
    return;
  }

  auto load_q = [&](bool both) {
    tc::mbar_arrive_expect_tx(bar(Q_FULL), (both ? 2 : 1) * L::kTileBytes);
    for (int t = 0; t < (both ? 2 : 1); ++t)
#pragma unroll
      for (int c = 0; c < L::NCH; ++c)
        tc::tma_load_3d(sQ + t * L::kTileBytes + c * kChunkBytes, &tmap_q, c * 64, w.head, w.q0 + w.m_base + t * 128, bar(Q_FULL));
  };
  auto load_k = [&](int j, int st, int c_blk) {
    tc::mbar_arrive_expect_tx(bar(FULL0 + st), L::kTileBytes);
#pragma unroll
    for (int c = 0; c < L::NCH; ++c)
      tc::tma_load_3d(c < 2 ? sRing + st * kVBytes + c * kChunkBytes : sRest + (c_blk & 1) * kChunkBytes, &tmap_k, c * 64, w.head / group, w.k0 + j * 128, bar(FULL0 + st));
  };
  auto load_v = [&](int j, int st) {
    tc::mbar_arrive_expect_tx(bar(FULL0 + st), kVBytes);
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tma_load_3d(sRing + st * kVBytes + c * kChunkBytes, &tmap_v, c * 64, w.head / group, w.k0 + j * 128, bar(FULL0 + st));
  };
  // The n-th tile of this CTA is described in sTile[n & 1]; tiles from the second on are taken over from other CTAs.
  auto put_tile = [&](int n, const DenseTile& t) {
    volatile int* d = sTile + (n & 1) * 8;
    d[0] = t.valid ? 1 : 0; d[1] = t.q0; d[2] = t.lq; d[3] = t.k0; d[4] = t.lk; d[5] = t.m_base; d[6] = t.head;
  };
  auto get_tile = [&](int n) {
    volatile int* d = sTile + (n & 1) * 8;
    DenseTile t;
    t.valid = d[0] != 0; t.q0 = d[1]; t.lq = d[2]; t.k0 = d[3]; t.lk = d[4]; t.m_base = d[5]; t.head = d[6];
    return t;
  };
  // Waits for the description of tile n >= 1; whole warp.  Another tile is claimed when every consuming warp has begun this one and
  // its loads near their end.
  auto await_tile = [&](int n) {
    const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(bar(TILE_FULL), (n - 1) & 1, status, 50));
    if (lane == 0) tc::mbar_arrive(bar(TILE_EMPTY));
    return ok;
  };
  if (warp == kSoftmaxWarps) {
    // the thread that makes the barriers starts the first loads at once, before the others have tensor memory
    if (tc::elect_one()) {
      tc::prefetch_tensormap(&tmap_q);
      tc::prefetch_tensormap(&tmap_k);
      tc::prefetch_tensormap(&tmap_v);
      for (int i = 0; i < (kTakeOver ? NUM_BARS : CLAIMED); ++i)
        tc::mbar_init(bar(i), (i >= P_HEAD0 && i <= P_FULL1) ? kSoftmaxWarps / 2 : i == TILE_EMPTY ? kSoftmaxWarps + 2 : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      if (kTakeOver) put_tile(0, w);
      const int n1 = dense_blocks(p, w, 1);
      if (max(dense_blocks(p, w, 0), n1) > 0) {
        load_q(n1 > 0);
        load_k(0, 0, 0);
        load_v(0, 1);
      }
    }
    __syncwarp();
  }
  if (warp == kSoftmaxWarps + 1) tc::tmem_alloc(sbase + L::MISC_OFF, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *sTmem;

  if (warp == kSoftmaxWarps) {
    // ================================ TMA producer =====================================
    if (tc::elect_one()) {
      int qc = 0, kc = 0;                  // Q tiles, key blocks so far
      tc::RingPos<L::kStages> at = {0, 0u};
      bool alive = true;
      for (int n = 0; alive; ++n) {
        const int n1 = dense_blocks(p, w, 1), nblk = max(dense_blocks(p, w, 0), n1);
        for (int j = 0; j < nblk && alive; ++j, ++kc) {
          if (n == 0 && j == 0) {                               // under way since the start
            if (kTakeOver && nblk == 1) tc::mbar_arrive(bar(TILE_EMPTY));
            at.step(2);
            continue;
          }
          alive = tc::mbar_wait(bar(EMPTY0 + at.st), at.ph ^ 1, status, 41);
          if (!alive) break;
          load_k(j, at.st, kc);
          at.step(1);
          if (kTakeOver && j == nblk - 1) tc::mbar_arrive(bar(TILE_EMPTY));      // two blocks to go: the next tile may be claimed
          if (j == 0) {                                         // every S of the tile before has been formed
            alive = tc::mbar_wait(bar(Q_EMPTY), (qc & 1) ^ 1, status, 40);
            if (!alive) break;
            load_q(n1 > 0);
          }
          alive = tc::mbar_wait(bar(EMPTY0 + at.st), at.ph ^ 1, status, 42);
          if (alive) load_v(j, at.st);
          at.step(1);
        }
        if (!kTakeOver) break;
        if (nblk > 0) ++qc;
        else tc::mbar_arrive(bar(TILE_EMPTY));
        if (!alive || !tc::mbar_wait(bar(TILE_FULL), n & 1, status, 50)) break;
        w = get_tile(n + 1);
        if (!w.valid) break;
      }
    }
  } else if (warp == kSoftmaxWarps + 1) {
    // ================================ MMA issuer =======================================
    if (tc::elect_one()) {
      constexpr uint32_t idesc_s = tc::idesc_bf16_f32(128, 128, 0, 0);
      constexpr uint32_t idesc_o = tc::idesc_bf16_f32(128, 128, 0, 1);
      const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);               // A of S: K-major (tile 0)
      const uint64_t desc_k = tc::smem_desc_sw128(sRing, 16, 1024);            // B of S: K-major (stage 0)
      const uint64_t desc_r = tc::smem_desc_sw128(sRest, 16, 1024);            // the same, columns 128 to 191 (slot 0)
      const uint64_t desc_v = tc::smem_desc_sw128(sRing, kChunkBytes, 1024);   // B of PV: MN-major, 64-wide column groups 16 KB apart (stage 0)
      tc::RingPos<L::kStages> at_k = {0, 0u}, at_v = {1, 0u};
      int qc = 0, kc = 0, c0 = 0, c1 = 0;      // Q tiles, key blocks, blocks of either tile before this one
      bool alive = true;
      if (kTakeOver) tc::mbar_arrive(bar(TILE_EMPTY));
      for (int n = 0; alive; ++n) {
        const int n0 = dense_blocks(p, w, 0), n1 = dense_blocks(p, w, 1), nblk = max(n0, n1);
        if (nblk > 0) alive = tc::mbar_wait(bar(Q_FULL), qc & 1, status, 43);
        for (int j = -1; j < nblk && alive; ++j) {
          if (j >= 0) alive = tc::mbar_wait(bar(FULL0 + at_v.st), at_v.ph, status, 44);
          // S overwrites the columns P of its tile was just read from: the tensor pipe runs in order.  (The first P V of the next
          // CTA tile overwrites O: its P arrives after the epilogue, which the same warps run before, has read O.)
#pragma unroll 1
          for (int t = 0; t < 2 && alive; ++t) {
            const int n_t = t ? n1 : n0;
            const bool pv = j >= 0 && j < n_t, s = j + 1 < n_t;
            const bool last_tile = t == 1 || n1 == 0;                   // the last one to read K, V and Q (n1 >= n0 or n1 == 0)
            if (pv) {
              const uint32_t parity = ((t ? c1 : c0) + j) & 1, tmem_o = tmem + TMEM_O + t * 128, tmem_p = tmem + TMEM_S + t * 128;
              const uint64_t v = tc::desc_advance(desc_v, at_v.st * kVBytes);
              alive = tc::mbar_wait(bar(P_HEAD0 + t), parity, status, 45);
              if (!alive) break;
              tc::tc_fence_after();
              dense_pv_steps<0, 4>(tmem_o, tmem_p, v, idesc_o, j == 0);
              alive = tc::mbar_wait(bar(P_FULL0 + t), parity, status, 48);
              if (!alive) break;
              tc::tc_fence_after();
              dense_pv_steps<4, 8>(tmem_o, tmem_p, v, idesc_o, false);
              if (!s) tc::tc_commit(bar(O_DONE0 + t));
              if (last_tile) tc::tc_commit(bar(EMPTY0 + at_v.st));
            }
            if (t == 0 && j + 1 < nblk) {
              alive = tc::mbar_wait(bar(FULL0 + at_k.st), at_k.ph, status, 46);
              if (!alive) break;
              tc::tc_fence_after();
            }
            if (s) {
              dense_s_block<D_QK>(tmem + TMEM_S + t * 128, tc::desc_advance(desc_q, t * L::kTileBytes), tc::desc_advance(desc_k, at_k.st * kVBytes),
                                  tc::desc_advance(desc_r, ((kc + j + 1) & 1) * kChunkBytes), idesc_s);
              tc::tc_commit(bar(S_FULL0 + t));
              if (last_tile) {
                tc::tc_commit(bar(EMPTY0 + at_k.st));
                if (j + 1 == nblk - 1) tc::tc_commit(bar(Q_EMPTY));
              }
            }
          }
          if (j >= 0) at_v.step(2);
          if (j + 1 < nblk) at_k.step(2);
        }
        if (!kTakeOver || !alive) break;
        if (nblk > 0) ++qc;
        kc += nblk;
        c0 += n0;
        c1 += n1;
        alive = tc::mbar_wait(bar(TILE_FULL), n & 1, status, 50);
        tc::mbar_arrive(bar(TILE_EMPTY));
        w = get_tile(n + 1);
        if (!w.valid) break;
      }
    }
  } else if (kTakeOver && warp == kSoftmaxWarps + 2) {
    // ================================ next tiles =======================================
    // Tile n is claimed when every consuming warp has begun tile n - 1, and so is done with tile n - 2, in whose place it is
    // described, and when the loads of tile n - 1 near their end: a tile claimed a whole tile ahead waits for its CTA while others
    // run out of work (4 sequences of 2000 to 4000 tokens, 16 heads, 192/128: 252 -> 276 us).
    if (tc::elect_one()) {
      int claims = 0;
      bool alive = true;
      for (int n = 1; alive; ++n) {
        alive = tc::mbar_wait(bar(TILE_EMPTY), (n - 1) & 1, status, 38);
        if (!alive) break;
        DenseTile t = {};
        for (;;) {
          tc::fence_proxy_async_smem();                // the answer before has been read
          tc::mbar_arrive_expect_tx(bar(CLAIMED), 16);
          claim_next_cta(sbase + L::CLAIM_OFF, bar(CLAIMED));
          alive = tc::mbar_wait(bar(CLAIMED), claims & 1, status, 39);
          ++claims;
          const int index = alive ? claimed_cta(sbase + L::CLAIM_OFF) : -1;
          t.valid = index >= 0;
          if (!t.valid) break;
          t = dense_tile(p, index);
          if (t.m_base < t.lq) break;
        }
        if (t.valid) {                                 // its Q comes from HBM: into L2 while the tile before is worked on
          const int tiles = dense_blocks(p, t, 1) > 0 ? 2 : 1;
          for (int i = 0; i < tiles; ++i)
#pragma unroll
            for (int c = 0; c < L::NCH; ++c) tma_prefetch_l2_3d(&tmap_q, c * 64, t.head, t.q0 + t.m_base + i * 128);
        }
        put_tile(n, t);
        tc::mbar_arrive(bar(TILE_FULL));
        if (!t.valid) break;
      }
    }
  } else {
    // ================================ softmax / epilogue ================================
    const int t = warp >> 2;                                   // the tile this warp works for
    const int rl = (warp & 3) * 32 + lane;                     // row within the tile = TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lane_addr + TMEM_S + t * 128;
    const uint32_t o_addr = tmem + lane_addr + TMEM_O + t * 128;
    bool alive = true;
    int c_blk = 0, c_o = 0, c_key = 0;                         // blocks and accumulators of this tile position, key blocks so far
    if (kTakeOver && lane == 0) tc::mbar_arrive(bar(TILE_EMPTY));
    for (int n = 0; alive; ++n) {
      int n_mine, n_key, limit, tail;                          // tail: keys of the sequence's last block, if it is among these
      bool first_pv;                                           // in the last key block this tile's P V comes first
      {
        const DenseTile tile = kTakeOver ? get_tile(n) : w;
        n_mine = dense_blocks(p, tile, t);
        const int n_other = dense_blocks(p, tile, t ^ 1);
        n_key = max(n_mine, n_other);
        first_pv = n_mine == n_key && (t == 0 || n_other < n_mine);
        tail = tile.lk - (n_key - 1) * 128;
        // number of keys this row may see: bottom-right aligned causal mask, clipped to the sequence
        limit = p.is_causal ? max(0, min(tile.lk, tile.m_base + t * 128 + rl + (tile.lk - tile.lq) + 1)) : tile.lk;
      }
      float m_used = neg_inf();    // the scale O and l carry (-inf: no visible key yet)
      float m_limit = neg_inf();   // the largest scaled logit for which it serves
      F2 l_run = f2(0.f);          // row sum, of even and odd keys
      for (int j = 0; j < n_mine; ++j, ++c_blk) {
        alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(S_FULL0 + t), c_blk & 1, status, 47));
        if (!alive) break;
        tc::tc_fence_after();
        const int cnt = limit - j * 128;                       // visible keys of this block: [0, cnt)
        if (__builtin_expect(!__all_sync(0xffffffffu, cnt >= 128), 0)) {
          // masked logits become -inf in tensor memory: the code below, short as it is, serves every block
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t sv[32];
            tc::tmem_ld32(s_addr + c * 32, sv);
            tc::tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= cnt) sv[i] = 0xff800000u;      // a select: what lies beyond may hold anything
            tc::tmem_st32(s_addr + c * 32, sv);
          }
          tc::tmem_wait_st();
          // V rows past the end of the sequence belong to the next sequence (or are the zero fill): the tile whose P V comes
          // first clears them, so that 0 * (Inf or NaN) cannot reach O
          if (tail < 128 && first_pv && j == n_key - 1) {
            const int item = 2 * (c_key + j) + 1, st = item % L::kStages;
            alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(FULL0 + st), (item / L::kStages) & 1, status, 51));
            unsigned char* v = smem + L::RING_OFF + st * kVBytes;
            for (int i = rl; i < (128 - tail) * 16; i += 128) {
              const int row = tail + (i >> 4), c16 = i & 15;
              *reinterpret_cast<uint4*>(v + (c16 >> 3) * kChunkBytes + row * 128 + (c16 & 7) * 16) = make_uint4(0, 0, 0, 0);
            }
            tc::fence_proxy_async_smem();
          }
        }
        float top, mx;
        {
          uint32_t sv[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tc::tmem_ld32(s_addr + c * 32, sv[c]);
          tc::tmem_wait_ld();
          float m4[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            m4[c] = __uint_as_float(sv[c][0]);
#pragma unroll
            for (int i = 1; i + 1 < 32; i += 2) m4[c] = max3_nan(m4[c], __uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1]));
            m4[c] = max3_nan(m4[c], m4[c], __uint_as_float(sv[c][31]));
          }
          top = max3_nan(max3_nan(m4[0], m4[1], m4[2]), m4[3], m4[3]);
          mx = top * p.scale_log2;
        }
        // The scale moves only when a logit exceeds it by more than the threshold (or is NaN).
        const bool up = !(mx <= m_limit);
        if (__any_sync(0xffffffffu, up)) {
          float alpha = 1.f;
          if (up) {
            float m_new = !(mx <= m_used) ? mx : m_used;
            // An infinite logit makes the row NaN, as inf - inf would; so does an exponent above 2^7, which takes the rounding of a
            // scaled logit of 2^32 and more: each block of such a row comes here.  (A cut of every exponent costs every call 1 to 2.5 %: 4 x 1000
            // tokens, 8 heads, 192/128, causal 21.2 -> 21.7 us.)
            if (mx == pos_inf() || fmaf(top, p.scale_log2, -m_new) >= 128.f) m_new = __int_as_float(0x7fffffff);
            // the first visible key sets the scale: O and l are exactly zero so far
            if (m_used != neg_inf()) alpha = exp2f(m_used - m_new);
            m_used = m_new;
            m_limit = fabsf(m_new) >= kWideScale ? neg_inf() : m_new + kRescaleThreshold;
          }
          l_run.lo *= alpha;
          l_run.hi *= alpha;
          // O is complete: the P V before this S has been through the tensor pipe before it
          if (j > 0) {
#pragma unroll 1
            for (int c = 0; c < 8; ++c) {
              uint32_t ov[16];
              tc::tmem_ld16(o_addr + c * 16, ov);
              tc::tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tc::tmem_st16(o_addr + c * 16, ov);
            }
          }
        }
        // P = 2^(s * scale - m) as bf16 pairs over the first 64 of the 128 columns S came from
        const F2 scale = f2(p.scale_log2), m_neg = f2(m_used == neg_inf() ? 0.f : -m_used);
        F2 sum[2] = {f2(0.f), f2(0.f)};
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          uint32_t sv[2][32];
#pragma unroll
          for (int c = 0; c < 2; ++c) tc::tmem_ld32(s_addr + h * 64 + c * 32, sv[c]);
          tc::tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              F2 x = f2_fma(F2{__uint_as_float(sv[c][2 * i]), __uint_as_float(sv[c][2 * i + 1])}, scale, m_neg);
              if (i % kPolyPeriod == kPolyPeriod - 1) {
                x = f2_exp2_to_128(x);
              } else {
                x.lo = exp2f(x.lo);
                x.hi = exp2f(x.hi);
              }
              sum[i & 1] = f2_add(sum[i & 1], x);
              pk[i] = pack_bf16x2(x.lo, x.hi);
            }
            tc::tmem_st16(s_addr + h * 32 + c * 16, pk);
          }
          tc::tmem_wait_st();
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(bar((h ? P_FULL0 : P_HEAD0) + t));
        }
        l_run = f2_add(l_run, f2_add(sum[0], sum[1]));
      }
      c_key += n_key;

      // ---- epilogue -------------------------------------------------------------------------
      bool have_o = n_mine > 0 && alive;
      if (have_o) {
        have_o = alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(O_DONE0 + t), c_o & 1, status, 49));
        ++c_o;
        tc::tc_fence_after();
      }
      const DenseTile tile = kTakeOver ? get_tile(n) : w;      // (read again: it need not stay in registers through the loop)
      const int row = tile.m_base + t * 128 + rl;              // query row within its sequence
      const bool row_ok = row < tile.lq;
      const float l_row = l_run.lo + l_run.hi;
      const float inv = (l_row == 0.f || !have_o) ? 0.f : 1.f / l_row;
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.o) + (int64_t)(tile.q0 + row) * p.o_stride_t + tile.head * p.o_stride_h;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t ov[32];
        if (have_o) {
          tc::tmem_ld32(o_addr + c * 32, ov);
          tc::tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = 0u;
        }
        if (row_ok) {
#pragma unroll
          for (int q8 = 0; q8 < 2; ++q8) {
            uint32_t o8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
              o8[i] = pack_bf16x2(__uint_as_float(ov[q8 * 16 + 2 * i]) * inv, __uint_as_float(ov[q8 * 16 + 2 * i + 1]) * inv);
            st_global_32B(orow + c * 32 + q8 * 16, o8);
          }
        }
      }
      if (row_ok)
        p.lse[(int64_t)(tile.q0 + row) * p.lse_stride_t + tile.head * p.lse_stride_h] = inv == 0.f ? neg_inf() : (log2f(l_row) + m_used) * kLn2;
      if (!kTakeOver) break;
      tc::tc_fence_before();                                   // O has been read: the next tile's first P V comes after its P
      if (!alive || !await_tile(n + 1) || !get_tile(n + 1).valid) break;
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if (warp == kSoftmaxWarps + 1) tc::tmem_dealloc(tmem, 512);
}

// ---- host side ----------------------------------------------------------------------------------
template <int D_QK>
static cudaError_t launch_fwd_tc(DenseKernelParams p, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                 cudaStream_t stream) {
  using L = dft::Layout<D_QK>;
  // Order of the CTAs.  Tiles outermost (all heads of all sequences start with their longest tile, the shortest ones fill the
  // last wave) pays with a causal mask while the keys and values of all heads stay in L2 together: device time of tiles
  // innermost over outermost 1.02 to 1.64 up to 64 MB of them (24 MB, 3 sequences of 2048, 8 heads: 64 against 39 us), 0.93 to
  // 1.19 from there to 200 MB, 0.80 to 1.05 beyond.  Otherwise the tiles of one head run side by side and read its keys from
  // L2; without a mask all tiles are alike, and innermost over outermost is 0.75 to 1.06.
  p.tiles_outer = p.is_causal && (int64_t)p.total_k * p.h_k * (p.d_qk + p.d_v) * 2 <= (64 << 20);
  const int64_t ctas = (int64_t)((p.max_seqlen_q + 255) / 256) * p.h_q * p.batch;
  if (ctas > INT32_MAX) return cudaErrorInvalidConfiguration;
  // Taking CTAs over pays as soon as there are more CTAs with rows than SMs, and costs 0.2 to 0.3 us below.  Sequences shorter than the
  // longest leave CTAs without rows, which count for nothing here: no more than (total_q / 256 + batch) per head have some.  Device
  // time in a graph, plain -> taking over: 80 CTAs (4 sequences of 500 tokens, 10 heads, 192/128) 13.5 -> 13.9 us, 144 (18 heads) 14.3 -> 14.6, 160
  // (4 of 200, 40 heads) 18.5 -> 16.5, 256 (32 heads) 24.3 -> 21.0, 512 (8 of 512, 32 heads, 128/128) 47.6 -> 37.6, 2048 (64 of 64) 81.6 -> 47.7;
  // 480 of which 208 have rows (1500, 700, 300, 100 and 20 tokens, 16 heads, 192/128) 28.8 -> 29.4.  So the line, 1.9 CTAs per SM, lies too high
  // for the present kernel: it was drawn for one that lost up to 8 % below it, and has not been moved since.
  // Neither has that of 2048 keys at 192/128: longer tiles lost 2 to 3 % once, and would gain 1 to 7 % now (4 of 8192 tokens, 16 heads,
  // causal 1268 -> 1217 us, 8 of 4096 696 -> 648, no mask 1196 -> 1165).
  int dev = 0, sms = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  if (cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); e != cudaSuccess) return e;
  const int64_t with_rows = std::min<int64_t>(ctas, (static_cast<int64_t>(p.total_q / 256) + p.batch) * p.h_q);
  const int64_t keys = p.total_k / p.batch / (p.is_causal ? 2 : 1);
  const bool takes_over = with_rows * 8 >= sms * 15 && (D_QK == 128 || keys <= 2048);
  auto launch = [&](auto take_over) {
    constexpr auto kern = dense_fwd_tc_kernel<D_QK, decltype(take_over)::value>;
    if (cudaError_t e = allow_smem<kern>(L::SMEM_BYTES); e != cudaSuccess) return e;
    kern<<<static_cast<unsigned>(ctas), dft::threads(decltype(take_over)::value), L::SMEM_BYTES, stream>>>(p, tq, tk, tv);
    return cudaGetLastError();
  };
  return takes_over ? launch(std::true_type{}) : launch(std::false_type{});
}

cudaError_t launch_dense_fwd_tc(const DenseKernelParams& p, cudaStream_t stream) {
  CUtensorMap tq, tk, tv;
  if (!tmah::make_map_thd(&tq, p.q, p.d_qk, p.h_q, p.total_q, p.q_stride_h, p.q_stride_t, 128)) return cudaErrorInvalidValue;
  if (!tmah::make_map_thd(&tk, p.k, p.d_qk, p.h_k, p.total_k, p.k_stride_h, p.k_stride_t, 128)) return cudaErrorInvalidValue;
  if (!tmah::make_map_thd(&tv, p.v, p.d_v, p.h_k, p.total_k, p.v_stride_h, p.v_stride_t, 128)) return cudaErrorInvalidValue;
  if (p.d_qk == 192) return launch_fwd_tc<192>(p, tq, tk, tv, stream);
  return launch_fwd_tc<128>(p, tq, tk, tv, stream);
}

cudaError_t set_status_mirror_dense_fwd(int* mapped_host_word) { return tc::set_status_mirror(mapped_host_word); }

cudaError_t read_dense_tc_status(int* host_status, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(host_status, g_dense_tc_status, sizeof(int));
  if (e != cudaSuccess) return e;
  if (reset && *host_status != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_dense_tc_status, &zero, sizeof(int));
  }
  return e;
}

}  // namespace fmla
