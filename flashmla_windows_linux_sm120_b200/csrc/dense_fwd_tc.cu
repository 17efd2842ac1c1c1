// Dense variable-length MHA forward (bf16, head dims 192/128 and 128/128) for sm_100a on
// tcgen05 / TMA / tensor memory.
//
// One CTA = 256 query rows (two tiles of 128) of one (sequence, head) at a time; keys are walked in blocks of 128.
//   warps 0-7  softmax of tile 0, warps 8-15 softmax of tile 1: two threads per query row (TMEM lane = row), one for each
//              half of the 128 keys: S -> registers, mask, P (bf16) written back into the columns S came from, row
//              sums, final 1/l normalisation and stores
//   warp 16    TMA: both Q tiles once; K blocks into a 2-stage ring, V blocks into a single stage (two at 128/128)
//              (64-column chunks of [128 rows x 128 bytes], 128-byte swizzle)
//   warp 17    MMA: S_t = Q_t K^T (tcgen05.mma m128n128k16, both operands from shared memory),
//              O_t += P_t V (m128n128k16, P from tensor memory, V from shared memory MN-major), in the
//              order  P V of tile 0, S of tile 0 for the next block, P V of tile 1, S of tile 1 for the
//              next block: while the softmax of one tile runs, the tensor pipe works for the other tile.
//   warp 18    in large grids: takes over CTAs that have not been started (clusterlaunchcontrol), one after the other
// What bounds it: a tile's chain S -> softmax -> P V -> S (P lies over S, and tensor memory has no room for a second S), of
// which the tensor pipe can hide the part that is as long as the other tile's two GEMMs (1280 clk at 192/128, 1024 at
// 128/128).  Hence two threads per row: with one, the 128 logits of a row took a thread longer than that.
// The scale m_used of a row moves only when one of its logits exceeds it by more than 2^8: each of the two threads
// compares its own maximum, and one barrier-with-reduction of their two warps decides; only then the maxima are
// exchanged, O is rescaled and the exponentials are formed again.
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
constexpr int kSoftmaxWarps = 16;
constexpr int threads(bool take_over) { return (kSoftmaxWarps + 2 + take_over) * 32; }
enum Bar { Q_FULL = 0, Q_EMPTY, K_FULL0, K_FULL1, K_EMPTY0, K_EMPTY1, V_FULL0, V_FULL1, V_EMPTY0, V_EMPTY1, S_FULL0, S_FULL1, P_FULL0, P_FULL1, PV_DONE0,
           PV_DONE1, O_DONE0, O_DONE1, CLAIMED, TILE_FULL, TILE_EMPTY, NUM_BARS };
constexpr int TMEM_S = 0, TMEM_O = 256;
constexpr float kRescaleThreshold = 8.0f;         // log2 units; below it O keeps its stale scale
template <int D_QK>
struct Layout {
  static constexpr int NCH = D_QK / 64;           // 64-column chunks of Q and K
  static constexpr int kTileBytes = NCH * kChunkBytes;    // one Q tile / one K block
  static constexpr int Q_OFF = 0;                 // 2 tiles
  static constexpr int K_OFF = 2 * kTileBytes;    // 2 stages
  static constexpr int V_OFF = K_OFF + 2 * kTileBytes;
  static constexpr int kVStages = D_QK == 192 ? 1 : 2;
  static constexpr int BAR_OFF = V_OFF + kVStages * kVBytes;
  static constexpr int X_OFF = BAR_OFF + 192;     // float [tile][half][128]: exchange between the two threads of a row
  static constexpr int MISC_OFF = X_OFF + 2048;
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
__device__ __forceinline__ void dense_s_block(uint32_t tmem_s, uint64_t desc_q, uint64_t desc_k, uint32_t idesc) {
  using L = dft::Layout<D_QK>;
#pragma unroll
  for (int c = 0; c < L::NCH; ++c)
#pragma unroll
    for (int s = 0; s < 4; ++s)
      tc::mma_ss(tmem_s, tc::desc_advance(desc_q, c * dft::kChunkBytes + s * 32), tc::desc_advance(desc_k, c * dft::kChunkBytes + s * 32), idesc,
                 (c | s) ? 1u : 0u);
}
// O += P V of one tile and key block: P from the S columns of the tile (8 columns per 16-token step; the second half of
// the tokens 64 columns further on: each softmax warp writes over the half it has read).
__device__ __forceinline__ void dense_pv_block(uint32_t tmem_o, uint32_t tmem_p, uint64_t desc_v, uint32_t idesc, bool first) {
#pragma unroll
  for (int s = 0; s < 8; ++s)
    tc::mma_ts(tmem_o, tmem_p + (s >> 2) * 64 + (s & 3) * 8, tc::desc_advance(desc_v, s * 2048), idesc, (first && s == 0) ? 0u : 1u);
}

// barrier over the 64 threads of two warps that also tells whether any of them passed true
__device__ __forceinline__ bool pair_any(int id, bool x) {
  uint32_t r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %2, 0;\nbarrier.cta.red.or.aligned.pred q, %1, 64, p;\nselp.u32 %0, 1, 0, q;\n}\n"
               : "=r"(r)
               : "r"(id), "r"(static_cast<uint32_t>(x))
               : "memory");
  return r != 0;
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
// CTAs that have not been started (warp 18), so that the loads and first products of its next tile overlap the last softmax,
// the read of O and the stores of the present one; barriers, tensor memory and tensor maps are set up once.
template <int D_QK, bool kTakeOver>
__global__ void __launch_bounds__(dft::threads(kTakeOver), 1)
dense_fwd_tc_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_q,
                    const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v) {
  using namespace dft;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + L::Q_OFF, sK = sbase + L::K_OFF, sV = sbase + L::V_OFF;
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
  auto load_k = [&](int j, int st) {
    tc::mbar_arrive_expect_tx(bar(K_FULL0 + st), L::kTileBytes);
#pragma unroll
    for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(sK + st * L::kTileBytes + c * kChunkBytes, &tmap_k, c * 64, w.head / group, w.k0 + j * 128, bar(K_FULL0 + st));
  };
  auto load_v = [&](int j, int st) {
    tc::mbar_arrive_expect_tx(bar(V_FULL0 + st), kVBytes);
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tma_load_3d(sV + st * kVBytes + c * kChunkBytes, &tmap_v, c * 64, w.head / group, w.k0 + j * 128, bar(V_FULL0 + st));
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
        tc::mbar_init(bar(i), (i == P_FULL0 || i == P_FULL1) ? kSoftmaxWarps / 2 : i == TILE_EMPTY ? kSoftmaxWarps + 2 : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      if (kTakeOver) put_tile(0, w);
      const int n1 = dense_blocks(p, w, 1);
      if (max(dense_blocks(p, w, 0), n1) > 0) {
        load_q(n1 > 0);
        load_k(0, 0);
        load_v(0, 0);
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
      int qc = 0, kc = 0;                  // Q tiles, key blocks of the tiles before
      bool alive = true;
      for (int n = 0; alive; ++n) {
        const int n1 = dense_blocks(p, w, 1), nblk = max(dense_blocks(p, w, 0), n1);
        for (int j = 0; j < nblk && alive; ++j) {
          if (n == 0 && j == 0) {                               // under way since the start
            if (kTakeOver && nblk == 1) tc::mbar_arrive(bar(TILE_EMPTY));
            continue;
          }
          const int c = kc + j;
          alive = tc::mbar_wait(bar(K_EMPTY0 + (c & 1)), ((c >> 1) & 1) ^ 1, status, 41);
          if (!alive) break;
          load_k(j, c & 1);
          if (kTakeOver && j == nblk - 1) tc::mbar_arrive(bar(TILE_EMPTY));      // two blocks to go: the next tile may be claimed
          if (j == 0) {                                         // every S of the tile before has been formed
            alive = tc::mbar_wait(bar(Q_EMPTY), (qc & 1) ^ 1, status, 40);
            if (!alive) break;
            load_q(n1 > 0);
          }
          alive = tc::mbar_wait(bar(V_EMPTY0 + c % L::kVStages), ((c / L::kVStages) & 1) ^ 1, status, 42);
          if (alive) load_v(j, c % L::kVStages);
        }
        if (!kTakeOver) break;
        kc += nblk;
        if (nblk > 0) ++qc;
        else tc::mbar_arrive(bar(TILE_EMPTY));
        if (!alive || !tc::mbar_wait(bar(TILE_FULL), n & 1, status, 50)) break;
        w = get_tile(n + 1);
        if (!w.valid) break;
      }
    }
  } else if (warp == kSoftmaxWarps + 1) {
    // ================================ MMA issuer =======================================
    constexpr uint32_t idesc_s = tc::idesc_bf16_f32(128, 128, 0, 0);
    constexpr uint32_t idesc_o = tc::idesc_bf16_f32(128, 128, 0, 1);
    const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);               // A of S: K-major (tile 0)
    const uint64_t desc_k = tc::smem_desc_sw128(sK, 16, 1024);               // B of S: K-major (stage 0)
    const uint64_t desc_v = tc::smem_desc_sw128(sV, kChunkBytes, 1024);      // B of PV: MN-major, 64-wide column groups 16 KB apart (stage 0)
    int qc = 0, kc = 0, c0 = 0, c1 = 0;      // Q tiles, key blocks, blocks of either tile before this one
    bool alive = true;
    if (kTakeOver && lane == 0) tc::mbar_arrive(bar(TILE_EMPTY));
    for (int n = 0; alive; ++n) {
      const int n0 = dense_blocks(p, w, 0), n1 = dense_blocks(p, w, 1), nblk = max(n0, n1);
      if (nblk > 0) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(Q_FULL), qc & 1, status, 43));
      for (int j = -1; j < nblk && alive; ++j) {
        const int stv = (kc + j) % L::kVStages, stk = (kc + j + 1) & 1;
        if (j >= 0) {
          alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(V_FULL0 + stv), ((kc + j) / L::kVStages) & 1, status, 44));
          if (!alive) break;
          // V rows past the end of the sequence belong to the next sequence (or are the zero fill) and are
          // cleared first, so that 0 * (Inf or NaN) cannot reach O
          const int rows_valid = w.lk - j * 128;
          if (rows_valid < 128) {
            unsigned char* v = smem + L::V_OFF + stv * kVBytes;
            const int nrows = 128 - rows_valid;
            for (int i = lane; i < nrows * 16; i += 32) {
              const int row = rows_valid + (i >> 4), c16 = i & 15;
              *reinterpret_cast<uint4*>(v + (c16 >> 3) * kChunkBytes + row * 128 + (c16 & 7) * 16) = make_uint4(0, 0, 0, 0);
            }
            tc::fence_proxy_async_smem();
            __syncwarp();
          }
        }
        // S overwrites the columns P of its tile was just read from: the tensor pipe runs in order.  (The first P V of the next
        // CTA tile overwrites O: its P arrives after the epilogue, which the same warps run before, has read O.)
        // The issuing thread is held until the pipe has taken its instructions, and a wait after that costs some 100 clk even for a
        // barrier that is complete; still, an issuing warp per tile (the instructions of both tiles interleave, and both
        // chains get longer: 600 keys, 8 heads 18.4 -> 22.5 us) and key blocks of 64 with two S buffers (twice the waits: three
        // sequences of 1129 to 1950 tokens, 32 heads 102 -> 127 us) were slower, P V and S in one go no faster.
#pragma unroll 1
        for (int t = 0; t < 2 && alive; ++t) {
          const int n_t = t ? n1 : n0;
          const bool pv = j >= 0 && j < n_t, s = j + 1 < n_t;
          const bool last_tile = t == 1 || n1 == 0;                     // the last one to read K, V and Q (n1 >= n0 or n1 == 0)
          if (pv) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(P_FULL0 + t), ((t ? c1 : c0) + j) & 1, status, 45));
          if (!alive) break;
          tc::tc_fence_after();
          if (pv && tc::elect_one()) {
            dense_pv_block(tmem + TMEM_O + t * 128, tmem + TMEM_S + t * 128, tc::desc_advance(desc_v, stv * kVBytes), idesc_o, j == 0);
            tc::tc_commit(bar(PV_DONE0 + t));
            if (!s) tc::tc_commit(bar(O_DONE0 + t));
            if (last_tile) tc::tc_commit(bar(V_EMPTY0 + stv));
          }
          __syncwarp();
          if (t == 0 && j + 1 < nblk) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(K_FULL0 + stk), ((kc + j + 1) >> 1) & 1, status, 46));
          if (!alive) break;
          tc::tc_fence_after();
          if (s && tc::elect_one()) {
            dense_s_block<D_QK>(tmem + TMEM_S + t * 128, tc::desc_advance(desc_q, t * L::kTileBytes), tc::desc_advance(desc_k, stk * L::kTileBytes), idesc_s);
            tc::tc_commit(bar(S_FULL0 + t));
            if (last_tile) {
              tc::tc_commit(bar(K_EMPTY0 + stk));
              if (j + 1 == nblk - 1) tc::tc_commit(bar(Q_EMPTY));
            }
          }
          __syncwarp();
        }
      }
      if (!kTakeOver || !alive) break;
      if (nblk > 0) ++qc;
      kc += nblk;
      c0 += n0;
      c1 += n1;
      alive = await_tile(n + 1);
      w = get_tile(n + 1);
      if (!w.valid) break;
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
    const int t = warp >> 3, half = (warp >> 2) & 1;           // the tile this warp works for, its half of the columns
    const int rl = (warp & 3) * 32 + lane;                     // row within the tile = TMEM lane
    const int pair_bar = 1 + t * 4 + (warp & 3);               // this warp and the one with the other half of its rows
    float* x_mine = reinterpret_cast<float*>(smem + L::X_OFF) + t * 256 + half * 128 + rl;
    float* x_other = reinterpret_cast<float*>(smem + L::X_OFF) + t * 256 + (half ^ 1) * 128 + rl;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lane_addr + TMEM_S + t * 128 + half * 64;
    const uint32_t o_addr = tmem + lane_addr + TMEM_O + t * 128 + half * 64;
    // A wait that expires clears `alive`; the warp then walks the rest of its blocks without work, because the other warp
    // of the pair counts on it at their barriers, and both leave after the tile.
    bool alive = true;
    int c_blk = 0, c_o = 0;                                    // blocks and accumulators of this tile position so far
    if (kTakeOver && lane == 0) tc::mbar_arrive(bar(TILE_EMPTY));
    for (int n = 0;; ++n) {
      int n_mine, limit;
      {
        const DenseTile tile = kTakeOver ? get_tile(n) : w;
        n_mine = dense_blocks(p, tile, t);
        // number of keys this row may see: bottom-right aligned causal mask, clipped to the sequence
        limit = p.is_causal ? max(0, min(tile.lk, tile.m_base + t * 128 + rl + (tile.lk - tile.lq) + 1)) : tile.lk;
      }
      float m_used = neg_inf();    // the scale O and l carry (-inf: no visible key yet)
      float l_run = 0.f;           // this thread's share of the row sum
      for (int j = 0; j < n_mine; ++j, ++c_blk) {
        if (alive) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(S_FULL0 + t), c_blk & 1, status, 47));
        tc::tc_fence_after();
        const int cnt = limit - j * 128 - half * 64;           // visible keys of this half block: [0, cnt)
        const bool full = __all_sync(0xffffffffu, cnt >= 64);
        // 32 logits at a time: 64 beside their P do not fit into the 96 registers that 18 or 19 warps leave a thread
        auto load_logits = [&](int c, uint32_t (&sv)[32]) {
          tc::tmem_ld32(s_addr + c * 32, sv);
          tc::tmem_wait_ld();
          if (!full) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= cnt) sv[i] = 0xff800000u;      // a select: what lies beyond may hold anything
          }
        };
        // P = 2^(s * scale - m) of this thread's 64 logits as bf16 pairs, their sum and their largest logit
        uint32_t pk[2][16];
        float row_sum = 0.f, mx = neg_inf();
        auto exponentials = [&](float m) {
          const float m_ref = m == neg_inf() ? 0.f : m;
          float rs4[4] = {0.f, 0.f, 0.f, 0.f}, mx4[4] = {neg_inf(), neg_inf(), neg_inf(), neg_inf()};      // independent chains
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t sv[32];
            load_logits(c, sv);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float s0 = __uint_as_float(sv[2 * i]), s1 = __uint_as_float(sv[2 * i + 1]);
              mx4[i & 3] = fmaxf(mx4[i & 3], fmaxf(s0, s1));
              const float p0 = exp2f(fmaf(s0, p.scale_log2, -m_ref)), p1 = exp2f(fmaf(s1, p.scale_log2, -m_ref));
              rs4[i & 3] += p0 + p1;
              pk[c][i] = pack_bf16x2(p0, p1);
            }
          }
          row_sum = (rs4[0] + rs4[1]) + (rs4[2] + rs4[3]);
          mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
        };
        // The exponentials are formed with the scale of the blocks before, beside the maximum that says whether it still
        // serves; in the rare block where it does not they are formed again (S stays until P is stored).  The first block has
        // no scale yet: its maximum alone (200 tokens with 8 heads took 12.1 us with exponentials formed in vain, 11.3 without).
        if (alive && j > 0) exponentials(m_used);
        if (alive && j == 0) {
          float mx4[4] = {neg_inf(), neg_inf(), neg_inf(), neg_inf()};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t sv[32];
            load_logits(c, sv);
#pragma unroll
            for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sv[i]));
          }
          mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
        }
        if (j == 0 || pair_any(pair_bar, alive && mx > m_used + kRescaleThreshold)) {
          *x_mine = mx;
          bar_sync(pair_bar, 64);
          const float m_blk = fmaxf(mx, *x_other);
          const bool up = m_blk > m_used + kRescaleThreshold;
          // the first visible key sets the scale: O and l are exactly zero so far
          const float alpha = (up && m_used != neg_inf()) ? exp2f(m_used - m_blk) : 1.f;
          if (up) m_used = m_blk;
          l_run *= alpha;
          if (pair_any(pair_bar, alpha != 1.f)) {              // (also: x is free for the next exchange)
            // the previous P V of this tile must be complete before O is rescaled
            if (alive) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(PV_DONE0 + t), (c_blk - 1) & 1, status, 48));
            tc::tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 2 && alive; ++c) {
              uint32_t ov[32];
              tc::tmem_ld32(o_addr + c * 32, ov);
              tc::tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tc::tmem_st32(o_addr + c * 32, ov);
            }
          }
          if (alive) exponentials(m_used);
        }
        if (!alive) continue;
        // P goes over the first 32 of the 64 columns S came from
#pragma unroll
        for (int c = 0; c < 2; ++c) tc::tmem_st16(s_addr + c * 16, pk[c]);
        l_run += row_sum;
        tc::tmem_wait_st();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(P_FULL0 + t));
      }

      // ---- epilogue -------------------------------------------------------------------------
      bool have_o = n_mine > 0 && alive;
      if (have_o) {
        have_o = alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(O_DONE0 + t), c_o & 1, status, 49));
        ++c_o;
        tc::tc_fence_after();
      }
      *x_mine = l_run;
      bar_sync(pair_bar, 64);
      l_run += *x_other;
      const DenseTile tile = kTakeOver ? get_tile(n) : w;      // (read again: it need not stay in registers through the loop)
      const int row = tile.m_base + t * 128 + rl;              // query row within its sequence
      const bool row_ok = row < tile.lq;
      const float inv = (l_run == 0.f || !have_o) ? 0.f : 1.f / l_run;
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.o) + (int64_t)(tile.q0 + row) * p.o_stride_t + tile.head * p.o_stride_h + half * 64;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
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
      if (row_ok && half == 0)
        p.lse[(int64_t)(tile.q0 + row) * p.lse_stride_t + tile.head * p.lse_stride_h] = inv == 0.f ? neg_inf() : (log2f(l_run) + m_used) * kLn2;
      if (!kTakeOver) break;
      tc::tc_fence_before();                                   // O has been read: the next tile's first P V comes after its P_FULL
      if (alive) alive = await_tile(n + 1);
      if (pair_any(pair_bar, !alive) || !get_tile(n + 1).valid) break;      // (also: x has been read)
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
  // Taking CTAs over pays from nearly two CTAs with rows per SM on; below, its longer code costs what it saves.  Sequences shorter than the
  // longest leave CTAs without rows, which count for nothing here: no more than (total_q / 256 + batch) per head have some.  Device
  // time in a graph, plain -> taking over: 128 CTAs (4 sequences of 1000 tokens, 8 heads, 192/128) 24.6 -> 26.3 us, 192 (6 of 500 to 1000, 8
  // heads, 128/128) 21.9 -> 23.7, 256 (8 of 500 to 1000, 8 heads) 27.6 -> 28.6; 480 of which 208 have rows (1500, 700, 300, 100 and 20
  // tokens, 16 heads, 192/128, causal) 32.4 -> 34.8, 448 of which 160 (1000 and 6 of 30, 16 heads) 23.7 -> 25.4; 288 (9 of 250, 32 heads) 24.5 -> 21.8,
  // 288 (3 of 700) 33.7 -> 31.7, 320 (20 of 256, 16 heads) 35.8 -> 30.7, 768 (3 of 1129 to 1950, 128/128) 103.4 -> 98.2, 16384 of which 560
  // (16384 and 255 of 128, 4 heads) 863 -> 574.
  // With long tiles the loop, some 3 % slower at 192/128, outweighs the borders.  192/128, tiles of 8 blocks (16 of 1024, 16 heads, no
  // mask) 199 -> 191, 16 blocks (4 of 2048, 24 heads) 282 -> 275, 32 (8 of 4096) 1293 -> 1302, 64 (4 of 8192) 2455 -> 2524; with a causal
  // mask, which halves them, 16 of 2048 437 -> 411, 4 of 8192 1318 -> 1352; at 128/128 1194 -> 1151.
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
