// Dense variable-length MHA forward (bf16, head dims 192/128 and 128/128) for sm_100a on
// tcgen05 / TMA / tensor memory.
//
// One CTA = 256 query rows (two tiles of 128) of one (sequence, head); keys are walked in blocks of 128.
//   warps 0-7  softmax of tile 0, warps 8-15 softmax of tile 1: two threads per query row (TMEM lane = row), one for each
//              half of the 128 keys: S -> registers, mask, P (bf16) written back into the columns S came from, row
//              sums, final 1/l normalisation and stores
//   warp 16    TMA: both Q tiles once; K blocks into a 2-stage ring, V blocks into a single stage
//              (64-column chunks of [128 rows x 128 bytes], 128-byte swizzle)
//   warp 17    MMA: S_t = Q_t K^T (tcgen05.mma m128n128k16, both operands from shared memory),
//              O_t += P_t V (m128n128k16, P from tensor memory, V from shared memory MN-major), in the
//              order  P V of tile 0, S of tile 0 for the next block, P V of tile 1, S of tile 1 for the
//              next block: while the softmax of one tile runs, the tensor pipe works for the other tile.
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

namespace fmla {

namespace dft {
constexpr int kChunkBytes = 128 * 128;            // [128 rows x 64 bf16], 128-byte rows
constexpr int kVBytes = 2 * kChunkBytes;          // 128 x 128 bf16
constexpr int kSoftmaxWarps = 16, kThreads = (kSoftmaxWarps + 2) * 32;
enum Bar { Q_FULL = 0, K_FULL0, K_FULL1, K_EMPTY0, K_EMPTY1, V_FULL, V_EMPTY, S_FULL0, S_FULL1, P_FULL0, P_FULL1, PV_DONE0, PV_DONE1, NUM_BARS };
constexpr int TMEM_S = 0, TMEM_O = 256;
constexpr float kRescaleThreshold = 8.0f;         // log2 units; below it O keeps its stale scale
template <int D_QK>
struct Layout {
  static constexpr int NCH = D_QK / 64;           // 64-column chunks of Q and K
  static constexpr int kTileBytes = NCH * kChunkBytes;    // one Q tile / one K block
  static constexpr int Q_OFF = 0;                 // 2 tiles
  static constexpr int K_OFF = 2 * kTileBytes;    // 2 stages
  static constexpr int V_OFF = K_OFF + 2 * kTileBytes;
  static constexpr int BAR_OFF = V_OFF + kVBytes;
  static constexpr int X_OFF = BAR_OFF + 128;     // float [tile][half][128]: exchange between the two threads of a row
  static constexpr int MISC_OFF = X_OFF + 2048;
  static constexpr int SMEM_BYTES = MISC_OFF + 16;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared memory limit per CTA");
};
static_assert(NUM_BARS * 8 <= 128, "barrier area too small");
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

// grid: ceil(max_seqlen_q/256) * h_q * batch CTAs in the order `p.tiles_outer` selects, 576 threads
template <int D_QK>
__global__ void __launch_bounds__(dft::kThreads, 1)
dense_fwd_tc_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_q,
                    const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v) {
  using namespace dft;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + L::Q_OFF, sK = sbase + L::K_OFF, sV = sbase + L::V_OFF;
  auto bar = [&](int i) { return sbase + L::BAR_OFF + i * 8; };
  volatile uint32_t* sTmem = reinterpret_cast<volatile uint32_t*>(smem + L::MISC_OFF);
  int* status = &g_dense_tc_status;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // with a causal mask the last tiles have the most keys: they are started first
  const int n_tiles = (p.max_seqlen_q + 255) / 256, n_heads = p.h_q * p.batch;
  const int tile_rank = p.tiles_outer ? blockIdx.x / n_heads : blockIdx.x % n_tiles;
  const int bh = p.tiles_outer ? blockIdx.x % n_heads : blockIdx.x / n_tiles;
  const int b = bh / p.h_q, head = bh % p.h_q, kv_head = head / (p.h_q / p.h_k);
  const int q0 = __ldg(p.cu_q + b), lq = __ldg(p.cu_q + b + 1) - q0;
  const int k0 = __ldg(p.cu_k + b), lk = __ldg(p.cu_k + b + 1) - k0;
  const int m_base = (n_tiles - 1 - tile_rank) * 256;
  if (m_base >= lq) return;
  if ((sbase & 1023u) != 0) {   // the swizzled tiles need a 1024-byte aligned base
    if (tid == 0) tc::report_status(status, 30);
    return;
  }
  // key blocks a tile needs: those its last row sees; none for a tile without rows
  auto blocks_of = [&](int t) {
    const int first = m_base + t * 128;
    if (first >= lq) return 0;
    const int all = (lk + 127) >> 7;
    if (!p.is_causal) return all;
    const int last_key = min(first + 127, lq - 1) + (lk - lq);   // inclusive
    return last_key < 0 ? 0 : min(all, (last_key >> 7) + 1);
  };
  const int n0 = blocks_of(0), n1 = blocks_of(1), nblk = max(n0, n1);      // n1 >= n0, or n1 == 0

  auto load_q = [&] {
    tc::mbar_arrive_expect_tx(bar(Q_FULL), (n1 > 0 ? 2 : 1) * L::kTileBytes);
    for (int t = 0; t < (n1 > 0 ? 2 : 1); ++t)
#pragma unroll
      for (int c = 0; c < L::NCH; ++c)
        tc::tma_load_3d(sQ + t * L::kTileBytes + c * kChunkBytes, &tmap_q, c * 64, head, q0 + m_base + t * 128, bar(Q_FULL));
  };
  auto load_k = [&](int j) {
    const int st = j & 1;
    tc::mbar_arrive_expect_tx(bar(K_FULL0 + st), L::kTileBytes);
#pragma unroll
    for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(sK + st * L::kTileBytes + c * kChunkBytes, &tmap_k, c * 64, kv_head, k0 + j * 128, bar(K_FULL0 + st));
  };
  auto load_v = [&](int j) {
    tc::mbar_arrive_expect_tx(bar(V_FULL), kVBytes);
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tma_load_3d(sV + c * kChunkBytes, &tmap_v, c * 64, kv_head, k0 + j * 128, bar(V_FULL));
  };
  if (warp == kSoftmaxWarps) {
    // the thread that makes the barriers starts the first loads at once, before the others have tensor memory
    if (tc::elect_one()) {
      tc::prefetch_tensormap(&tmap_q);
      tc::prefetch_tensormap(&tmap_k);
      tc::prefetch_tensormap(&tmap_v);
      for (int i = 0; i < NUM_BARS; ++i) tc::mbar_init(bar(i), (i == P_FULL0 || i == P_FULL1) ? kSoftmaxWarps / 2 : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      if (nblk > 0) {
        load_q();
        load_k(0);
        load_v(0);
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
      bool alive = true;
      for (int j = 1; j < nblk && alive; ++j) {
        alive = tc::mbar_wait(bar(K_EMPTY0 + (j & 1)), ((j >> 1) & 1) ^ 1, status, 41);
        if (!alive) break;
        load_k(j);
        alive = tc::mbar_wait(bar(V_EMPTY), (j & 1) ^ 1, status, 42);
        if (!alive) break;
        load_v(j);
      }
    }
  } else if (warp == kSoftmaxWarps + 1) {
    // ================================ MMA issuer =======================================
    constexpr uint32_t idesc_s = tc::idesc_bf16_f32(128, 128, 0, 0);
    constexpr uint32_t idesc_o = tc::idesc_bf16_f32(128, 128, 0, 1);
    const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);               // A of S: K-major (tile 0)
    const uint64_t desc_k = tc::smem_desc_sw128(sK, 16, 1024);               // B of S: K-major (stage 0)
    const uint64_t desc_v = tc::smem_desc_sw128(sV, kChunkBytes, 1024);      // B of PV: MN-major, 64-wide column groups 16 KB apart
    bool alive = nblk > 0;
    if (alive) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(Q_FULL), 0, status, 43));
    // S of tile t for block j (whole warp; K(j) must have been waited for)
    auto issue_s = [&](int t, int j) {
      const int st = j & 1;
      tc::tc_fence_after();
      if (tc::elect_one()) {
        dense_s_block<D_QK>(tmem + TMEM_S + t * 128, tc::desc_advance(desc_q, t * L::kTileBytes), tc::desc_advance(desc_k, st * L::kTileBytes), idesc_s);
        tc::tc_commit(bar(S_FULL0 + t));
        if (t == 1 || j >= n1) tc::tc_commit(bar(K_EMPTY0 + st));     // the last tile to read this K block
      }
      __syncwarp();
    };
    // P V of tile t for block j
    auto issue_pv = [&](int t, int j) {
      alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(P_FULL0 + t), j & 1, status, 45));
      if (!alive) return;
      tc::tc_fence_after();
      if (tc::elect_one()) {
        dense_pv_block(tmem + TMEM_O + t * 128, tmem + TMEM_S + t * 128, desc_v, idesc_o, j == 0);
        tc::tc_commit(bar(PV_DONE0 + t));
        if (t == 1 || j >= n1) tc::tc_commit(bar(V_EMPTY));           // the last tile to read this V block
      }
      __syncwarp();
    };
    for (int j = -1; j < nblk && alive; ++j) {
      if (j >= 0) {
        alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(V_FULL), j & 1, status, 44));
        if (!alive) break;
        // V rows past the end of the sequence belong to the next sequence (or are the zero fill) and are
        // cleared first, so that 0 * (Inf or NaN) cannot reach O
        const int rows_valid = lk - j * 128;
        if (rows_valid < 128) {
          unsigned char* v = smem + L::V_OFF;
          const int nrows = 128 - rows_valid;
          for (int i = lane; i < nrows * 16; i += 32) {
            const int row = rows_valid + (i >> 4), c16 = i & 15;
            *reinterpret_cast<uint4*>(v + (c16 >> 3) * kChunkBytes + row * 128 + (c16 & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          tc::fence_proxy_async_smem();
          __syncwarp();
        }
      }
#pragma unroll 1
      for (int t = 0; t < 2 && alive; ++t) {
        const int n_t = t ? n1 : n0;
        if (j >= 0 && j < n_t) issue_pv(t, j);
        if (t == 0 && j + 1 < nblk && alive)
          alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(K_FULL0 + ((j + 1) & 1)), ((j + 1) >> 1) & 1, status, 46));
        // S overwrites the columns P of its tile was just read from: the tensor pipe runs in order
        if (j + 1 < n_t && alive) issue_s(t, j + 1);
      }
    }
  } else {
    // ================================ softmax / epilogue ================================
    const int t = warp >> 3, half = (warp >> 2) & 1;           // the tile this warp works for, its half of the columns
    const int rl = (warp & 3) * 32 + lane;                     // row within the tile = TMEM lane
    const int row = m_base + t * 128 + rl;                     // query row within its sequence
    const int n_mine = t ? n1 : n0;
    const int pair_bar = 1 + t * 4 + (warp & 3);               // this warp and the one with the other half of its rows
    float* x_mine = reinterpret_cast<float*>(smem + L::X_OFF) + t * 256 + half * 128 + rl;
    float* x_other = reinterpret_cast<float*>(smem + L::X_OFF) + t * 256 + (half ^ 1) * 128 + rl;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem + lane_addr + TMEM_S + t * 128;
    const uint32_t o_addr = tmem + lane_addr + TMEM_O + t * 128 + half * 64;
    // number of keys this row may see: bottom-right aligned causal mask, clipped to the sequence
    const int limit = p.is_causal ? max(0, min(lk, row + (lk - lq) + 1)) : lk;
    float m_used = neg_inf();    // the scale O and l carry (-inf: no visible key yet)
    float l_run = 0.f;           // this thread's share of the row sum
    // A wait that expires clears `alive`; the warp then walks the rest of its blocks without work, because the other warp
    // of the pair counts on it at their barriers.
    bool alive = true;
    for (int j = 0; j < n_mine; ++j) {
      if (alive) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(S_FULL0 + t), j & 1, status, 47));
      tc::tc_fence_after();
      const int cnt = limit - j * 128 - half * 64;             // visible keys of this half block: [0, cnt)
      const bool full = __all_sync(0xffffffffu, cnt >= 64);
      // 32 logits at a time: 64 beside their P do not fit into the 96 registers that 18 warps leave a thread
      auto load_logits = [&](int c, uint32_t (&sv)[32]) {
        tc::tmem_ld32(s_addr + half * 64 + c * 32, sv);
        tc::tmem_wait_ld();
        if (!full) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= cnt) sv[i] = 0xff800000u;        // a select: what lies beyond may hold anything
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
      // no scale yet: its maximum alone (with exponentials
      // formed in vain 200 tokens with 8 heads took 12.1 us, now 11.3).
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
        if (pair_any(pair_bar, alpha != 1.f)) {                // (also: x is free for the next exchange)
          // the previous P V of this tile must be complete before O is rescaled
          if (alive) alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(PV_DONE0 + t), (j - 1) & 1, status, 48));
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
      for (int c = 0; c < 2; ++c) tc::tmem_st16(s_addr + half * 64 + c * 16, pk[c]);
      l_run += row_sum;
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(P_FULL0 + t));
    }

    // ---- epilogue ---------------------------------------------------------------------------
    bool have_o = n_mine > 0 && alive;
    if (have_o) {
      have_o = __all_sync(0xffffffffu, tc::mbar_wait(bar(PV_DONE0 + t), (n_mine - 1) & 1, status, 49));
      tc::tc_fence_after();
    }
    *x_mine = l_run;
    bar_sync(pair_bar, 64);
    l_run += *x_other;
    const bool row_ok = row < lq;
    const float inv = (l_run == 0.f || !have_o) ? 0.f : 1.f / l_run;
    __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.o) + (int64_t)(q0 + row) * p.o_stride_t + head * p.o_stride_h + half * 64;
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
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            w[i] = pack_bf16x2(__uint_as_float(ov[q8 * 16 + 2 * i]) * inv, __uint_as_float(ov[q8 * 16 + 2 * i + 1]) * inv);
          st_global_32B(orow + c * 32 + q8 * 16, w);
        }
      }
    }
    if (row_ok && half == 0)
      p.lse[(int64_t)(q0 + row) * p.lse_stride_t + head * p.lse_stride_h] = inv == 0.f ? neg_inf() : (log2f(l_run) + m_used) * kLn2;
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
  if (cudaError_t e = allow_smem<dense_fwd_tc_kernel<D_QK>>(L::SMEM_BYTES); e != cudaSuccess) return e;
  // Order of the CTAs.  Tiles outermost (all heads of all sequences start with their longest tile, the shortest ones fill the
  // last wave) pays with a causal mask while the keys and values of all heads stay in L2 together: device time of tiles
  // innermost over outermost 1.02 to 1.64 up to 64 MB of them (24 MB, 3 sequences of 2048, 8 heads: 64 against 39 us), 0.93 to
  // 1.19 from there to 200 MB, 0.80 to 1.05 beyond.  Otherwise the tiles of one head run side by side and read its keys from
  // L2; without a mask all tiles are alike, and innermost over outermost is 0.75 to 1.06.
  p.tiles_outer = p.is_causal && (int64_t)p.total_k * p.h_k * (p.d_qk + p.d_v) * 2 <= (64 << 20);
  const int64_t ctas = (int64_t)((p.max_seqlen_q + 255) / 256) * p.h_q * p.batch;
  if (ctas > INT32_MAX) return cudaErrorInvalidConfiguration;
  dense_fwd_tc_kernel<D_QK><<<static_cast<unsigned>(ctas), dft::kThreads, L::SMEM_BYTES, stream>>>(p, tq, tk, tv);
  return cudaGetLastError();
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
