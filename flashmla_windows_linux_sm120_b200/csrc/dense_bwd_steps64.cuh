// The dQ and dK / dV kernels of the dense backward with steps of 64 streamed rows, for short sequences: see dense_bwd_tc.cu, which includes
// this file, for the mathematics, the roles of the warps and the rule between the two.  Results are bit for bit those of steps of 128,
// which are worth more where there are many; with few, what counts is how many rows the last one works for in vain, and how long
// the chain of one step is (64 sequences of 64 tokens, 32 heads, 128/128: 163 us, with steps of 128 rows 189).
#pragma once

namespace fmla {

namespace dbt64 {
constexpr int kResChunk = 128 * 128;              // resident tiles: [128 rows x 64 bf16] chunks
constexpr int kStgChunk = 64 * 128;               // streamed tiles: [64 rows x 64 bf16] chunks
using dbt::kDkvThreads;
using dbt::kDqThreads;
using dbt::kEwWarps;
constexpr int kStages = 3;                        // ring of streamed tiles (the TMEM buffers alternate independently)
template <int D_QK>
struct Layout {
  static constexpr int NCH = D_QK / 64;
  static constexpr int kResA = NCH * kResChunk;   // resident [128 x D_QK]   (Q or K)
  static constexpr int kResB = 2 * kResChunk;     // resident [128 x 128]    (dO or V)
  static constexpr int kStgA = NCH * kStgChunk;   // streamed [64 x D_QK]    (K or Q)
  static constexpr int kStgB = 2 * kStgChunk;     // streamed [64 x 128]     (V or dO)
  static constexpr int kStage = kStgA + kStgB;
  static constexpr int RES_OFF = 0;
  static constexpr int STG_OFF = kResA + kResB;
  static constexpr int BAR_OFF = STG_OFF + kStages * kStage;
  static constexpr int VEC_OFF = BAR_OFF + 128;   // float [2][2][64]: per-query lse*log2(e) and delta (dK/dV kernel)
  static constexpr int MISC_OFF = VEC_OFF + 1024;
  static constexpr int SMEM_BYTES = MISC_OFF + 16;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared memory limit per CTA");
};
}  // namespace dbt64

// Zeroes rows [rows_valid, 64) of a streamed tile of NCHUNK 64-column chunks (the element-wise threads, before they hand over the P
// or dS that meets these rows).  Rows past
// the end of a sequence hold the next sequence's data or the TMA zero fill; they meet exact zeros of
// P / dS in the second GEMMs, and 0 * (Inf or NaN) must not reach the accumulators.  What the first GEMMs make of them is masked.
__device__ __forceinline__ void zero_stage_tail(unsigned char* tile, int nchunk, int rows_valid, int tid) {
  const int nrows = 64 - rows_valid;
  for (int i = tid; i < nrows * nchunk * 8; i += dbt64::kEwWarps * 32) {
    const int row = rows_valid + i / (nchunk * 8), c16 = i % (nchunk * 8);
    *reinterpret_cast<uint4*>(tile + (c16 >> 3) * dbt64::kStgChunk + row * 128 + (c16 & 7) * 16) = make_uint4(0, 0, 0, 0);
  }
  tc::fence_proxy_async_smem();
}

// The instructions of a step exist once: ring stage and buffer come in as run-time bases (warp-uniform), to which the
// unrolled code adds immediates.  With one unrolled copy per (stage, buffer) each copy came around once in three to six
// steps and its first MMA waited for the instruction fetch.
// D[128 x 64] (TMEM column d_col) = A[128 x 64*NCH] (resident, K-major) * B[64 x 64*NCH]^T (streamed, K-major)
template <int NCH>
__device__ __forceinline__ void mma_res_stg64(uint32_t d_tmem, uint64_t desc_a, uint64_t desc_b, uint32_t idesc) {
#pragma unroll
  for (int c = 0; c < NCH; ++c)
#pragma unroll
    for (int s = 0; s < 4; ++s)
      tc::mma_ss(d_tmem, tc::desc_advance(desc_a, c * dbt64::kResChunk + s * 32), tc::desc_advance(desc_b, c * dbt64::kStgChunk + s * 32), idesc,
                 (c | s) ? 1u : 0u);
}
// D[128 x N] += A[128 x 64] (bf16 in TMEM, 8 columns per 16-row step) * B[64 x N] (streamed tile read MN-major)
__device__ __forceinline__ void mma_tmem_stg64(uint32_t d_tmem, uint32_t a_tmem, uint64_t desc_b, uint32_t idesc, bool first) {
#pragma unroll
  for (int s = 0; s < 4; ++s) tc::mma_ts(d_tmem, a_tmem + s * 8, tc::desc_advance(desc_b, s * 2048), idesc, (first && s == 0) ? 0u : 1u);
}

// ---- dQ -----------------------------------------------------------------------------------------------
// grid (ceil(max_seqlen_q/128), h_q, batch), 352 threads (warps 0-7 element-wise, 8 TMA, 9 and 10 MMA).
// Resident: Q, dO tiles of 128 queries.
// Per step (64 keys): S = Q K^T and dP = dO V^T into one of two TMEM buffer pairs, dS (bf16) into one of two
// slots, then dQ += dS K.  TMEM: dQ = [0, D_QK), buffer b: S = [192 + 128 b, +64), dP = [256 + 128 b, +64),
// dS slot b = [448 + 32 b, +32).
namespace dbt64 {
enum BarQ { Q_RES_FULL = 0, Q_KV_FULL0, Q_KV_EMPTY0 = Q_KV_FULL0 + kStages, Q_SD_FULL0 = Q_KV_EMPTY0 + kStages, Q_SD_FULL1, Q_DS_FULL0, Q_DS_FULL1, Q_BUF_FREE0, Q_BUF_FREE1, Q_DONE, Q_NUM_BARS };
}

template <int D_QK>
__global__ void __launch_bounds__(dbt64::kDqThreads, 1)
dense_bwd_dq_tc64_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_q,
                       const __grid_constant__ CUtensorMap tmap_do, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v) {
  using namespace dbt64;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + L::RES_OFF, sDO = sQ + L::kResA, sStg = sbase + L::STG_OFF;
  auto bar = [&](int i) { return sbase + L::BAR_OFF + i * 8; };
  volatile uint32_t* sTmem = reinterpret_cast<volatile uint32_t*>(smem + L::MISC_OFF);
  int* status = &g_dense_bwd_tc_status;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.z, head = blockIdx.y;
  const int q0 = __ldg(p.cu_q + b), lq = __ldg(p.cu_q + b + 1) - q0;
  const int k0 = __ldg(p.cu_k + b), lk = __ldg(p.cu_k + b + 1) - k0;
  const int m_base = (gridDim.x - 1 - blockIdx.x) * 128;    // the tiles with the most keys first
  // The dQ kernel may start while the dK / dV kernel in front of it drains.  One CTA waits for that kernel's end, so that
  // this kernel ends after it and what follows in the stream sees both.
  const bool waits = blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0;
  if (m_base >= lq) {
    if (waits) pdl_wait();
    return;
  }
  if ((sbase & 1023u) != 0) {
    if (tid == 0) tc::report_status(status, 30);
    if (waits) pdl_wait();
    return;
  }
  int nblk = (lk + 63) >> 6;
  if (p.is_causal) {
    const int last_key = min(m_base + 127, lq - 1) + (lk - lq);   // inclusive
    nblk = last_key < 0 ? 0 : min(nblk, (last_key >> 6) + 1);
  }

  auto load_keys = [&](int j) {
    const int st = j % kStages, tok = k0 + j * 64;
    const uint32_t stage = sStg + st * L::kStage;
    tc::mbar_arrive_expect_tx(bar(Q_KV_FULL0 + st), L::kStage);
#pragma unroll
    for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(stage + c * kStgChunk, &tmap_k, c * 64, head, tok, bar(Q_KV_FULL0 + st));
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tma_load_3d(stage + L::kStgA + c * kStgChunk, &tmap_v, c * 64, head, tok, bar(Q_KV_FULL0 + st));
  };
  if (warp == kEwWarps) {
    // the thread that makes the barriers starts the first loads at once, before the others have tensor memory
    if (tc::elect_one()) {
      // one arrival per element-wise warp
      for (int i = 0; i < Q_NUM_BARS; ++i) tc::mbar_init(bar(i), (i == Q_DS_FULL0 || i == Q_DS_FULL1) ? kEwWarps : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      if (nblk > 0) {
        tc::mbar_arrive_expect_tx(bar(Q_RES_FULL), L::kResA + L::kResB);
#pragma unroll
        for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(sQ + c * kResChunk, &tmap_q, c * 64, head, q0 + m_base, bar(Q_RES_FULL));
#pragma unroll
        for (int c = 0; c < 2; ++c) tc::tma_load_3d(sDO + c * kResChunk, &tmap_do, c * 64, head, q0 + m_base, bar(Q_RES_FULL));
        for (int j = 0; j < min(kStages, nblk); ++j) load_keys(j);
      }
    }
    __syncwarp();
  }
  if (warp == kEwWarps + 1) tc::tmem_alloc(sbase + L::MISC_OFF, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *sTmem;
  constexpr int TM_DQ = 0, TM_SD = 192, TM_DS = 448;

  if (warp == kEwWarps) {
    // ================================ TMA producer =====================================
    if (tc::elect_one()) {
      bool alive = true;
      for (int j = kStages; j < nblk && alive; ++j) {
        alive = tc::mbar_wait(bar(Q_KV_EMPTY0 + j % kStages), ((j / kStages) & 1) ^ 1, status, 51);
        if (alive) load_keys(j);
      }
    }
  } else if (warp > kEwWarps) {
    // ================================ MMA issuers =======================================
    constexpr uint32_t idesc_sd = tc::idesc_bf16_f32(128, 64, 0, 0);
    constexpr uint32_t idesc_dq = tc::idesc_bf16_f32(128, D_QK, 0, 1);
    const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);
    const uint64_t desc_do = tc::smem_desc_sw128(sDO, 16, 1024);
    const uint64_t desc_k = tc::smem_desc_sw128(sStg, 16, 1024);                      // K tile of stage 0, K-major (B of S)
    const uint64_t desc_v = tc::smem_desc_sw128(sStg + L::kStgA, 16, 1024);           // V tile of stage 0, K-major (B of dP)
    const uint64_t desc_kt = tc::smem_desc_sw128(sStg, kStgChunk, 1024);              // K tile of stage 0, MN-major (B of dQ)
    bool alive = nblk > 0;
    // Two issuing threads: the first for the first GEMMs of a step (S, dP), the other for the second one (dQ); the waits of one
    // overlap the instructions of the other.
    if (tc::elect_one()) {
      if (warp == kEwWarps + 1) {
        if (alive) alive = tc::mbar_wait(bar(Q_RES_FULL), 0, status, 52);
        for (int j = 0; j < nblk && alive; ++j) {
          const int st = j % kStages, bf = j & 1;
          // the tile has landed, and the S / dP buffer pair bf is free (the element-wise warps have read step
          // j-2 out of it)
          alive = tc::mbar_wait(bar(Q_KV_FULL0 + st), (j / kStages) & 1, status, 54);
          if (alive) alive = tc::mbar_wait(bar(Q_DS_FULL0 + bf), ((j >> 1) & 1) ^ 1, status, 54);
          if (!alive) break;
          tc::tc_fence_after();
          const uint32_t off = st * L::kStage, col = tmem + TM_SD + bf * 128;
          mma_res_stg64<L::NCH>(col, desc_q, tc::desc_advance(desc_k, off), idesc_sd);
          mma_res_stg64<2>(col + 64, desc_do, tc::desc_advance(desc_v, off), idesc_sd);
          tc::tc_commit(bar(Q_SD_FULL0 + bf));
        }
      } else {
        for (int j = 0; j < nblk && alive; ++j) {
          const int st = j % kStages, bf = j & 1;
          alive = tc::mbar_wait(bar(Q_DS_FULL0 + bf), (j >> 1) & 1, status, 53);
          if (!alive) break;
          tc::tc_fence_after();
          mma_tmem_stg64(tmem + TM_DQ, tmem + TM_DS + bf * 32, tc::desc_advance(desc_kt, st * L::kStage), idesc_dq, j == 0);
          tc::tc_commit(bar(Q_KV_EMPTY0 + st));
          tc::tc_commit(bar(Q_BUF_FREE0 + bf));
          if (j == nblk - 1) tc::tc_commit(bar(Q_DONE));
        }
      }
    }
  } else {
    // ================================ element-wise / epilogue ==========================
    // Warps w and w + 4 share the TMEM lanes of 32 rows: warp w takes columns [0, 32) of every 64-key block, warp w + 4
    // the other half.  With four warps (one per scheduler) the chain TMEM load -> exponentials -> dS -> store of a step
    // outlasted the step's 1344 clk of MMAs, and the tensor pipe waited for it.
    const int half = warp >> 2, rl = tid & 127;
    const int row = m_base + rl;
    const bool row_ok = row < lq;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float lse2 = row_ok ? __ldg(p.lse + (int64_t)(q0 + row) * p.lse_stride_t + head * p.lse_stride_h) * kLog2e : 0.f;
    const float dl = row_ok ? __ldg(p.delta + (int64_t)head * p.total_q + q0 + row) : 0.f;
    const int limit = !row_ok ? 0 : (p.is_causal ? max(0, min(lk, row + (lk - lq) + 1)) : lk);
    bool alive = true;
    for (int j = 0; j < nblk && alive; ++j) {
      const int st = j & 1;
      const uint32_t sd_addr = tmem + lane_addr + TM_SD + st * 128 + half * 32;
      // S and dP of this step are there, and the dS slot st is free (it was last read by the dQ
      // instructions of step j-2; dS has slots of its own so that the fp32 buffers are free again as
      // soon as they have been read)
      alive = tc::mbar_wait2(bar(Q_SD_FULL0 + st), (j >> 1) & 1, bar(Q_BUF_FREE0 + st), ((j >> 1) & 1) ^ 1, status, 55);
      if (!alive) break;
      tc::tc_fence_after();
      uint32_t sv[32], dp[32], pk[16];
      tc::tmem_ld32(sd_addr, sv);
      tc::tmem_ld32(sd_addr + 64, dp);
      tc::tmem_wait_ld();
      const int cnt = limit - j * 64 - half * 32;              // visible keys of this half block: [0, cnt)
      const bool all_visible = __all_sync(0xffffffffu, cnt >= 32);
      row_exp2(sv, p.scale_log2, [&](int) { return f2(-lse2); });
      // two loops, not a test per element: the compiler makes a branch of each test (40 clk per element measured)
      auto to_ds = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const F2 d = f2_mul(F2{__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])},
                              f2_add(F2{__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1])}, f2(-dl)));
          float d0 = d.lo, d1 = d.hi;
          if constexpr (decltype(masked)::value) {             // a select, not a product: masked entries may hold Inf or NaN
            d0 = 2 * i < cnt ? d0 : 0.f;
            d1 = 2 * i + 1 < cnt ? d1 : 0.f;
          }
          pk[i] = pack_bf16x2(d0, d1);
        }
      };
      if (all_visible) to_ds(std::false_type{});
      else to_ds(std::true_type{});
      // K rows past the end of the sequence must be exact zeros for dQ += dS K
      if (lk - j * 64 < 64) zero_stage_tail(smem + L::STG_OFF + j % kStages * L::kStage, L::NCH, lk - j * 64, tid);
      tc::tmem_st16(tmem + lane_addr + TM_DS + st * 32 + half * 16, pk);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(Q_DS_FULL0 + st));
    }
    bool have = nblk > 0 && alive;
    if (have) {
      have = __all_sync(0xffffffffu, tc::mbar_wait(bar(Q_DONE), 0, status, 56));
      tc::tc_fence_after();
    }
    __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.dq) + (int64_t)(q0 + row) * p.dq_stride_t + head * p.dq_stride_h;
#pragma unroll 1
    for (int c = half; c < D_QK / 32; c += 2) store_grad_chunk(tmem + lane_addr + TM_DQ + c * 32, have, row_ok, p.scale, orow + c * 32);
  }

  tc::tc_fence_before();
  __syncthreads();
  if (warp == kEwWarps + 1) tc::tmem_dealloc(tmem, 512);
  if (waits) pdl_wait();
}

// ---- dK, dV -------------------------------------------------------------------------------------
// grid (ceil(max_seqlen_k/128), h, batch), 320 threads (warps 0-7 element-wise, 8 TMA, 9 MMA).  Resident: K, V tiles
// of 128 keys.  Per step (64 queries): S^T = K Q^T, dP^T = V dO^T, P^T and dS^T (bf16), dV += P^T dO, dK += dS^T Q.
// TMEM: dV = [0,128), dK = [128, 128 + D_QK), S^T = [320,384), dP^T = [384,448), P^T = [448,480), dS^T = [480,512).
// The 192 columns that dV and dK leave hold the fp32 tiles of ONE step and the bf16 tiles of ONE step: the element-wise
// warps take S^T and dP^T of step j into registers, which frees those columns for step j+1, and write P^T and dS^T of
// step j into columns of their own.  The tensor pipe runs S^T(j+1), dP^T(j+1), dV(j), dK(j) back to back while the
// element-wise work of a step hides behind the 1600 clk of MMAs of its neighbours.  (With the bf16 tiles written over
// the fp32 ones, two S^T buffers and a single dP^T buffer, dP^T(j+1) had to wait for dK(j) and dK(j) for the
// element-wise work on dP^T(j).)
namespace dbt64 {
enum BarK { K_RES_FULL = 0, K_QD_FULL0, K_QD_EMPTY0 = K_QD_FULL0 + kStages, K_S_FULL = K_QD_EMPTY0 + kStages, K_DP_FULL, K_P_FREE, K_DS_FREE,
            K_S_READ, K_DP_READ, K_P_FULL, K_DS_FULL, K_NUM_BARS };   // K_S_READ and later: one arrival per element-wise warp
}

template <int D_QK>
__global__ void __launch_bounds__(dbt64::kDkvThreads, 1)
dense_bwd_dkdv_tc64_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_k,
                         const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_q,
                         const __grid_constant__ CUtensorMap tmap_do) {
  using namespace dbt64;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sK = sbase + L::RES_OFF, sV = sK + L::kResA, sStg = sbase + L::STG_OFF;
  auto bar = [&](int i) { return sbase + L::BAR_OFF + i * 8; };
  float* sVec = reinterpret_cast<float*>(smem + L::VEC_OFF);
  volatile uint32_t* sTmem = reinterpret_cast<volatile uint32_t*>(smem + L::MISC_OFF);
  volatile int* sAbort = reinterpret_cast<volatile int*>(smem + L::MISC_OFF + 8);   // set by an element-wise thread whose wait expired
  int* status = &g_dense_bwd_tc_status;

  pdl_allow_dependents();      // the dQ kernel needs nothing of this one: its CTAs fill the SMs that run out of key tiles
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.z, head = blockIdx.y;
  const int q0 = __ldg(p.cu_q + b), lq = __ldg(p.cu_q + b + 1) - q0;
  const int k0 = __ldg(p.cu_k + b), lk = __ldg(p.cu_k + b + 1) - k0;
  const int n_base = blockIdx.x * 128;                       // with a causal mask the first key tiles see the most queries
  if (n_base >= lk) return;
  if ((sbase & 1023u) != 0) {
    if (tid == 0) tc::report_status(status, 30);
    return;
  }
  // query blocks [jb_lo, jb_hi) of 64 rows that see at least one key of this tile
  const int jb_hi = (lq + 63) >> 6;
  const int jb_lo = p.is_causal ? min(jb_hi, max(0, n_base - (lk - lq)) >> 6) : 0;
  const int nstep = jb_hi - jb_lo;

  auto load_queries = [&](int j) {
    const int st = j % kStages, tok = q0 + (jb_lo + j) * 64;
    const uint32_t stage = sStg + st * L::kStage;
    tc::mbar_arrive_expect_tx(bar(K_QD_FULL0 + st), L::kStage);
#pragma unroll
    for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(stage + c * kStgChunk, &tmap_q, c * 64, head, tok, bar(K_QD_FULL0 + st));
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tma_load_3d(stage + L::kStgA + c * kStgChunk, &tmap_do, c * 64, head, tok, bar(K_QD_FULL0 + st));
  };
  if (warp == kEwWarps) {
    // as in the dQ kernel: barriers and first loads before the others have tensor memory
    if (tc::elect_one()) {
      for (int i = 0; i < K_NUM_BARS; ++i) tc::mbar_init(bar(i), i >= K_S_READ ? kEwWarps : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      *sAbort = 0;
      if (nstep > 0) {
        tc::mbar_arrive_expect_tx(bar(K_RES_FULL), L::kResA + L::kResB);
#pragma unroll
        for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(sK + c * kResChunk, &tmap_k, c * 64, head, k0 + n_base, bar(K_RES_FULL));
#pragma unroll
        for (int c = 0; c < 2; ++c) tc::tma_load_3d(sV + c * kResChunk, &tmap_v, c * 64, head, k0 + n_base, bar(K_RES_FULL));
        for (int j = 0; j < min(kStages, nstep); ++j) load_queries(j);
      }
    }
    __syncwarp();
  }
  if (warp == kEwWarps + 1) tc::tmem_alloc(sbase + L::MISC_OFF, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *sTmem;
  constexpr int TM_DV = 0, TM_DK = 128, TM_ST = 320, TM_DPT = 384, TM_P = 448, TM_DS = 480;

  if (warp == kEwWarps) {
    // ================================ TMA producer =====================================
    if (tc::elect_one()) {
      bool alive = true;
      for (int j = kStages; j < nstep && alive; ++j) {
        alive = tc::mbar_wait(bar(K_QD_EMPTY0 + j % kStages), ((j / kStages) & 1) ^ 1, status, 61);
        if (alive) load_queries(j);
      }
    }
  } else if (warp == kEwWarps + 1) {
    // ================================ MMA issuer =======================================
    constexpr uint32_t idesc_sd = tc::idesc_bf16_f32(128, 64, 0, 0);
    constexpr uint32_t idesc_dv = tc::idesc_bf16_f32(128, 128, 0, 1);
    constexpr uint32_t idesc_dk = tc::idesc_bf16_f32(128, D_QK, 0, 1);
    const uint64_t desc_k = tc::smem_desc_sw128(sK, 16, 1024);
    const uint64_t desc_v = tc::smem_desc_sw128(sV, 16, 1024);
    const uint64_t desc_q = tc::smem_desc_sw128(sStg, 16, 1024);                      // Q tile of stage 0, K-major (B of S^T)
    const uint64_t desc_do = tc::smem_desc_sw128(sStg + L::kStgA, 16, 1024);          // dO tile of stage 0, K-major (B of dP^T)
    const uint64_t desc_qt = tc::smem_desc_sw128(sStg, kStgChunk, 1024);              // Q tile, MN-major (B of dK)
    const uint64_t desc_dot = tc::smem_desc_sw128(sStg + L::kStgA, kStgChunk, 1024);  // dO tile, MN-major (B of dV)
    if (tc::elect_one() && nstep > 0) {
      bool alive = tc::mbar_wait(bar(K_RES_FULL), 0, status, 62);
      auto wait = [&](int i, int ph, int code) {
        if (alive) alive = tc::mbar_wait(bar(i), ph, status, code);
        return alive;
      };
      // step j = -1 issues the first GEMMs of step 0 (the instructions of a step exist once)
      for (int j = -1; j < nstep && alive; ++j) {
        if (j + 1 < nstep) {                           // S^T and dP^T of the next step, once those of this one have been read
          const int st = (j + 1) % kStages;
          if (!wait(K_QD_FULL0 + st, ((j + 1) / kStages) & 1, 63)) break;
          if (!wait(K_S_READ, j & 1, 64)) break;
          tc::tc_fence_after();
          mma_res_stg64<L::NCH>(tmem + TM_ST, desc_k, tc::desc_advance(desc_q, st * L::kStage), idesc_sd);
          tc::tc_commit(bar(K_S_FULL));
          if (!wait(K_DP_READ, j & 1, 67)) break;
          tc::tc_fence_after();
          mma_res_stg64<2>(tmem + TM_DPT, desc_v, tc::desc_advance(desc_do, st * L::kStage), idesc_sd);
          tc::tc_commit(bar(K_DP_FULL));
        }
        if (j >= 0) {
          const int st = j % kStages;
          if (!wait(K_P_FULL, j & 1, 68)) break;
          tc::tc_fence_after();
          mma_tmem_stg64(tmem + TM_DV, tmem + TM_P, tc::desc_advance(desc_dot, st * L::kStage), idesc_dv, j == 0);
          tc::tc_commit(bar(K_P_FREE));
          if (!wait(K_DS_FULL, j & 1, 69)) break;
          tc::tc_fence_after();
          mma_tmem_stg64(tmem + TM_DK, tmem + TM_DS, tc::desc_advance(desc_qt, st * L::kStage), idesc_dk, j == 0);
          tc::tc_commit(bar(K_DS_FREE));               // completes after dV of this step: the tensor pipe runs in order
          tc::tc_commit(bar(K_QD_EMPTY0 + st));
        }
      }
    }
  } else {
    // ================================ element-wise / epilogue ==========================
    // warps w and w + 4 share the TMEM lanes of 32 keys: warp w takes queries [0, 32) of every block, warp w + 4 the rest
    const int half = warp >> 2, rl = tid & 127;
    const int key = n_base + rl;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int shift = lk - lq;                                 // query i sees keys <= i + shift
    // per-query vectors of a step: -lse * log2(e) (threads 0-63) and -delta (threads 64-127); each value is loaded one
    // step ahead and not touched before the next, so that no step waits for global memory
    const float* vec = tid < 64 ? p.lse + (int64_t)q0 * p.lse_stride_t + head * p.lse_stride_h : p.delta + (int64_t)head * p.total_q + q0;
    const int64_t vec_stride = tid < 64 ? p.lse_stride_t : 1;
    const float vec_mul = tid < 64 ? -kLog2e : -1.f;
    auto load_vec = [&](int j) {
      const int i = (jb_lo + j) * 64 + (tid & 63);
      return tid < 128 && i < lq ? __ldg(vec + i * vec_stride) : 0.f;
    };
    float v_next = nstep > 0 ? load_vec(0) : 0.f;
    bool alive = true;
    for (int j = 0; j < nstep && alive; ++j) {
      const int jb = jb_lo + j, vb = j & 1;
      if (tid < 128) sVec[vb * 128 + tid] = v_next * vec_mul;
      if (j + 1 < nstep) v_next = load_vec(j + 1);
      if (!tc::mbar_wait(bar(K_S_FULL), j & 1, status, 65)) *sAbort = 1;
      bar_sync(1, kEwWarps * 32);                              // vectors visible; also keeps the two buffers of sVec apart
      if (*sAbort) { alive = false; break; }                   // read right after the barrier: the same for all threads
      tc::tc_fence_after();
      uint32_t sv[32], dp[32], pk[16];
      tc::tmem_ld32(tmem + lane_addr + TM_ST + half * 32, sv);
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_S_READ));
      const int c_max = lq - jb * 64 - half * 32;              // columns (queries) [c_min, c_max) see this key
      const int c_min = p.is_causal ? key - shift - jb * 64 - half * 32 : 0;
      const bool all_visible = __all_sync(0xffffffffu, c_min <= 0 && c_max >= 32);
      const float4* vl = reinterpret_cast<const float4*>(sVec + vb * 128 + half * 32);
      const float4* vd = reinterpret_cast<const float4*>(sVec + vb * 128 + 64 + half * 32);
      row_exp2(sv, p.scale_log2, [&](int i) {
        const float4 l4 = vl[i >> 1];
        return i & 1 ? F2{l4.z, l4.w} : F2{l4.x, l4.y};
      });
      auto to_p = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if constexpr (decltype(masked)::value) {             // a select: see the dQ kernel
            if (!(2 * i >= c_min && 2 * i < c_max)) sv[2 * i] = 0u;
            if (!(2 * i + 1 >= c_min && 2 * i + 1 < c_max)) sv[2 * i + 1] = 0u;
          }
          pk[i] = pack_bf16x2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1]));
        }
      };
      if (all_visible) to_p(std::false_type{});
      else to_p(std::true_type{});
      // a wait that gives up here lets the step run on; the flag ends the loop at the next barrier
      if (!tc::mbar_wait(bar(K_P_FREE), (j & 1) ^ 1, status, 70)) *sAbort = 1;       // dV of step j-1 has read P^T
      // the last step: rows past the end of the sequence must be exact zeros for dV and dK
      if (lq - jb * 64 < 64) zero_stage_tail(smem + L::STG_OFF + j % kStages * L::kStage, L::NCH + 2, lq - jb * 64, tid);
      tc::tc_fence_after();
      __syncwarp();
      tc::tmem_st16(tmem + lane_addr + TM_P + half * 16, pk);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_P_FULL));
      if (!tc::mbar_wait(bar(K_DP_FULL), j & 1, status, 71)) *sAbort = 1;
      tc::tc_fence_after();
      __syncwarp();
      tc::tmem_ld32(tmem + lane_addr + TM_DPT + half * 32, dp);
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_DP_READ));
      auto to_ds = [&](auto masked) {
#pragma unroll
        for (int i4 = 0; i4 < 8; ++i4) {
          const float4 d4 = vd[i4];
          const F2 minus_d[2] = {{d4.x, d4.y}, {d4.z, d4.w}};
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int col = i4 * 4 + e * 2;
            F2 dv = f2_mul(F2{__uint_as_float(sv[col]), __uint_as_float(sv[col + 1])},
                           f2_add(F2{__uint_as_float(dp[col]), __uint_as_float(dp[col + 1])}, minus_d[e]));
            if constexpr (decltype(masked)::value) {
              dv.lo = col >= c_min && col < c_max ? dv.lo : 0.f;
              dv.hi = col + 1 >= c_min && col + 1 < c_max ? dv.hi : 0.f;
            }
            pk[i4 * 2 + e] = pack_bf16x2(dv.lo, dv.hi);
          }
        }
      };
      if (all_visible) to_ds(std::false_type{});
      else to_ds(std::true_type{});
      if (!tc::mbar_wait(bar(K_DS_FREE), (j & 1) ^ 1, status, 72)) *sAbort = 1;      // dK of step j-1 has read dS^T
      tc::tc_fence_after();
      __syncwarp();
      tc::tmem_st16(tmem + lane_addr + TM_DS + half * 16, pk);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_DS_FULL));
    }
    bool have = nstep > 0 && alive;
    if (have) {
      have = __all_sync(0xffffffffu, tc::mbar_wait(bar(K_DS_FREE), (nstep - 1) & 1, status, 66));   // the last dK, hence all of them
      tc::tc_fence_after();
    }
    const bool row_ok = key < lk;
    __nv_bfloat16* dv_row = reinterpret_cast<__nv_bfloat16*>(p.dv) + (int64_t)(k0 + key) * p.dv_stride_t + head * p.dv_stride_h;
    __nv_bfloat16* dk_row = reinterpret_cast<__nv_bfloat16*>(p.dk) + (int64_t)(k0 + key) * p.dk_stride_t + head * p.dk_stride_h;
#pragma unroll 1
    for (int c = half; c < (128 + D_QK) / 32; c += 2)          // dV columns first, then dK
      store_grad_chunk(tmem + lane_addr + c * 32, have, row_ok, c < 4 ? 1.f : p.scale, c < 4 ? dv_row + c * 32 : dk_row + (c - 4) * 32);
  }

  tc::tc_fence_before();
  __syncthreads();
  if (warp == kEwWarps + 1) tc::tmem_dealloc(tmem, 512);
}

}  // namespace fmla
