// Dense variable-length MHA backward (bf16, head dims 192/128 and 128/128) for sm_100a on
// tcgen05 / TMA / tensor memory.
//
// Math of the reference backward (csrc/sm100/prefill/dense/device/fmha_device_bwd.hpp:290-316 and
// kernel/sm100_fmha_bwd_mla_kernel_tma_warpspecialized.hpp:1308-1324): with P = exp(S*scale - lse),
//   delta = rowsum(dO * O),  dP = dO V^T,  dS = P * (dP - delta),
//   dV = P^T dO,  dK = scale * dS^T Q,  dQ = scale * dS K,
// P and dS rounded to bf16 before the second GEMMs.  Unlike the reference, whose dQ is accumulated
// with floating-point reduce-adds in a launch-dependent order, every output here is produced by
// exactly one CTA in a fixed order, so dQ, dK and dV are bitwise reproducible.  Three kernels:
//   1. delta pre-pass                         (FmhaKernelBwdSumOdO's job)
//   2. dQ:    one CTA per (128-query tile, head, sequence), walks the keys in blocks of 128, or of 64 (dense_bwd_steps64.cuh)
//   3. dK/dV: one CTA per (128-key tile, head, sequence), walks the queries in blocks of 128, or of 64
// Requires h_q == h_k (as flash_mla/flash_mla_interface.py:413-415).
//
// Both main kernels: warps 0-7 element-wise (two threads per row of the resident tile = TMEM lane, one per half of the
// streamed columns), then a TMA warp and the MMA issuing warps.  The two first GEMMs of a step write
// fp32 tiles [128 x 128] into tensor memory; the element-wise warps turn them into bf16 P / dS in columns
// of their own; the second GEMMs read those as their A operand straight from tensor memory and the
// streamed tile, read MN-major, as B.
// What bounds them: the tensor pipe and the shared memory it reads.  With both operands in shared memory an m128nNk16 product
// reads 4 KB of A and N * 32 bytes of B at 128 bytes per clock: 48 clk where 32 are needed for N = 64, 64 where 64 are needed for
// N = 128.  Hence steps of 128 streamed rows, which also halve the waits, barriers and TMEM round trips per row.  Against
// steps of 64 (8 sequences of 1 k to 8 k tokens, 128 heads, 192/128, causal, under the power cap at 1.65 to 1.7 GHz): dK/dV and
// dQ together 32.6 -> 29.5 ms, forward and backward 41.9 -> 39.3 ms.
// The GEMMs are issued by single threads (waits, votes and branches of whole warps left the tensor pipe idle), the element-wise
// warps clear what lies past the end of a sequence, and the second GEMM on the wide tile goes chunk by chunk of its columns, each
// followed by the load of that chunk for the step after next: with one release for the whole tile the next loads came 500 clk late at
// 192/128.  A step of dK/dV took 4 130 clk at 192/128 and 3 810 at 128/128 and takes 3 220 and 2 935, one of dQ 3 240 and 2 900, now 2 715 and 2 420
// (two sequences of 4 096, 32 heads, no mask, one time stamp per step); the element-wise warps (with trace points 1 300 clk for P, 650 for dS)
// now set the pace of dK/dV.  Sixteen of them, with half the columns each, were no faster.  4 x 1 000 tokens, 8 heads, 192/128, causal (steps of 64) 72.0 ->
// 64.2 us, 6 x 1 000, 8 heads, 128/128, no mask 121.8 -> 109.4, 2 x 4 096, 32 heads, no mask 1 916 -> 1 863.
// Every mbarrier wait is bounded (tc_common.cuh); a pipeline fault sets a status word and lets the
// CTA drain and free its tensor memory.
#include "kernels.h"
#include "launch.cuh"
#include "tc_common.cuh"
#include "tma_host.cuh"

#include <type_traits>

namespace fmla {

namespace dbt {
constexpr int kChunk = 128 * 128;                 // every tile: [128 rows x 64 bf16] chunks, 128-byte swizzled rows
constexpr int kMaxChunks = 3;
constexpr int kEwWarps = 8;                       // element-wise warps (two per 32 accumulator rows)
constexpr int kDqThreads = (kEwWarps + 3) * 32;   // + TMA + two MMA issuers
constexpr int kDkvThreads = (kEwWarps + 2) * 32;  // + TMA + MMA issuer
// Streamed tiles: the wide one (K or Q) is needed from the first GEMM of a step to its last and has two stages, the narrow one
// (V or dO) is needed for a shorter stretch and has what is left of shared memory.
template <int D_QK>
struct Layout {
  static constexpr int NCH = D_QK / 64;
  static constexpr int kWide = NCH * kChunk;      // [128 x D_QK]
  static constexpr int kNarrow = 2 * kChunk;      // [128 x 128]
  static constexpr int kWideStages = 2;
  static constexpr int kNarrowStages = D_QK == 192 ? 1 : 2;
  static constexpr int RES_OFF = 0;               // resident Q and dO, or K and V
  static constexpr int WIDE_OFF = kWide + kNarrow;
  static constexpr int NARROW_OFF = WIDE_OFF + kWideStages * kWide;
  static constexpr int BAR_OFF = NARROW_OFF + kNarrowStages * kNarrow;
  static constexpr int VEC_OFF = BAR_OFF + 256;   // float [2][2][128]: per-query lse*log2(e) and delta (dK/dV kernel)
  static constexpr int MISC_OFF = VEC_OFF + 2048;
  static constexpr int SMEM_BYTES = MISC_OFF + 16;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB shared memory limit per CTA");
};
}  // namespace dbt

__device__ int g_dense_bwd_tc_status = 0;

// Optional timeline of the first steps of CTA (0,0,0) of the dQ kernel, compiled in with -DFMLA_TRACE only.
#ifdef FMLA_TRACE
__device__ long long g_dense_bwd_trace[64 * 16];
#define DBT_TRACE_AT(blk, slot)                                                          \
  do {                                                                                     \
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && (blk) < 64) g_dense_bwd_trace[(blk) * 16 + (slot)] = clock64(); \
  } while (0)
#else
#define DBT_TRACE_AT(blk, slot) do {} while (0)
#endif

// ---- 1. delta[h, t] = sum_d dO * O --------------------------------------------------------------
// Bound by HBM (512 bytes read per row): 16 lanes per row with 16-byte loads, kDeltaRows rows per half warp in flight.
constexpr int kDeltaRows = 4;
__global__ void __launch_bounds__(256) dense_bwd_delta_tc_kernel(const __grid_constant__ DenseKernelParams p) {
  const int group = (blockIdx.x * 256 + threadIdx.x) >> 4, l16 = threadIdx.x & 15;
  const int64_t rows = (int64_t)p.total_q * p.h_q, first = (int64_t)group * kDeltaRows;
  uint4 ov[kDeltaRows], dv[kDeltaRows];
#pragma unroll
  for (int r = 0; r < kDeltaRows; ++r) {
    ov[r] = dv[r] = make_uint4(0, 0, 0, 0);
    if (first + r < rows) {
      const int t = static_cast<int>((first + r) / p.h_q), h = static_cast<int>((first + r) % p.h_q);
      ov[r] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.o) + (int64_t)t * p.o_stride_t + h * p.o_stride_h) + l16);
      dv[r] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.d_o) + (int64_t)t * p.do_stride_t + h * p.do_stride_h) + l16);
    }
  }
#pragma unroll
  for (int r = 0; r < kDeltaRows; ++r) {
    const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&ov[r]);
    const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&dv[r]);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = __bfloat1622float2(o2[i]), g = __bfloat1622float2(d2[i]);
      s += a.x * g.x + a.y * g.y;
    }
#pragma unroll
    for (int off = 8; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (l16 == 0 && first + r < rows) p.delta[(first + r) % p.h_q * p.total_q + (first + r) / p.h_q] = s;
  }
}

// 16-row steps that the valid rows of a streamed tile reach: what lies beyond is neither multiplied nor accumulated
__device__ __forceinline__ int k_steps(int rows_valid) { return (min(rows_valid, 128) + 15) >> 4; }

// Zeroes the rows from rows_valid to the end of its 16-row step in a streamed tile of NCHUNK 64-column chunks (the element-wise
// threads, before they hand over the P or dS that meets these rows).
// Rows past the end of a sequence hold the next sequence's data or the TMA zero fill; they meet exact zeros of
// P / dS in the second GEMMs, and 0 * (Inf or NaN) must not reach the accumulators.  What the first GEMMs make of them is masked.
__device__ __forceinline__ void zero_tail(unsigned char* tile, int nchunk, int rows_valid, int tid) {
  const int nrows = k_steps(rows_valid) * 16 - rows_valid;
  for (int i = tid; i < nrows * nchunk * 8; i += dbt::kEwWarps * 32) {
    const int row = rows_valid + i / (nchunk * 8), c16 = i % (nchunk * 8);
    *reinterpret_cast<uint4*>(tile + (c16 >> 3) * dbt::kChunk + row * 128 + (c16 & 7) * 16) = make_uint4(0, 0, 0, 0);
  }
  tc::fence_proxy_async_smem();
}

// The instructions of a step exist once: ring stage and buffer come in as run-time bases (warp-uniform), to which the
// unrolled code adds immediates.  With one unrolled copy per (stage, buffer) each copy came around once in three to six
// steps and its first MMA waited for the instruction fetch.
// D[128 x N] (TMEM column d_tmem) = A[128 x 64*NCH] (resident, K-major) * B[N x 64*NCH]^T (streamed, K-major), N in idesc;
// landed(c) waits for chunk c of B
template <int NCH, class Landed>
__device__ __forceinline__ bool mma_res_stg(uint32_t d_tmem, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, Landed landed) {
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    if (!landed(c)) return false;
#pragma unroll
    for (int s = 0; s < 4; ++s)
      tc::mma_ss(d_tmem, tc::desc_advance(desc_a, c * dbt::kChunk + s * 32), tc::desc_advance(desc_b, c * dbt::kChunk + s * 32), idesc,
                 (c | s) ? 1u : 0u);
  }
  return true;
}
// D[128 x N] += A[128 x 16*ks] (bf16 in TMEM, 8 columns per 16-row step) * B[16*ks x N] (streamed tile read MN-major)
__device__ __forceinline__ void mma_tmem_stg(uint32_t d_tmem, uint32_t a_tmem, uint64_t desc_b, uint32_t idesc, bool first, int ks) {
  if (__builtin_expect(ks == 8, 1)) {
#pragma unroll
    for (int s = 0; s < 8; ++s) tc::mma_ts(d_tmem, a_tmem + s * 8, tc::desc_advance(desc_b, s * 2048), idesc, (first && s == 0) ? 0u : 1u);
  } else {
#pragma unroll 1
    for (int s = 0; s < ks; ++s) tc::mma_ts(d_tmem, a_tmem + s * 8, tc::desc_advance(desc_b, s * 2048), idesc, (first && s == 0) ? 0u : 1u);
  }
}
// 64 fp32 columns of the calling warp's lanes
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&v)[64]) {
  tc::tmem_ld32(taddr, reinterpret_cast<uint32_t (&)[32]>(v[0]));
  tc::tmem_ld32(taddr + 32, reinterpret_cast<uint32_t (&)[32]>(v[32]));
}

// P = 2^(s * scale - lse) of 32 or 64 logits in place; minus_lse(i) is -lse of elements 2i and 2i + 1.  One pair in three on the multiply-add
// pipe: the special function unit alone takes 1 024 clk for a step, as long as the products that it has to keep up with.
template <int N, class MinusLse>
__device__ __forceinline__ void row_exp2(uint32_t (&sv)[N], float scale, MinusLse minus_lse) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    F2 x = f2_fma(F2{__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])}, f2(scale), minus_lse(i));
    if (i % 16 % 3 == 2) {      // (alike in steps of either length)
      x = f2_exp2(x);
    } else {
      x.lo = exp2f(x.lo);
      x.hi = exp2f(x.hi);
    }
    sv[2 * i] = __float_as_uint(x.lo);
    sv[2 * i + 1] = __float_as_uint(x.hi);
  }
}

// 32 fp32 columns of an accumulator row -> bf16, times `mul`, as full 32-byte sectors (zeros when nothing was computed)
__device__ __forceinline__ void store_grad_chunk(uint32_t taddr, bool have, bool row_ok, float mul, __nv_bfloat16* dst) {
  uint32_t ov[32];
  if (have) {
    tc::tmem_ld32(taddr, ov);
    tc::tmem_wait_ld();
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) ov[i] = 0u;
  }
  if (!row_ok) return;
#pragma unroll
  for (int q8 = 0; q8 < 2; ++q8) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      w[i] = pack_bf16x2(__uint_as_float(ov[q8 * 16 + 2 * i]) * mul, __uint_as_float(ov[q8 * 16 + 2 * i + 1]) * mul);
    st_global_32B(dst + q8 * 16, w);
  }
}

// ---- 2. dQ ------------------------------------------------------------------------------------------
// grid (ceil(max_seqlen_q/128), h_q, batch), 352 threads (warps 0-7 element-wise, 8 TMA, 9 and 10 MMA).
// Resident: Q, dO tiles of 128 queries.
// Per step (128 keys): S = Q K^T, dP = dO V^T, dS (bf16), dQ += dS K.
// TMEM: dQ = [0, D_QK), S = [192,320), dP = [320,448), dS = [448,512).
// The element-wise warps take S and dP into registers, which frees those columns for the next step: S(j+1) and dP(j+1) run
// beside the element-wise work of step j, dQ(j) beside that of step j+1.
namespace dbt {
// dP of a step and the release of its V, dQ of a chunk of columns and the release of that chunk of K (the last one: and of dS), are one
// event each, with two barriers in turn
enum BarQ { Q_RES_FULL = 0, Q_K_FULL0, Q_DQ_DONE0 = Q_K_FULL0 + 2 * kMaxChunks, Q_V_FULL0 = Q_DQ_DONE0 + 2 * kMaxChunks, Q_V_FULL1, Q_DP_FULL0, Q_DP_FULL1, Q_S_FULL,
            Q_S_READ, Q_DP_READ, Q_DS_FULL, Q_NUM_BARS };   // Q_S_READ and later: one arrival per element-wise warp
}

template <int D_QK>
__global__ void __launch_bounds__(dbt::kDqThreads, 1)
dense_bwd_dq_tc_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_q,
                       const __grid_constant__ CUtensorMap tmap_do, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v) {
  using namespace dbt;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase + L::RES_OFF, sDO = sQ + L::kWide, sK = sbase + L::WIDE_OFF, sV = sbase + L::NARROW_OFF;
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
  int nblk = (lk + 127) >> 7;
  if (p.is_causal) {
    const int last_key = min(m_base + 127, lq - 1) + (lk - lq);   // inclusive
    nblk = last_key < 0 ? 0 : min(nblk, (last_key >> 7) + 1);
  }

  // chunk c of the K tile of step j, and dQ of its columns: the barriers
  auto k_full = [&](int j, int c) { return bar(Q_K_FULL0 + (j & 1) * kMaxChunks + c); };
  auto dq_done = [&](int j, int c) { return bar(Q_DQ_DONE0 + (j & 1) * kMaxChunks + c); };
  auto load_k = [&](int j, int c) {
    DBT_TRACE_AT(j, 0);
    tc::mbar_arrive_expect_tx(k_full(j, c), kChunk);
    tc::tma_load_3d(sK + (j & 1) * L::kWide + c * kChunk, &tmap_k, c * 64, head, k0 + j * 128, k_full(j, c));
  };
  auto load_v = [&](int j) {
    const int st = j % L::kNarrowStages;
    DBT_TRACE_AT(j, 1);
    tc::mbar_arrive_expect_tx(bar(Q_V_FULL0 + st), L::kNarrow);
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tma_load_3d(sV + st * L::kNarrow + c * kChunk, &tmap_v, c * 64, head, k0 + j * 128, bar(Q_V_FULL0 + st));
  };
  if (warp == kEwWarps) {
    // the thread that makes the barriers starts the first loads at once, before the others have tensor memory
    if (tc::elect_one()) {
      for (int i = 0; i < Q_NUM_BARS; ++i) tc::mbar_init(bar(i), i >= Q_S_READ ? kEwWarps : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      if (nblk > 0) {
        tc::mbar_arrive_expect_tx(bar(Q_RES_FULL), L::kWide + L::kNarrow);
#pragma unroll
        for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(sQ + c * kChunk, &tmap_q, c * 64, head, q0 + m_base, bar(Q_RES_FULL));
#pragma unroll
        for (int c = 0; c < L::NCH; ++c) load_k(0, c);
#pragma unroll
        for (int c = 0; c < 2; ++c) tc::tma_load_3d(sDO + c * kChunk, &tmap_do, c * 64, head, q0 + m_base, bar(Q_RES_FULL));
        load_v(0);
      }
    }
    __syncwarp();
  }
  if (warp == kEwWarps + 1) tc::tmem_alloc(sbase + L::MISC_OFF, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *sTmem;
  constexpr int TM_DQ = 0, TM_S = 192, TM_DP = 320, TM_DS = 448;

  if (warp == kEwWarps) {
    // ================================ TMA producer =====================================
    // K(j) takes the stage that dQ(j-2) frees, V(j) the one that dP(j-1) (or dP(j-2)) frees, which comes later
    if (tc::elect_one()) {
      bool alive = true;
      for (int j = 1; j < nblk && alive; ++j) {
#pragma unroll 1
        for (int c = 0; c < L::NCH && alive; ++c) {
          alive = tc::mbar_wait(dq_done(j, c), ((j >> 1) & 1) ^ 1, status, 51);
          if (alive) load_k(j, c);
        }
        if (!alive) break;
        const int before = j - L::kNarrowStages;                 // the step whose V the stage holds
        if (before >= 0) alive = tc::mbar_wait(bar(Q_DP_FULL0 + (before & 1)), (before >> 1) & 1, status, 57);
        if (alive) load_v(j);
      }
    }
  } else if (warp > kEwWarps) {
    // ================================ MMA issuers =======================================
    constexpr uint32_t idesc_dq = tc::idesc_bf16_f32(128, 64, 0, 1);
    const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);
    const uint64_t desc_do = tc::smem_desc_sw128(sDO, 16, 1024);
    const uint64_t desc_k = tc::smem_desc_sw128(sK, 16, 1024);              // K tile of stage 0, K-major (B of S)
    const uint64_t desc_v = tc::smem_desc_sw128(sV, 16, 1024);              // V tile of stage 0, K-major (B of dP)
    const uint64_t desc_kt = tc::smem_desc_sw128(sK, kChunk, 1024);         // K tile of stage 0, MN-major (B of dQ)
    bool alive = nblk > 0;
    // Two issuing threads: the first for the first GEMMs of a step (S, dP), the other for the second one (dQ); the waits of one
    // overlap the instructions of the other.
    if (tc::elect_one()) {
      if (warp == kEwWarps + 1) {
        if (alive) alive = tc::mbar_wait(bar(Q_RES_FULL), 0, status, 52);
        for (int j = 0; j < nblk && alive; ++j) {
          const int st = j & 1, stv = j % L::kNarrowStages;
          const uint32_t idesc_sd = tc::idesc_bf16_f32(128, k_steps(lk - j * 128) * 16, 0, 0);
          alive = tc::mbar_wait(bar(Q_S_READ), (j & 1) ^ 1, status, 54);      // the element-wise warps have read S of step j-1
          if (!alive) break;
          DBT_TRACE_AT(j, 2);
          alive = mma_res_stg<L::NCH>(tmem + TM_S, desc_q, tc::desc_advance(desc_k, st * L::kWide), idesc_sd, [&](int c) {
            const bool ok = tc::mbar_wait(k_full(j, c), (j >> 1) & 1, status, 54);
            tc::tc_fence_after();
            return ok;
          });
          if (!alive) break;
          tc::tc_commit(bar(Q_S_FULL));
          alive = tc::mbar_wait(bar(Q_V_FULL0 + stv), (j / L::kNarrowStages) & 1, status, 58);
          if (alive) alive = tc::mbar_wait(bar(Q_DP_READ), (j & 1) ^ 1, status, 58);
          if (!alive) break;
          tc::tc_fence_after();
          DBT_TRACE_AT(j, 3);
          mma_res_stg<2>(tmem + TM_DP, desc_do, tc::desc_advance(desc_v, stv * L::kNarrow), idesc_sd, [](int) { return true; });
          tc::tc_commit(bar(Q_DP_FULL0 + (j & 1)));
        }
      } else {
        for (int j = 0; j < nblk && alive; ++j) {
          const int st = j & 1;
          alive = tc::mbar_wait(bar(Q_DS_FULL), j & 1, status, 53);
          if (!alive) break;
          tc::tc_fence_after();
          DBT_TRACE_AT(j, 4);
#pragma unroll
          for (int c = 0; c < L::NCH; ++c) {
            mma_tmem_stg(tmem + TM_DQ + c * 64, tmem + TM_DS, tc::desc_advance(desc_kt, st * L::kWide + c * kChunk), idesc_dq, j == 0, k_steps(lk - j * 128));
            tc::tc_commit(dq_done(j, c));
          }
          DBT_TRACE_AT(j, 5);
        }
      }
    }
  } else {
    // ================================ element-wise / epilogue ==========================
    // Warps w and w + 4 share the TMEM lanes of 32 rows: warp w takes columns [0, 64) of every 128-key block, warp w + 4
    // the other half.
    const int half = warp >> 2, rl = tid & 127;
    const int row = m_base + rl;
    const bool row_ok = row < lq;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float lse2 = row_ok ? __ldg(p.lse + (int64_t)(q0 + row) * p.lse_stride_t + head * p.lse_stride_h) * kLog2e : 0.f;
    const float dl = row_ok ? __ldg(p.delta + (int64_t)head * p.total_q + q0 + row) : 0.f;
    const int limit = !row_ok ? 0 : (p.is_causal ? max(0, min(lk, row + (lk - lq) + 1)) : lk);
    bool alive = true;
    for (int j = 0; j < nblk && alive; ++j) {
      uint32_t sv[64], dp[64], pk[32];
      alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(Q_S_FULL), j & 1, status, 55));
      if (!alive) break;
      if (tid == 0) DBT_TRACE_AT(j, 6);
      tc::tc_fence_after();
      tmem_ld64(tmem + lane_addr + TM_S + half * 64, sv);
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(Q_S_READ));
      if (tid == 0) DBT_TRACE_AT(j, 7);
      const int cnt = limit - j * 128 - half * 64;             // visible keys of this half block: [0, cnt)
      const bool all_visible = __all_sync(0xffffffffu, cnt >= 64);
      row_exp2(sv, p.scale_log2, [&](int) { return f2(-lse2); });
      if (tid == 0) DBT_TRACE_AT(j, 8);
      alive = __all_sync(0xffffffffu, tc::mbar_wait(bar(Q_DP_FULL0 + (j & 1)), (j >> 1) & 1, status, 59));
      if (!alive) break;
      tc::tc_fence_after();
      tmem_ld64(tmem + lane_addr + TM_DP + half * 64, dp);
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(Q_DP_READ));
      if (tid == 0) DBT_TRACE_AT(j, 9);
      // two loops, not a test per element: the compiler makes a branch of each test (40 clk per element measured)
      auto to_ds = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
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
      if (tid == 0) DBT_TRACE_AT(j, 10);
      // dQ of step j-1 has read dS
      if (j > 0) alive = __all_sync(0xffffffffu, tc::mbar_wait(dq_done(j - 1, L::NCH - 1), ((j - 1) >> 1) & 1, status, 60));
      if (!alive) break;
      // K rows past the end of the sequence must be exact zeros for dQ += dS K
      if (lk - j * 128 < 128) zero_tail(smem + L::WIDE_OFF + (j & 1) * L::kWide, L::NCH, lk - j * 128, tid);
      tc::tc_fence_after();
      tc::tmem_st32(tmem + lane_addr + TM_DS + half * 32, pk);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(Q_DS_FULL));
      if (tid == 0) DBT_TRACE_AT(j, 11);
    }
    bool have = nblk > 0 && alive;
    if (have) {
      have = __all_sync(0xffffffffu, tc::mbar_wait(dq_done(nblk - 1, L::NCH - 1), ((nblk - 1) >> 1) & 1, status, 56));    // the last dQ, hence all of them
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

// ---- 3. dK, dV ----------------------------------------------------------------------------------
// grid (ceil(max_seqlen_k/128), h, batch), 320 threads (warps 0-7 element-wise, 8 TMA, 9 MMA).  Resident: K, V tiles
// of 128 keys.  Per step (128 queries): S^T = K Q^T, dP^T = V dO^T, P^T and dS^T (bf16), dV += P^T dO, dK += dS^T Q.
// TMEM: dV = [0,128), dK = [128, 128 + D_QK), X = [320,448) fp32, Y = [448,512) bf16.
// The 192 columns that dV and dK leave (D_QK = 192) hold one fp32 tile X and one bf16 tile Y, each used twice per step: the
// element-wise warps take a tile of X into registers as soon as it is complete, which frees it for the next one.
//   X: S^T(j), dP^T(j), S^T(j+1), ..      Y: P^T(j) until dV(j) has read it, dS^T(j) until dK(j) has
// The tensor pipe runs dV(j), S^T(j+1), dK(j), dP^T(j+1): while the element-wise warps form P^T(j+1) (from S^T(j+1)), it
// works on dK(j) and dP^T(j+1); while they form dS^T(j), on dV(j) and S^T(j+1).
namespace dbt {
// dV of a step and the release of its dO, dK of a chunk of columns and the release of that chunk of Q (the last one: and of Y), are one
// event each, with two barriers in turn
enum BarK { K_RES_FULL = 0, K_Q_FULL0, K_DK_DONE0 = K_Q_FULL0 + 2 * kMaxChunks, K_DO_FULL0 = K_DK_DONE0 + 2 * kMaxChunks, K_DO_FULL1, K_DV_DONE0, K_DV_DONE1, K_S_FULL, K_DP_FULL,
            K_S_READ, K_DP_READ, K_P_FULL, K_DS_FULL, K_NUM_BARS };   // K_S_READ and later: one arrival per element-wise warp
}

template <int D_QK>
__global__ void __launch_bounds__(dbt::kDkvThreads, 1)
dense_bwd_dkdv_tc_kernel(const __grid_constant__ DenseKernelParams p, const __grid_constant__ CUtensorMap tmap_k,
                         const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_q,
                         const __grid_constant__ CUtensorMap tmap_do) {
  using namespace dbt;
  using L = Layout<D_QK>;
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sK = sbase + L::RES_OFF, sV = sK + L::kWide, sQ = sbase + L::WIDE_OFF, sDO = sbase + L::NARROW_OFF;
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
  // query blocks [jb_lo, jb_hi) of 128 rows that see at least one key of this tile
  const int jb_hi = (lq + 127) >> 7;
  const int jb_lo = p.is_causal ? min(jb_hi, max(0, n_base - (lk - lq)) >> 7) : 0;
  const int nstep = jb_hi - jb_lo;

  // chunk c of the Q tile of step j, and dK of its columns: the barriers
  auto q_full = [&](int j, int c) { return bar(K_Q_FULL0 + (j & 1) * kMaxChunks + c); };
  auto dk_done = [&](int j, int c) { return bar(K_DK_DONE0 + (j & 1) * kMaxChunks + c); };
  auto load_q = [&](int j, int c) {
    tc::mbar_arrive_expect_tx(q_full(j, c), kChunk);
    tc::tma_load_3d(sQ + (j & 1) * L::kWide + c * kChunk, &tmap_q, c * 64, head, q0 + (jb_lo + j) * 128, q_full(j, c));
  };
  auto load_do = [&](int j) {
    const int st = j % L::kNarrowStages;
    tc::mbar_arrive_expect_tx(bar(K_DO_FULL0 + st), L::kNarrow);
#pragma unroll
    for (int c = 0; c < 2; ++c)
      tc::tma_load_3d(sDO + st * L::kNarrow + c * kChunk, &tmap_do, c * 64, head, q0 + (jb_lo + j) * 128, bar(K_DO_FULL0 + st));
  };
  if (warp == kEwWarps) {
    // as in the dQ kernel: barriers and first loads before the others have tensor memory
    if (tc::elect_one()) {
      for (int i = 0; i < K_NUM_BARS; ++i) tc::mbar_init(bar(i), i >= K_S_READ ? kEwWarps : 1);
      tc::fence_mbar_init();
      tc::fence_proxy_async_smem();
      *sAbort = 0;
      if (nstep > 0) {
        tc::mbar_arrive_expect_tx(bar(K_RES_FULL), L::kWide + L::kNarrow);
#pragma unroll
        for (int c = 0; c < L::NCH; ++c) tc::tma_load_3d(sK + c * kChunk, &tmap_k, c * 64, head, k0 + n_base, bar(K_RES_FULL));
#pragma unroll
        for (int c = 0; c < L::NCH; ++c) load_q(0, c);
#pragma unroll
        for (int c = 0; c < 2; ++c) tc::tma_load_3d(sV + c * kChunk, &tmap_v, c * 64, head, k0 + n_base, bar(K_RES_FULL));
        load_do(0);
      }
    }
    __syncwarp();
  }
  if (warp == kEwWarps + 1) tc::tmem_alloc(sbase + L::MISC_OFF, 512);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *sTmem;
  constexpr int TM_DV = 0, TM_DK = 128, TM_X = 320, TM_Y = 448;

  if (warp == kEwWarps) {
    // ================================ TMA producer =====================================
    // Q(j) takes the stage that dK(j-2) frees, dO(j) the one that dV(j-1) (or dV(j-2)) frees, which comes later
    if (tc::elect_one()) {
      bool alive = true;
      for (int j = 1; j < nstep && alive; ++j) {
#pragma unroll 1
        for (int c = 0; c < L::NCH && alive; ++c) {
          alive = tc::mbar_wait(dk_done(j, c), ((j >> 1) & 1) ^ 1, status, 61);
          if (alive) load_q(j, c);
        }
        if (!alive) break;
        const int before = j - L::kNarrowStages;                 // the step whose dO the stage holds
        if (before >= 0) alive = tc::mbar_wait(bar(K_DV_DONE0 + (before & 1)), (before >> 1) & 1, status, 73);
        if (alive) load_do(j);
      }
    }
  } else if (warp == kEwWarps + 1) {
    // ================================ MMA issuer =======================================
    constexpr uint32_t idesc_dv = tc::idesc_bf16_f32(128, 128, 0, 1);
    constexpr uint32_t idesc_dk = tc::idesc_bf16_f32(128, 64, 0, 1);
    const uint64_t desc_k = tc::smem_desc_sw128(sK, 16, 1024);
    const uint64_t desc_v = tc::smem_desc_sw128(sV, 16, 1024);
    const uint64_t desc_q = tc::smem_desc_sw128(sQ, 16, 1024);              // Q tile of stage 0, K-major (B of S^T)
    const uint64_t desc_do = tc::smem_desc_sw128(sDO, 16, 1024);            // dO tile of stage 0, K-major (B of dP^T)
    const uint64_t desc_qt = tc::smem_desc_sw128(sQ, kChunk, 1024);         // Q tile, MN-major (B of dK)
    const uint64_t desc_dot = tc::smem_desc_sw128(sDO, kChunk, 1024);       // dO tile, MN-major (B of dV)
    if (tc::elect_one() && nstep > 0) {
      bool alive = tc::mbar_wait(bar(K_RES_FULL), 0, status, 62);
      auto wait = [&](int i, int ph, int code) {
        if (alive) alive = tc::mbar_wait(bar(i), ph, status, code);
        return alive;
      };
      auto rows_valid = [&](int j) { return lq - (jb_lo + j) * 128; };
      // S^T of step j, once its Q tile has landed and dP^T of step j-1 has been read; dP^T of step j likewise
      auto issue_s = [&](int j) {
        const int st = j & 1;
        if (!wait(K_DP_READ, (j & 1) ^ 1, 67)) return;
        alive = mma_res_stg<L::NCH>(tmem + TM_X, desc_k, tc::desc_advance(desc_q, st * L::kWide), tc::idesc_bf16_f32(128, k_steps(rows_valid(j)) * 16, 0, 0), [&](int c) {
          const bool ok = tc::mbar_wait(q_full(j, c), (j >> 1) & 1, status, 63);
          tc::tc_fence_after();
          return ok;
        });
        if (alive) tc::tc_commit(bar(K_S_FULL));
      };
      auto issue_dp = [&](int j) {
        const int st = j % L::kNarrowStages;
        if (!wait(K_DO_FULL0 + st, (j / L::kNarrowStages) & 1, 74)) return;
        if (!wait(K_S_READ, j & 1, 64)) return;
        tc::tc_fence_after();
        mma_res_stg<2>(tmem + TM_X, desc_v, tc::desc_advance(desc_do, st * L::kNarrow), tc::idesc_bf16_f32(128, k_steps(rows_valid(j)) * 16, 0, 0), [](int) { return true; });
        tc::tc_commit(bar(K_DP_FULL));
      };
      // step j = -1 issues the first GEMMs of step 0 (the instructions of a step exist once)
      for (int j = -1; j < nstep && alive; ++j) {
        const int st = j & 1, std = (j & 1) % L::kNarrowStages, ks = k_steps(rows_valid(j));
        if (j >= 0) {
          if (!wait(K_P_FULL, j & 1, 68)) break;
          tc::tc_fence_after();
          mma_tmem_stg(tmem + TM_DV, tmem + TM_Y, tc::desc_advance(desc_dot, std * L::kNarrow), idesc_dv, j == 0, ks);
          tc::tc_commit(bar(K_DV_DONE0 + st));
        }
        if (j + 1 < nstep) issue_s(j + 1);
        if (j >= 0) {
          if (!wait(K_DS_FULL, j & 1, 69)) break;
          tc::tc_fence_after();
#pragma unroll
          for (int c = 0; c < L::NCH; ++c) {
            mma_tmem_stg(tmem + TM_DK + c * 64, tmem + TM_Y, tc::desc_advance(desc_qt, st * L::kWide + c * kChunk), idesc_dk, j == 0, ks);
            tc::tc_commit(dk_done(j, c));              // completes after dV of this step: the tensor pipe runs in order
          }
        }
        if (j + 1 < nstep) issue_dp(j + 1);
      }
    }
  } else {
    // ================================ element-wise / epilogue ==========================
    // warps w and w + 4 share the TMEM lanes of 32 keys: warp w takes queries [0, 64) of every block, warp w + 4 the rest
    const int half = warp >> 2, rl = tid & 127;
    const int key = n_base + rl;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int shift = lk - lq;                                 // query i sees keys <= i + shift
    // Per-query vectors of a step: -lse * log2(e) (threads 0-127) and -delta (threads 128-255).  Each value is loaded one step ahead and
    // not touched before the next: a product right behind the load waited for it, some 800 clk of a step's 3 900.
    const float* vec = tid < 128 ? p.lse + (int64_t)q0 * p.lse_stride_t + head * p.lse_stride_h : p.delta + (int64_t)head * p.total_q + q0;
    const int64_t vec_stride = tid < 128 ? p.lse_stride_t : 1;
    const float vec_mul = tid < 128 ? -kLog2e : -1.f;
    auto load_vec = [&](int j) {
      const int i = (jb_lo + j) * 128 + rl;
      return i < lq ? __ldg(vec + i * vec_stride) : 0.f;
    };
    float v_next = nstep > 0 ? load_vec(0) : 0.f;
    bool alive = true;
    for (int j = 0; j < nstep && alive; ++j) {
      const int jb = jb_lo + j, vb = j & 1;
      sVec[vb * 256 + tid] = v_next * vec_mul;
      if (j + 1 < nstep) v_next = load_vec(j + 1);
      if (!tc::mbar_wait(bar(K_S_FULL), j & 1, status, 65)) *sAbort = 1;
      bar_sync(1, kEwWarps * 32);                              // vectors visible; also keeps the two buffers of sVec apart
      if (*sAbort) { alive = false; break; }                   // read right after the barrier: the same for all threads
      tc::tc_fence_after();
      uint32_t sv[64], dp[64], pk[32];
      tmem_ld64(tmem + lane_addr + TM_X + half * 64, sv);
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_S_READ));
      const int c_max = lq - jb * 128 - half * 64;             // columns (queries) [c_min, c_max) see this key
      const int c_min = p.is_causal ? key - shift - jb * 128 - half * 64 : 0;
      const bool all_visible = __all_sync(0xffffffffu, c_min <= 0 && c_max >= 64);
      const float4* vl = reinterpret_cast<const float4*>(sVec + vb * 256 + half * 64);
      const float4* vd = reinterpret_cast<const float4*>(sVec + vb * 256 + 128 + half * 64);
      // two loops, not a test per element: the compiler makes a branch of each test (40 clk per element measured)
      row_exp2(sv, p.scale_log2, [&](int i) {
        const float4 l4 = vl[i >> 1];
        return i & 1 ? F2{l4.z, l4.w} : F2{l4.x, l4.y};
      });
      auto to_p = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
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
      if (j > 0 && !tc::mbar_wait(dk_done(j - 1, L::NCH - 1), ((j - 1) >> 1) & 1, status, 70)) *sAbort = 1;      // dK of step j-1 has read Y
      if (lq - jb * 128 < 128) {      // the last step: rows past the end of the sequence must be exact zeros for dV and dK
        const int std = j % L::kNarrowStages;
        if (!tc::mbar_wait(bar(K_DO_FULL0 + std), (j / L::kNarrowStages) & 1, status, 74)) *sAbort = 1;
        zero_tail(smem + L::NARROW_OFF + std * L::kNarrow, 2, lq - jb * 128, tid);
        zero_tail(smem + L::WIDE_OFF + (j & 1) * L::kWide, L::NCH, lq - jb * 128, tid);
      }
      tc::tc_fence_after();
      __syncwarp();
      tc::tmem_st32(tmem + lane_addr + TM_Y + half * 32, pk);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_P_FULL));
      if (!tc::mbar_wait(bar(K_DP_FULL), j & 1, status, 71)) *sAbort = 1;
      tc::tc_fence_after();
      __syncwarp();
      tmem_ld64(tmem + lane_addr + TM_X + half * 64, dp);
      tc::tmem_wait_ld();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_DP_READ));
      auto to_ds = [&](auto masked) {
#pragma unroll
        for (int i4 = 0; i4 < 16; ++i4) {
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
      if (!tc::mbar_wait(bar(K_DV_DONE0 + (j & 1)), (j >> 1) & 1, status, 72)) *sAbort = 1;            // dV of this step has read Y
      tc::tc_fence_after();
      __syncwarp();
      tc::tmem_st32(tmem + lane_addr + TM_Y + half * 32, pk);
      tc::tmem_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(K_DS_FULL));
    }
    bool have = nstep > 0 && alive;
    if (have) {
      have = __all_sync(0xffffffffu, tc::mbar_wait(dk_done(nstep - 1, L::NCH - 1), ((nstep - 1) >> 1) & 1, status, 66));   // the last dK, hence all of them
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

#include "dense_bwd_steps64.cuh"

namespace fmla {

// ---- host side ----------------------------------------------------------------------------------
// Kernels and shared memory of either step
template <int D_QK, bool STEPS64>
struct BwdForm {
  static constexpr auto kq = dense_bwd_dq_tc_kernel<D_QK>;
  static constexpr auto kk = dense_bwd_dkdv_tc_kernel<D_QK>;
  static constexpr int kSmem = dbt::Layout<D_QK>::SMEM_BYTES, kStep = 128;
};
template <int D_QK>
struct BwdForm<D_QK, true> {
  static constexpr auto kq = dense_bwd_dq_tc64_kernel<D_QK>;
  static constexpr auto kk = dense_bwd_dkdv_tc64_kernel<D_QK>;
  static constexpr int kSmem = dbt64::Layout<D_QK>::SMEM_BYTES, kStep = 64;
};

template <int D_QK, bool STEPS64>
static cudaError_t launch_bwd_tc(const DenseKernelParams& p, cudaStream_t stream) {
  using namespace dbt;
  using Form = BwdForm<D_QK, STEPS64>;
  // of each tensor a map for resident tiles and one for streamed tiles
  CUtensorMap q, d_o, k, v, q_step, do_step, k_step, v_step;
  auto maps = [&](CUtensorMap& tile, CUtensorMap& step, const void* x, int d, int heads, int tokens, int64_t stride_h, int64_t stride_t) {
    if (!tmah::make_map_thd(&tile, x, d, heads, tokens, stride_h, stride_t, 128)) return false;
    if (Form::kStep == 128) { step = tile; return true; }
    return tmah::make_map_thd(&step, x, d, heads, tokens, stride_h, stride_t, Form::kStep);
  };
  if (!(maps(q, q_step, p.q, p.d_qk, p.h_q, p.total_q, p.q_stride_h, p.q_stride_t) && maps(d_o, do_step, p.d_o, p.d_v, p.h_q, p.total_q, p.do_stride_h, p.do_stride_t) &&
        maps(k, k_step, p.k, p.d_qk, p.h_k, p.total_k, p.k_stride_h, p.k_stride_t) && maps(v, v_step, p.v, p.d_v, p.h_k, p.total_k, p.v_stride_h, p.v_stride_t)))
    return cudaErrorInvalidValue;
  constexpr auto kq = Form::kq;
  constexpr auto kk = Form::kk;
  if (cudaError_t e = allow_smem<kq>(Form::kSmem); e != cudaSuccess) return e;
  if (cudaError_t e = allow_smem<kk>(Form::kSmem); e != cudaSuccess) return e;
  const int64_t rows = (int64_t)p.total_q * p.h_q;
  const int64_t per_block = 16 * kDeltaRows;
  dense_bwd_delta_tc_kernel<<<static_cast<unsigned>((rows + per_block - 1) / per_block), 256, 0, stream>>>(p);
  kk<<<dim3((p.max_seqlen_k + 127) / 128, p.h_q, p.batch), kDkvThreads, Form::kSmem, stream>>>(p, k, v, q_step, do_step);
  if (cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
  const dim3 grid((p.max_seqlen_q + 127) / 128, p.h_q, p.batch);
  // dQ written over Q or dO (which its own kernel reads tile by tile, before it writes) must wait until dK / dV has read them
  const auto overlaps = [&](const void* x, int d, int64_t stride_t, int64_t stride_h) {
    const auto end = [&](const void* base, int dim, int64_t st, int64_t sh) {
      return reinterpret_cast<uintptr_t>(base) + 2 * ((p.total_q - 1) * st + (p.h_q - 1) * sh + dim);
    };
    return reinterpret_cast<uintptr_t>(p.dq) < end(x, d, stride_t, stride_h) &&
           reinterpret_cast<uintptr_t>(x) < end(p.dq, p.d_qk, p.dq_stride_t, p.dq_stride_h);
  };
  if (overlaps(p.q, p.d_qk, p.q_stride_t, p.q_stride_h) || overlaps(p.d_o, p.d_v, p.do_stride_t, p.do_stride_h)) {
    kq<<<grid, kDqThreads, Form::kSmem, stream>>>(p, q, d_o, k_step, v_step);
    return cudaGetLastError();
  }
  return launch_dependent(kq, grid, kDqThreads, Form::kSmem, stream, p, q, d_o, k_step, v_step);
}

cudaError_t launch_dense_bwd_tc(const DenseKernelParams& p, cudaStream_t stream) {
  // Steps of 64 rows for short sequences: the last step of 128 works for up to 127 rows in vain, and with a causal mask tiles walk half of
  // a sequence.  By the mean length, which is what the host has; steps of 64 -> steps of 128, at this length and a multiple of a step or
  // half of one beyond it, some 2 400 tokens in all.  Causal, 16 heads, 192/128: 64 tokens 49.4 -> 59.7 us, 320 47.7 -> 51.6, 512 47.8 -> 46.8, 704
  // 57.8 -> 60.1, 1088 72.7 -> 73.1, 1216 48.4 -> 46.4, 1500 63.9 -> 61.5, 2000 99.1 -> 92.0; 64 heads, 128/128: 320 163 -> 172, 512 157 -> 150, 704 190 -> 193,
  // 1088 240 -> 236, 1500 201 -> 193.  Without a mask, 64 heads, 128/128: 64 tokens 179 -> 207, 320 185 -> 195, 384 185 -> 180, 448 215 -> 222, 512 193 -> 183;
  // 192/128: 320 212 -> 226, 384 216 -> 208, 448 255 -> 256, 512 226 -> 219.  Up to the lines steps of 64 win more on the odd halves of a step than
  // they lose on whole ones.
  const int64_t mean = (static_cast<int64_t>(p.total_q) + p.total_k) / (2 * static_cast<int64_t>(p.batch));
  const bool short_sequences = mean <= (p.is_causal ? 1088 : 352);
  if (p.d_qk == 192) return short_sequences ? launch_bwd_tc<192, true>(p, stream) : launch_bwd_tc<192, false>(p, stream);
  return short_sequences ? launch_bwd_tc<128, true>(p, stream) : launch_bwd_tc<128, false>(p, stream);
}

#ifdef FMLA_TRACE
extern "C" int fmla_debug_read_dense_bwd_trace(long long* host, int n) {
  return (int)cudaMemcpyFromSymbol(host, g_dense_bwd_trace, sizeof(long long) * n);
}
#endif

cudaError_t set_status_mirror_dense_bwd(int* mapped_host_word) { return tc::set_status_mirror(mapped_host_word); }

cudaError_t read_dense_bwd_tc_status(int* host_status, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(host_status, g_dense_bwd_tc_status, sizeof(int));
  if (e != cudaSuccess) return e;
  if (reset && *host_status != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_dense_bwd_tc_status, &zero, sizeof(int));
  }
  return e;
}

}  // namespace fmla
