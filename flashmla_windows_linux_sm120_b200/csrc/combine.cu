// Log-sum-exp merge of split-KV partial results.
//
// Math of csrc/smxx/mla_combine.cu:71-107, 128-151: with base-2 partial LSEs
// lse_i and normalised partial outputs o_i,
//   lse = log2(sum_i 2^lse_i)  (computed max-shifted; all -inf -> +inf),
//   o   = sum_i 2^(lse_i - lse) * o_i,
// written as natural-log LSE and bf16 O.  One warp per output row, any number of
// parts (the reference is limited to 64, mla_combine.cu:156-167).  Each lane
// owns 16 of the 512 output columns as 4 float4 so a warp reads 512 B
// contiguous per load instruction.
#include "fmla_common.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "mla_work.cuh"
#include "tc_common.cuh"

namespace fmla {

constexpr int kCombineWarps = 8;

// Weights 2^(lse_i - lse) of the parts of a row -> s_w (whole warp); returns the base-2 LSE of the row.  A NaN among the parts gives NaN
// outputs and, for requests that the schedule splits, +inf.  keep_nan: what one CTA gives for the whole row, NaN; for rows that the
// schedule, or the caller, knows as whole.  Each part's LSE is read once by rows of up to 32 parts: the lane keeps it.
template <class LseAt>
__device__ __forceinline__ float combine_weights(int nparts, LseAt lse_at, float* s_w, bool keep_nan = false) {
  const int lane = threadIdx.x & 31;
  const float own = lane < nparts ? lse_at(lane) : neg_inf();
  float mx = own;
#pragma unroll 1
  for (int i = lane + 32; i < nparts; i += 32) mx = fmaxf(mx, lse_at(i));
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if (mx == neg_inf()) mx = 0.f;
  float sum = lane < nparts ? exp2f(own - mx) : 0.f;
#pragma unroll 1
  for (int i = lane + 32; i < nparts; i += 32) sum += exp2f(lse_at(i) - mx);
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  const float glse = (sum == 0.f || (sum != sum && !keep_nan)) ? pos_inf() : log2f(sum) + mx;
  if (lane < nparts) s_w[lane] = exp2f(own - glse);
#pragma unroll 1
  for (int i = lane + 32; i < nparts; i += 32) s_w[i] = exp2f(lse_at(i) - glse);
  __syncwarp();
  return glse;
}

// Weighted sum of the parts share, share + SHARES, .. over column groups [first, first + NG) of 128 columns (lane = 4 columns of a
// group), in the order of the parts; with several shares each has the CTA's warps 4 share .. 4 share + 3, and those of share 0 add up
// what the others leave in s_acc.  weights() fills s_w; the first loads are in flight meanwhile.  A part with weight 0 is left out of
// the sum (0 * (Inf or NaN) must not reach it) and, past the first loads, not read.
// What bounds a merge of few rows is its chain of round trips to L2 (about 0.6 us each): the schedule, the LSEs, then PARTS parts at
// a time.  With the schedule read ahead of the wait, the first parts asked for together with the LSEs and these read once, a decode
// with a merge takes 0.7 to 2 us less: 64 heads, 4 x 400 tokens 18.9 -> 17.7 us, 128 heads, 4 x 500 17.2 -> 15.7.
// PARTS is what keeps four 16-byte loads per lane in flight, and more where that leaves all CTAs resident (launch_decode_combine).  With
// four parts of four groups each the merge needed 98 registers, too many to wait beside an attention CTA, and 1024 of its CTAs
// (64 requests x 128 heads) took three and a half waves.
// COHERENT: the partial outputs may have been written by another GPU while this kernel was already resident (peer
// merge), so they are read with ld.global.cv.  Otherwise plain loads: the merge of a decode call is resident, waiting in
// pdl_wait(), while the attention kernel writes the partials, and the non-coherent path (__ldg) is undefined for memory
// modified during the kernel's lifetime.
template <int NG, bool COHERENT, int SHARES = 1, int PARTS = 4 / NG, class OAt, class Weights>
__device__ __forceinline__ void combine_columns(int nparts, OAt o_at, const float* s_w, Weights weights, __nv_bfloat16* out_row, int first, bool f16,
                                                int share = 0, float4 (*s_acc)[4][32] = nullptr) {
  const int lane = threadIdx.x & 31;
  float4 acc[NG], v[PARTS][NG];
  float w[PARTS];
#pragma unroll
  for (int j = 0; j < NG; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
  const auto load = [&](int i, float4 (&to)[NG]) {
    const float4* src = reinterpret_cast<const float4*>(o_at(i)) + first * 32 + lane;
#pragma unroll
    for (int j = 0; j < NG; ++j) to[j] = COHERENT ? __ldcv(src + j * 32) : src[j * 32];
  };
  const auto add = [&] {
#pragma unroll
    for (int u = 0; u < PARTS; ++u) {
      if (w[u] == 0.f) continue;
#pragma unroll
      for (int j = 0; j < NG; ++j) {
        acc[j].x += w[u] * v[u][j].x;
        acc[j].y += w[u] * v[u][j].y;
        acc[j].z += w[u] * v[u][j].z;
        acc[j].w += w[u] * v[u][j].w;
      }
    }
  };
#pragma unroll
  for (int u = 0; u < PARTS; ++u)
    if (share + u * SHARES < nparts) load(share + u * SHARES, v[u]);
  weights();
#pragma unroll
  for (int u = 0; u < PARTS; ++u) w[u] = share + u * SHARES < nparts ? s_w[share + u * SHARES] : 0.f;
  add();
#pragma unroll 1
  for (int i0 = share + PARTS * SHARES; i0 < nparts; i0 += PARTS * SHARES) {
#pragma unroll
    for (int u = 0; u < PARTS; ++u) {
      const int i = i0 + u * SHARES;
      w[u] = i < nparts ? s_w[i] : 0.f;
      if (w[u] != 0.f) load(i, v[u]);
    }
    add();
  }
  if constexpr (SHARES > 1) {
    static_assert(NG == 1, "one column group per warp");
    if (share > 0) s_acc[share - 1][first][lane] = acc[0];
    __syncthreads();
    if (share > 0) return;
#pragma unroll
    for (int i = 0; i < SHARES - 1; ++i) {
      const float4 v = s_acc[i][first][lane];
      acc[0].x += v.x;
      acc[0].y += v.y;
      acc[0].z += v.z;
      acc[0].w += v.w;
    }
  }
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    // out_row addresses 16-bit elements: bf16, or fp16 when the queries were fp16
    uint2 packed = f16 ? make_uint2(pack_f16x2(acc[j].x, acc[j].y), pack_f16x2(acc[j].z, acc[j].w))
                       : make_uint2(pack_bf16x2(acc[j].x, acc[j].y), pack_bf16x2(acc[j].z, acc[j].w));
    *reinterpret_cast<uint2*>(out_row + ((first + j) * 32 + lane) * 4) = packed;
  }
}

template <bool COHERENT = false, class LseAt, class OAt>
__device__ __forceinline__ void combine_row(int nparts, LseAt lse_at, OAt o_at, float* s_w, __nv_bfloat16* out_row,
                                            float* lse_out) {
  const auto weights = [&] {
    const float glse = combine_weights(nparts, lse_at, s_w);
    if ((threadIdx.x & 31) == 0) *lse_out = glse * kLn2;
  };
  combine_columns<4, COHERENT>(nparts, o_at, s_w, weights, out_row, 0, false);
}

// grid (b, ceil(h_k*q_seq_per_hk / rows per CTA)); requests with a single part were written
// in final form by the attention kernel and are skipped (mla_combine.cu:30-32).
// WPR warps per row, each for 4 / WPR of the row's four 128-column groups; with more than four, a CTA takes one row and every four
// warps a share of its parts.
constexpr int combine_warps(int wpr) { return wpr > kCombineWarps ? wpr : kCombineWarps; }
// PARTS: parts in flight per warp where a row has several shares.
template <int WPR, bool SHARED, int PARTS>
__global__ void __launch_bounds__(combine_warps(WPR) * 32) decode_combine_kernel(const __grid_constant__ DecodeKernelParams p) {
  extern __shared__ float s_weights[];  // [8][num_sm_parts]
  // The schedule is read before the wait for the attention kernel: each of its CTAs waits for the kernels in front of it before it
  // lets this one start, so whoever writes the schedule has completed.  That its writes are visible here by then is not written
  // down for a kernel two places behind; it holds because the wait of the attention kernel completes them to L2 and this grid starts later, with
  // nothing of the schedule in its SMs' L1.  Plain loads all the same (mla_work.cuh).
  const int batch = blockIdx.x;
  int lo = p.num_splits[batch], hi = p.num_splits[batch + 1];
  const bool whole = hi - lo == 1;      // in the schedule
  if constexpr (SHARED) {
    const int k = sub_splits<false>(p);
    lo *= k;
    hi *= k;
  }
  const int nparts = hi - lo;
  const int q_seq_per_hk = p.s_q * p.hq_per_hk;
  const int rows = p.h_k * q_seq_per_hk;
  constexpr int kShares = WPR > 4 ? WPR / 4 : 1, kGroups = WPR > 4 ? 4 : WPR;
  static_assert(kShares == 1 || combine_warps(WPR) == WPR, "the warps of a CTA meet at a barrier");
  __shared__ float4 s_acc[kShares > 1 ? kShares - 1 : 1][4][32];
  const int warp = threadIdx.x >> 5, sub = warp % WPR;
  const int r = blockIdx.y * (combine_warps(WPR) / WPR) + warp / WPR;
  const int kh = r / q_seq_per_hk, row = r % q_seq_per_hk;
  const int sq = row / p.hq_per_hk, head = kh * p.hq_per_hk + row % p.hq_per_hk;
  const float* lse_base = p.lse_accum + (int64_t)lo * rows + r;
  const float* o_base = p.o_accum + ((int64_t)lo * rows + r) * 512;
  const int64_t part_stride = rows;
  float* w = s_weights + warp * p.num_sm_parts;
  const auto weights = [&] {
    const float glse = combine_weights(nparts, [&](int i) { return lse_base[i * part_stride]; }, w, SHARED && whole);
    if (sub == 0 && (threadIdx.x & 31) == 0) p.softmax_lse[((int64_t)batch * p.h_q + head) * p.s_q + sq] = glse * kLn2;
  };
  // Launched as a programmatic dependent of the attention kernel: plain loads of what it leaves.  Warps without a part to merge wait
  // too: what follows in the stream, or in a graph, is ordered behind this kernel alone, which must not end before that one, and
  // where no request is split all of it is without parts.
  pdl_wait();
  if (nparts <= 1 || r >= rows) return;
  combine_columns<4 / kGroups, false, kShares, PARTS>(
      nparts, [&](int i) { return o_base + i * part_stride * 512; }, w, weights,
      reinterpret_cast<__nv_bfloat16*>(p.out) + batch * p.o_stride_b + sq * p.o_stride_s + head * p.o_stride_h, sub % kGroups * (4 / kGroups),
      p.is_f16 != 0, sub / kGroups, s_acc);
}

// The same for the query tokens of a sparse prefill that are cut (SparsePrefillKernelParams): grid (such tokens, h_q / rows per
// CTA); base-2 log-sum-exp and largest logit beside the output, -inf where no part has a valid index.
template <int WPR>
__global__ void __launch_bounds__(kCombineWarps * 32) sparse_prefill_combine_kernel(const __grid_constant__ SparsePrefillKernelParams p) {
  extern __shared__ float s_weights[];  // [8][per]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = warp % WPR;
  const int head = blockIdx.y * (kCombineWarps / WPR) + warp / WPR;
  const int64_t first = (int64_t)blockIdx.x * p.per * p.h_q + head;
  pdl_wait();                           // launched as a programmatic dependent of the attention kernel: plain loads from here on
  float* w = s_weights + warp * p.per;
  const int64_t out_row = (int64_t)(p.whole + blockIdx.x) * p.h_q + head;
  const auto weights = [&] {
    const float glse = combine_weights(p.per, [&](int i) { return p.lse_accum[first + (int64_t)i * p.h_q]; }, w, true);
    if (sub == 0) {
      float mx = neg_inf();
      for (int i = lane; i < p.per; i += 32) mx = fmaxf(mx, p.max_accum[first + (int64_t)i * p.h_q]);
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      if (lane == 0) {
        p.max_logits[out_row] = mx;
        p.lse[out_row] = glse == pos_inf() ? neg_inf() : glse;
      }
    }
  };
  combine_columns<4 / WPR, false>(p.per, [&](int i) { return p.o_accum + (first + (int64_t)i * p.h_q) * 512; }, w, weights,
                                  reinterpret_cast<__nv_bfloat16*>(p.out) + out_row * 512, sub * (4 / WPR), false);
}

__global__ void __launch_bounds__(kCombineWarps * 32)
combine_partials_kernel(const float* __restrict__ lse_accum, const float* __restrict__ o_accum, int nparts, int rows,
                        __nv_bfloat16* __restrict__ out, int64_t o_stride_row, float* __restrict__ lse) {
  extern __shared__ float s_weights[];  // [8][nparts]
  const int warp = threadIdx.x >> 5;
  const int r = blockIdx.x * kCombineWarps + warp;
  if (r >= rows) return;
  combine_row(
      nparts, [&](int i) { return __ldg(lse_accum + (int64_t)i * rows + r); },
      [&](int i) { return o_accum + ((int64_t)i * rows + r) * 512; }, s_weights + warp * nparts, out + r * o_stride_row,
      lse + r);
}

// ---- KV-sharded decode across GPUs ---------------------------------------------------------------
// Each rank merges its local splits per row and stores the normalised fp32 result + base-2 LSE
// into its slot of every destination's partial buffers with plain (peer) stores; the last CTA to
// finish publishes the epoch in the destinations' flag words (release, system scope).
__device__ __forceinline__ void st_release_sys(unsigned int* addr, unsigned int v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;\n" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys(const unsigned int* addr) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];\n" : "=r"(v) : "l"(addr) : "memory");
  return v;
}

__global__ void __launch_bounds__(kCombineWarps * 32) decode_combine_push_kernel(const __grid_constant__ DecodeKernelParams p) {
  extern __shared__ float s_weights[];  // [8][num_sm_parts]
  const int batch = blockIdx.x;
  const int lo = __ldg(p.num_splits + batch), hi = __ldg(p.num_splits + batch + 1);
  const int nparts = hi - lo;
  const int q_seq_per_hk = p.s_q * p.hq_per_hk;
  const int rows = p.h_k * q_seq_per_hk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.y * kCombineWarps + warp;
  if (r < rows) {
    const float* lse_base = p.lse_accum + (int64_t)lo * rows + r;
    const float* o_base = p.o_accum + ((int64_t)lo * rows + r) * 512;
    float* w = s_weights + warp * p.num_sm_parts;
    float mx = neg_inf();
    for (int i = lane; i < nparts; i += 32) mx = fmaxf(mx, __ldg(lse_base + (int64_t)i * rows));
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float mref = mx == neg_inf() ? 0.f : mx;
    float sum = 0.f;
    for (int i = lane; i < nparts; i += 32) sum += exp2f(__ldg(lse_base + (int64_t)i * rows) - mref);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float glse = (sum == 0.f || sum != sum) ? neg_inf() : log2f(sum) + mref;   // base 2, -inf = empty shard
    for (int i = lane; i < nparts; i += 32) w[i] = glse == neg_inf() ? 0.f : exp2f(__ldg(lse_base + (int64_t)i * rows) - glse);
    __syncwarp();
    float4 acc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = 0; i < nparts; ++i) {
      const float wi = w[i];
      if (wi == 0.f) continue;
      const float4* src = reinterpret_cast<const float4*>(o_base + (int64_t)i * rows * 512);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 v = __ldg(src + j * 32 + lane);
        acc[j].x += wi * v.x; acc[j].y += wi * v.y; acc[j].z += wi * v.z; acc[j].w += wi * v.w;
      }
    }
    const int64_t total_rows = (int64_t)p.b * rows;
    const int64_t grow = (int64_t)p.push_slot * total_rows + (int64_t)batch * rows + r;
    for (int d = 0; d < p.push_num_dst; ++d) {
      float4* dst = reinterpret_cast<float4*>(p.push_o[d] + grow * 512);
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[j * 32 + lane] = acc[j];
      if (lane == 0) p.push_lse[d][grow] = glse;
    }
  }
  // publish: every thread's peer stores are ordered before the flag by fence + barrier + release
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int total = gridDim.x * gridDim.y;
    const unsigned int done = atomicAdd(p.push_counter, 1u) + 1u;
    if (done == total) {
      __threadfence_system();
      for (int d = 0; d < p.push_num_dst; ++d) st_release_sys(p.push_flag[d] + p.push_slot, p.push_epoch);
      *p.push_counter = 0u;
    }
  }
}

// Merge of per-rank partials that arrive through peer stores: wait (bounded) for every rank's flag.
__global__ void __launch_bounds__(kCombineWarps * 32)
merge_peer_partials_kernel(const float* __restrict__ lse_accum, const float* __restrict__ o_accum, int nparts, int rows,
                           __nv_bfloat16* __restrict__ out, int64_t o_stride_row, float* __restrict__ lse,
                           const unsigned int* __restrict__ flags, unsigned int epoch, int max_polls, int* status) {
  extern __shared__ float s_weights[];  // [8][nparts]
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 1;
    for (int i = 0; i < nparts && ok; ++i) {
      int polls = 0;
      while (ld_acquire_sys(flags + i) != epoch) {
        if (++polls > max_polls) { ok = 0; break; }
        __nanosleep(200);
      }
    }
    if (!ok) tc::report_status(status, 20);
    s_ok = ok;
  }
  __syncthreads();
  if (!s_ok) return;     // the caller reads the status word; outputs are left untouched
  const int warp = threadIdx.x >> 5;
  const int r = blockIdx.x * kCombineWarps + warp;
  if (r >= rows) return;
  combine_row<true>(
      nparts, [&](int i) { return __ldcv(lse_accum + (int64_t)i * rows + r); },
      [&](int i) { return o_accum + ((int64_t)i * rows + r) * 512; }, s_weights + warp * nparts, out + r * o_stride_row,
      lse + r);
}

__device__ int g_merge_status = 0;

cudaError_t set_status_mirror_merge(int* mapped_host_word) { return tc::set_status_mirror(mapped_host_word); }

// The merge kernels keep one weight per (warp, part) in dynamic shared memory; above 48 KB the limit of the
// kernel has to be raised first.
template <class Kernel>
static cudaError_t allow_dynamic_smem(Kernel kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

cudaError_t launch_decode_combine_push(const DecodeKernelParams& p, cudaStream_t stream) {
  const int rows = p.h_k * p.s_q * p.hq_per_hk;
  dim3 grid(p.b, (rows + kCombineWarps - 1) / kCombineWarps);
  const size_t smem = sizeof(float) * kCombineWarps * p.num_sm_parts;
  if (cudaError_t e = allow_dynamic_smem(decode_combine_push_kernel, smem); e != cudaSuccess) return e;
  decode_combine_push_kernel<<<grid, kCombineWarps * 32, smem, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_merge_peer_partials(const float* lse_accum, const float* o_accum, int num_parts, int rows, void* out,
                                       int64_t o_stride_row, float* lse, const unsigned int* flags, unsigned int epoch,
                                       int max_polls, cudaStream_t stream) {
  int* status = nullptr;
  cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&status), g_merge_status);
  if (e != cudaSuccess) return e;
  const size_t smem = sizeof(float) * kCombineWarps * num_parts;
  e = allow_dynamic_smem(merge_peer_partials_kernel, smem);
  if (e != cudaSuccess) return e;
  merge_peer_partials_kernel<<<(rows + kCombineWarps - 1) / kCombineWarps, kCombineWarps * 32, smem, stream>>>(
      lse_accum, o_accum, num_parts, rows, reinterpret_cast<__nv_bfloat16*>(out), o_stride_row, lse, flags, epoch, max_polls,
      status);
  return cudaGetLastError();
}

cudaError_t read_merge_status(int* host_status, bool reset) {
  cudaError_t e = cudaMemcpyFromSymbol(host_status, g_merge_status, sizeof(int));
  if (e != cudaSuccess) return e;
  if (reset && *host_status != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_merge_status, &zero, sizeof(int));
  }
  return e;
}

template <int WPR, bool SHARED, int PARTS = WPR < 4 ? 1 : 4>
static cudaError_t launch_decode_combine_wpr(const DecodeKernelParams& p, int rows, cudaStream_t stream) {
  constexpr int kWarps = combine_warps(WPR), kRows = kWarps / WPR;
  const size_t smem = sizeof(float) * kWarps * p.num_sm_parts;
  if (cudaError_t e = allow_dynamic_smem(decode_combine_kernel<WPR, SHARED, PARTS>, smem); e != cudaSuccess) return e;
  return launch_dependent(decode_combine_kernel<WPR, SHARED, PARTS>, dim3(p.b, (rows + kRows - 1) / kRows), kWarps * 32, smem, stream, p);
}

cudaError_t launch_decode_combine(const DecodeKernelParams& p, cudaStream_t stream) {
  const int rows = p.h_k * p.s_q * p.hq_per_hk;
  int dev = 0, sms = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  if (cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); e != cudaSuccess) return e;
  // Few rows with many parts each (4 requests x 16 heads split 37 ways): one warp per row walks its parts one after the
  // other on a handful of SMs, so a row is spread over four warps as long as that fits on the chip at once
  // (64 warps per SM); beyond that the rows alone fill it and four times the CTAs would only cost their launch.  Device time
  // of decode steps, 24 shapes each with 16 / 32 / 64 heads and 48 with 128: one warp always 2.7 / 4.8 / 4.8 / 0 % more than
  // this rule, four always 0 / 0 / 0.8 / 3 % more.
  // Where rows of the schedule may be shared a request has more parts still: while eight rows of the schedule and more fall on a request,
  // 16 warps per row as long as they fill half of the chip at most, or 8.  At most four -> this rule: 16 heads, 4 x 1 024 tokens
  // 17.5 -> 13.4 us, 16 x 1 000 17.2 -> 15.4; 64 heads, 1 x 8 000 30.0 -> 21.7, 8 x 3 000 26.2 -> 23.3, 12 x 600 19.6 -> 19.2.  16 warps on more than half of
  // the chip: 8 x 3 000 25.1, 8 x 400 (few parts) 21.7 -> 23.0.  With the line at 32 rows of the schedule 16 x 1 000 stays at 17.2.
  const int64_t all = (int64_t)p.b * rows, room = (int64_t)sms * 64;
  if (!p.sub_split) return all * 4 <= room ? launch_decode_combine_wpr<4, false>(p, rows, stream) : launch_decode_combine_wpr<1, false>(p, rows, stream);
  const bool many = p.num_sm_parts >= 8 * p.b;
  // Parts in flight: the most with which all CTAs are resident, by their registers: eight with one CTA of 16 warps (88 registers) or three of
  // eight (80) per SM, six with four of eight (62), or four.  Four / six / eight: 64 heads, 1 x 8 000 19.2 / 19.4 / 18.3 us; 16 heads,
  // 16 x 1 000 (256 CTAs of 16 warps) 12.1 / 12.5 / 14.0; 32 heads, 10 x 800 (320 of eight) 13.6 / 13.6 / 12.7; 64 heads, 9 x 900 (576)
  // 16.2 / 15.8 / 17.4; sparse, 5 requests of two tokens (640) 15.6 / 16.3 / 17.0.
  if (many && all * 32 <= room) return all <= sms ? launch_decode_combine_wpr<16, true, 8>(p, rows, stream) : launch_decode_combine_wpr<16, true>(p, rows, stream);
  if (many && all * 8 <= room) {
    if (all <= 3 * sms) return launch_decode_combine_wpr<8, true, 8>(p, rows, stream);
    return all <= 4 * sms ? launch_decode_combine_wpr<8, true, 6>(p, rows, stream) : launch_decode_combine_wpr<8, true>(p, rows, stream);
  }
  return all * 4 <= room ? launch_decode_combine_wpr<4, true>(p, rows, stream) : launch_decode_combine_wpr<1, true>(p, rows, stream);
}

template <int WPR>
static cudaError_t launch_sparse_prefill_combine_wpr(const SparsePrefillKernelParams& sp, cudaStream_t stream) {
  return launch_dependent(sparse_prefill_combine_kernel<WPR>, dim3(sp.s_q - sp.whole, sp.h_q / (kCombineWarps / WPR)), kCombineWarps * 32,
                          sizeof(float) * kCombineWarps * sp.per, stream, sp);
}

cudaError_t launch_sparse_prefill_combine(const SparsePrefillKernelParams& sp, cudaStream_t stream) {
  int dev = 0, sms = 0;
  if (cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
  if (cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); e != cudaSuccess) return e;
  if ((int64_t)(sp.s_q - sp.whole) * sp.h_q * 4 <= (int64_t)sms * 64) return launch_sparse_prefill_combine_wpr<4>(sp, stream);      // as in launch_decode_combine
  return launch_sparse_prefill_combine_wpr<1>(sp, stream);
}

cudaError_t launch_combine_partials(const float* lse_accum, const float* o_accum, int num_parts, int rows, void* out,
                                    int64_t o_stride_row, float* lse, cudaStream_t stream) {
  const size_t smem = sizeof(float) * kCombineWarps * num_parts;
  if (cudaError_t e = allow_dynamic_smem(combine_partials_kernel, smem); e != cudaSuccess) return e;
  combine_partials_kernel<<<(rows + kCombineWarps - 1) / kCombineWarps, kCombineWarps * 32, smem, stream>>>(
      lse_accum, o_accum, num_parts, rows, reinterpret_cast<__nv_bfloat16*>(out), o_stride_row, lse);
  return cudaGetLastError();
}

}  // namespace fmla
