// Split-KV tile scheduler: cuts the (request, 64-token block) work list of a decode batch into num_sm_parts
// contiguous partitions.
//
// Output contract of csrc/smxx/get_mla_metadata.cu:8-89 of the reference (rows [begin_idx, begin_block,
// end_idx inclusive, end_block exclusive, begin_n_split_idx, 0, 0, 0]; num_splits = exclusive prefix of the number
// of partitions that touch each request), computed differently: the reference walks the partitions one after
// the other on a single thread; here every cut is a closed-form position on the line of request costs, found
// by a binary search over the cost prefix sums, so all partitions are computed in parallel by one thread
// block (a few microseconds for any batch size).
//
//   cost of a request = its block count (a zero-length request counts one block) + a fixed overhead of 5,
//                       laid out on a line as [overhead | blocks]
//   cut k             = k * pitch on that line; pitch = ceil(total / parts) when there are more requests than
//                       parts (a partition then carries at most pitch + one overhead, the bound of the
//                       reference's greedy walk), ceil(total / parts) + overhead otherwise (the slack lets a
//                       batch of similar requests fall one request per partition instead of being cut everywhere)
//   a cut inside an overhead stretch moves to the start of that request
//   partition k       = everything between cuts k and k+1; equal cuts give an empty partition (begin_idx = batch)
// The integer statement of the same algorithm, against which the kernel is checked bit for bit, is
// oracle/scheduler.py:schedule_cut_ref.
#include "fmla_common.cuh"
#include "kernels.h"

namespace fmla {

constexpr int kFixedOverheadBlocks = 5;   // csrc/pybind.cpp:308,323,341
constexpr int kBlockN = 64;
constexpr int kSchedThreads = 1024;
constexpr int kMaxParts = 1023;           // one thread per cut
constexpr int kSharedBatch = 4096;        // 16 KB

struct Cut { int req, off; };

// One block of whole warps, at least num_sm_parts + 1 threads.  The kernel is a chain of barriers and of dependent reads (a binary
// search over the prefix sums), nothing else: prefix sums and counts live in shared memory up to kSharedBatch requests, with
// no more warps at the barriers than requests or cuts ask for (4 requests, 148 parts: 4.5 us with 1024 threads and the sums in
// `num_splits`, 3.4 us now).  Larger batches use num_splits ([batch + 1] ints) itself: it is only overwritten with its final
// contents after every cut has been located.
__global__ void __launch_bounds__(kSchedThreads) get_mla_metadata_kernel(const int* __restrict__ seqlens_k, int batch,
                                                                         int num_sm_parts, int topk, int* __restrict__ md,
                                                                         int* num_splits) {
  __shared__ int s_warp[2][kSchedThreads / 32];
  __shared__ int s_work[kSharedBatch + 1];
  __shared__ Cut s_cut[kMaxParts + 2];
  __shared__ unsigned char s_new[kMaxParts + 2];     // cut k differs from cut k-1
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x;
  int* work = batch <= kSharedBatch ? s_work : num_splits;
  pdl_allow_dependents();      // the attention kernel may be set up meanwhile; it waits for this kernel before it reads the schedule
  auto len_of = [&](int i) { return topk == -1 ? __ldg(seqlens_k + i) : topk; };
  auto real_blocks = [&](int i) { const int l = len_of(i); return l == 0 ? 0 : (l + kBlockN - 1) / kBlockN; };
  auto cost_of = [&](int i) { return max(real_blocks(i), 1) + kFixedOverheadBlocks; };

  auto warp_scan = [&](int x) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int add = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += add;
    }
    return x;
  };
  // exclusive scan of `n` values produced by value(i) into dst[0..n] (dst[n] = total), one value per thread at a time; value(i)
  // may read dst[i].  Every warp adds up the warp totals for itself: one barrier per turn.  (Scanned with shuffles by every warp, 32 warps
  // kept each other waiting: 1000 requests, one part 4.0 -> 4.2 us.)
  auto exclusive_scan = [&](int n, auto value, int* dst) {
    int carry = 0, buf = 0;
    for (int base = 0; base < n; base += nthreads, buf ^= 1) {
      const int i = base + tid;
      const int v = i < n ? value(i) : 0;
      const int x = warp_scan(v);
      if (lane == 31) s_warp[buf][warp] = x;
      __syncthreads();
      const int t = lane < (nthreads >> 5) ? s_warp[buf][lane] : 0;
      const int before = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0);
      if (i < n) dst[i] = carry + before + x - v;
      if (warp == 0 || base + nthreads < n) carry += __reduce_add_sync(0xffffffffu, t);
    }
    if (tid == 0) dst[n] = carry;
    __syncthreads();
  };

  // 1. cost prefix sums
  exclusive_scan(batch, cost_of, work);
  const int total = work[batch];
  const int pitch = (total + num_sm_parts - 1) / num_sm_parts + (batch <= num_sm_parts ? kFixedOverheadBlocks : 0);

  // 2. cut k, k = 0 .. parts
  if (tid <= num_sm_parts) {
    Cut c;
    const long long x = static_cast<long long>(tid) * pitch;
    if (tid >= num_sm_parts || x >= total) {
      c.req = batch; c.off = 0;
    } else {
      int lo = 0, hi = batch;                 // last request r with prefix[r] <= x
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (work[mid] <= x) lo = mid; else hi = mid;
      }
      const int off = static_cast<int>(x) - work[lo] - kFixedOverheadBlocks;
      c.req = lo; c.off = off <= 0 ? 0 : off;
      if (c.off >= max(real_blocks(lo), 1)) { c.req = lo + 1; c.off = 0; }      // cannot happen for x < prefix[lo + 1]; kept as a guard
    }
    s_cut[tid] = c;
  }
  __syncthreads();
  if (tid <= num_sm_parts) s_new[tid] = tid == 0 || s_cut[tid].req != s_cut[tid - 1].req || s_cut[tid].off != s_cut[tid - 1].off;
  __syncthreads();

  // 3. every request is touched by one partition plus one per distinct cut strictly inside it
  for (int i = tid; i < batch; i += nthreads) work[i] = 1;
  __syncthreads();
  if (tid >= 1 && tid < num_sm_parts && s_new[tid] && s_cut[tid].off > 0) atomicAdd(work + s_cut[tid].req, 1);
  __syncthreads();

  // 4. metadata rows
  if (tid < num_sm_parts) {
    const Cut a = s_cut[tid], e = s_cut[tid + 1];
    int row[5] = {batch, 0, batch - 1, 0, 0};
    if (a.req != e.req || a.off != e.off) {
      int split = 0;
      if (a.off > 0)
        for (int j = tid; j >= 1 && s_cut[j].req == a.req && s_cut[j].off > 0; --j) split += s_new[j];
      row[0] = a.req; row[1] = a.off; row[4] = split;
      if (e.off > 0) { row[2] = e.req; row[3] = e.off; }
      else { row[2] = e.req - 1; row[3] = real_blocks(e.req - 1); }
    }
    int4* dst = reinterpret_cast<int4*>(md + tid * 8);
    dst[0] = make_int4(row[0], row[1], row[2], row[3]);
    dst[1] = make_int4(row[4], 0, 0, 0);
  }
  __syncthreads();

  // 5. counts -> exclusive prefix
  exclusive_scan(batch, [&](int i) { return work[i]; }, num_splits);
}

cudaError_t launch_get_mla_metadata(const int* seqlens_k, int batch, int num_sm_parts, int topk, int* md,
                                    int* num_splits, cudaStream_t stream) {
  if (num_sm_parts > kMaxParts) return cudaErrorInvalidValue;
  const int want = batch > num_sm_parts ? batch : num_sm_parts + 1;
  const int threads = want >= kSchedThreads ? kSchedThreads : (want + 31) / 32 * 32;
  get_mla_metadata_kernel<<<1, threads, 0, stream>>>(seqlens_k, batch, num_sm_parts, topk, md, num_splits);
  return cudaGetLastError();
}

}  // namespace fmla
