// Which kernel runs an MLA attention call: the CTA pair (mla_pair.cu) where 128 heads share a kv head, or the 64 heads of two
// query tokens -- its two CTAs read every cached token once for all of them.  Otherwise one CTA per 64 heads (mla_tile64.cu) for
// the sparse prefill and where several such tiles of a dense decode read the same pages, or per at most 64 query rows
// (mla_few_rows.cu).
#include "kernels.h"

#include <cstdlib>

namespace fmla {

// FMLA_DISABLE_PAIR=1 in the environment keeps the one-CTA kernels for every shape (A/B runs)
static bool pair_kernel_enabled() {
  static const bool on = [] {
    const char* v = getenv("FMLA_DISABLE_PAIR");
    return !(v && v[0] == '1');
  }();
  return on;
}

bool decode_dense_merges_in_kernel(const DecodeKernelParams& p) {
  return p.topk < 0 && decode_dense_pair_applies(p) && pair_kernel_enabled() && p.arrival_counters != nullptr && !p.force_partial;
}

cudaError_t launch_decode_dense_tc(const DecodeKernelParams& p, cudaStream_t stream) {
  if (decode_dense_pair_applies(p) && pair_kernel_enabled()) return launch_decode_dense_pair(p, stream);
  if (decode_dense_tile64_applies(p)) return launch_decode_dense_tile64(p, stream);
  return launch_decode_few_rows(p, stream);
}

cudaError_t launch_decode_sparse_tc(const DecodeKernelParams& p, cudaStream_t stream) {
  if (decode_sparse_pair_applies(p) && pair_kernel_enabled()) return launch_decode_sparse_pair(p, stream);
  return launch_decode_sparse_few_rows(p, stream);
}

cudaError_t launch_sparse_prefill_tc(const SparsePrefillKernelParams& sp, cudaStream_t stream) {
  if (sparse_prefill_pair_applies(sp) && pair_kernel_enabled()) return launch_sparse_prefill_pair(sp, stream);
  return launch_sparse_prefill_64(sp, stream);
}

}  // namespace fmla
