"""The "extension module" the public interface calls: same five functions, same
positional signatures and return conventions as the module csrc/pybind.cpp
builds in the reference (:870-911), implemented as a thin marshalling layer
over the C ABI.  Tensors are allocated with torch (device memory, streams);
everything else happens inside libflashmla_b200.so.  The calls are marshalled
natively (csrc/torch_binding.cpp).
"""
from __future__ import annotations

import os
from typing import List, Optional

import torch

from ._cabi import check, lib, native as _native

__flash_mla_variant__ = lib.fmla_variant().decode()


def _stream(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


# Arrival counters of the in-kernel merge of split requests (fmla_decode_params.arrival_counters): zero on entry,
# left zero by the kernel, so one array per (device, stream) is allocated once and reused -- calls on one stream
# are ordered, calls on different streams get different arrays.
_arrival_counters = {}
_MERGE_IN_KERNEL_DEFAULT = os.environ.get("FMLA_MERGE_IN_KERNEL", "0") == "1"


def _counters_for(t: torch.Tensor, n: int) -> torch.Tensor:
    key = (t.device.index, _stream(t))
    buf = _arrival_counters.get(key)
    if buf is None or buf.numel() < n:
        buf = torch.zeros((max(n, 4096),), dtype=torch.int32, device=t.device)
        _arrival_counters[key] = buf
    return buf


def _require(cond: bool, msg: str) -> None:
    if not cond:
        raise RuntimeError(msg)


def get_mla_decoding_metadata(seqlens_k: torch.Tensor, num_q_tokens_per_head_k: int, h_k: int,
                              h_q: Optional[int] = None, is_fp8_kvcache: bool = False,
                              topk: Optional[int] = None) -> List[torch.Tensor]:
    """csrc/pybind.cpp:383-428.  Returns [tile_scheduler_metadata int32[num_sm_parts, 8], num_splits int32[b+1]]."""
    md, ns, whole = _native.metadata(seqlens_k, num_q_tokens_per_head_k, h_k, h_q, is_fp8_kvcache, topk)
    if whole is not None:
        ns._fmla_no_split, ns._fmla_no_split_version = whole, ns._version
    return [md, ns]


def fwd_kvcache_mla(q: torch.Tensor, kcache: torch.Tensor, head_size_v: int, seqlens_k: torch.Tensor,
                    block_table: torch.Tensor, softmax_scale: float, is_causal: bool,
                    tile_scheduler_metadata: torch.Tensor, num_splits: torch.Tensor, is_fp8: bool = False,
                    indices: Optional[torch.Tensor] = None, profile_events=None,
                    indices_logical: bool = False, merge_in_kernel: Optional[bool] = None) -> List[torch.Tensor]:
    """csrc/pybind.cpp:430-720.  Returns [out [b,s_q,h_q,dv] (q dtype), softmax_lse [b,h_q,s_q] fp32].
    profile_events: optional (begin, end) pair of torch.cuda.Event(enable_timing=True) recorded around the
    attention kernel alone (they must have been recorded once already so that their handles exist).
    merge_in_kernel: dense decode with a multiple of 128 heads per kv head only -- the CTA that delivers the last
    partial of a split request merges it (one kernel per step) instead of a second, dependent-launched merge kernel.
    Default: the environment variable FMLA_MERGE_IN_KERNEL=1, else off (the inline merge stalls the pipeline of the
    merging CTA for longer than the separate kernel takes)."""
    counters = 0
    if merge_in_kernel is None:
        merge_in_kernel = _MERGE_IN_KERNEL_DEFAULT
    if merge_in_kernel and indices is None and q.dim() == 4 and kcache.dim() == 4:
        b, s_q, h_q, _ = q.shape
        if q.is_cuda and (h_q // kcache.shape[2]) % 128 == 0:
            counters = _counters_for(q, b * s_q * (h_q // 64)).data_ptr()
    begin, end = (e.cuda_event for e in profile_events) if profile_events is not None else (0, 0)
    return _native.decode(q, kcache, head_size_v, seqlens_k, block_table, softmax_scale, is_causal,
                          tile_scheduler_metadata, num_splits, is_fp8, indices, begin, end, indices_logical, counters,
                          _no_request_is_split(num_splits))


def _no_request_is_split(num_splits: torch.Tensor) -> bool:
    """True when the schedule is known to give every request to one partition: the merge kernel is then not launched.
    A sparse schedule is a function of numbers the host has (batch, topk, partitions), so get_mla_decoding_metadata
    says so on the tensor it returns.  An in-place write to that tensor withdraws it, and a copy that carries the mark
    (deepcopy, pickle, torch.save) never has its version; a write that torch cannot see (through .data, or by a kernel of
    the caller's) leaves it, and the attention kernel then reports device status 41.  The lengths of a dense batch are on
    the device, and reading the outcome back costs a synchronisation per plan (40 us) against 1 to 3 us of a merge kernel
    that finds nothing to do: it counts as not known."""
    if not getattr(num_splits, "_fmla_no_split", False) or num_splits.is_inference():
        return False
    return getattr(num_splits, "_fmla_no_split_version", None) in (None, num_splits._version)


def sparse_prefill_fwd(q: torch.Tensor, kv: torch.Tensor, indices: torch.Tensor, sm_scale: float,
                       d_v: int = 512) -> List[torch.Tensor]:
    """csrc/pybind.cpp:730-814.  Returns [out bf16 [s_q,h_q,d_v], max_logits fp32 [s_q,h_q], lse fp32 [s_q,h_q]]."""
    return _native.sparse_prefill(q, kv, indices, sm_scale, d_v)


def dense_prefill_fwd(workspace_buffer, q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse,
                      mask_mode_code: int, softmax_scale: float, max_seqlen_q: int, max_seqlen_kv: int,
                      is_varlen: bool = True) -> None:
    """csrc/pybind.cpp:817-839.  Writes o and lse in place.  workspace_buffer is accepted and unused
    (the reference's forward does not use it either, fmha_cutlass_fwd_sm100.cuh:302-306)."""
    _native.dense_fwd(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse, mask_mode_code, softmax_scale,
                      max_seqlen_q, max_seqlen_kv)


def dense_prefill_fwd_new(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, mask_mode_code: int, softmax_scale: float,
                          max_seqlen_q: int, max_seqlen_kv: int) -> List[torch.Tensor]:
    """dense_prefill_fwd into new tensors: [o [total_q, h_q, d_v], lse [total_q, h_q] contiguous along tokens]."""
    return _native.dense_fwd(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, None, None, mask_mode_code, softmax_scale,
                             max_seqlen_q, max_seqlen_kv)


def dense_prefill_bwd(workspace_buffer, d_o, q, k, v, o, lse, cumulative_seqlen_q, cumulative_seqlen_kv,
                      dq, dk, dv, mask_mode_code: int, softmax_scale: float, max_seqlen_q: int,
                      max_seqlen_kv: int, is_varlen: bool = True) -> None:
    """csrc/pybind.cpp:841-867.  Writes dq, dk, dv in place."""
    _native.dense_bwd(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse, mask_mode_code, softmax_scale,
                      max_seqlen_q, max_seqlen_kv, d_o, dq, dk, dv, workspace_buffer)


def dense_prefill_bwd_new(d_o, q, k, v, o, lse, cumulative_seqlen_q, cumulative_seqlen_kv, mask_mode_code: int,
                          softmax_scale: float, max_seqlen_q: int, max_seqlen_kv: int) -> List[torch.Tensor]:
    """dense_prefill_bwd into new tensors, with a workspace of its own: [dq, dk, dv]."""
    return _native.dense_bwd(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse, mask_mode_code, softmax_scale,
                             max_seqlen_q, max_seqlen_kv, d_o, None, None, None, None)


def combine_partials(lse_accum: torch.Tensor, o_accum: torch.Tensor):
    """Merge [num_parts, rows] base-2 LSEs and [num_parts, rows, 512] fp32 partial outputs.
    Returns (out bf16 [rows, 512], lse fp32 [rows] natural log)."""
    _require(lse_accum.is_cuda and o_accum.is_cuda and lse_accum.is_contiguous() and o_accum.is_contiguous(),
             "partials must be contiguous CUDA tensors")
    _require(lse_accum.dtype == torch.float32 and o_accum.dtype == torch.float32, "partials must be float32")
    n, rows = lse_accum.shape
    _require(tuple(o_accum.shape) == (n, rows, 512), "o_accum must be [num_parts, rows, 512]")
    with torch.cuda.device(o_accum.device):
        out = torch.empty((rows, 512), dtype=torch.bfloat16, device=o_accum.device)
        lse = torch.empty((rows,), dtype=torch.float32, device=o_accum.device)
        check(lib.fmla_combine_partials(lse_accum.data_ptr(), o_accum.data_ptr(), n, rows, 512, out.data_ptr(), 512,
                                        lse.data_ptr(), _stream(o_accum)))
    return out, lse


def quantize_kv_fp8(kv: torch.Tensor, cache: Optional[torch.Tensor] = None,
                    dst_slots: Optional[torch.Tensor] = None) -> torch.Tensor:
    """bf16 [n, 576] (or [num_blocks, 64, 1, 576]) -> FP8 records.  Without `cache` a fresh
    [*, 656] float8_e4m3fn tensor of the same leading shape is returned."""
    return _native.quantize(kv, cache, dst_slots)
