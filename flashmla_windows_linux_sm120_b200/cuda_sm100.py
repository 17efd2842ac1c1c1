"""The "extension module" the public interface calls: same five functions, same
positional signatures and return conventions as the module csrc/pybind.cpp
builds in the reference (:870-911), implemented as a thin marshalling layer
over the C ABI.  Tensors are allocated with torch (device memory, streams);
everything else happens inside libflashmla_b200.so.  The calls of a decode step
are marshalled natively (csrc/torch_binding.cpp), the dense ones here.
"""
from __future__ import annotations

import ctypes as C
import os
from typing import List, Optional

import torch

from . import _cabi
from ._cabi import DenseParams, check, lib, native as _native

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


def _cuda(t: torch.Tensor, name: str) -> None:
    _require(t.is_cuda, f"{name} must be on CUDA")


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


def _dense_params(q, k, v, cu_q, cu_k, o, lse, mask_mode_code, softmax_scale, max_q, max_k) -> DenseParams:
    for t, n in ((q, "q"), (k, "k"), (v, "v"), (cu_q, "cumulative_seqlen_q"), (cu_k, "cumulative_seqlen_kv"),
                 (o, "o"), (lse, "lse")):
        _cuda(t, n)
    _require(q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16 and v.dtype == torch.bfloat16 and
             o.dtype == torch.bfloat16, "q, k, v, o must be bfloat16")
    _require(lse.dtype == torch.float32, "lse must be float32")
    _require(cu_q.dtype == torch.int32 and cu_k.dtype == torch.int32, "cumulative seqlens must be int32")
    _require(q.dim() == 3 and k.dim() == 3 and v.dim() == 3 and o.dim() == 3 and lse.dim() == 2, "bad ranks")
    _require(q.stride(-1) == 1 and k.stride(-1) == 1 and v.stride(-1) == 1 and o.stride(-1) == 1,
             "last dimensions must be contiguous")
    _require(cu_q.is_contiguous() and cu_k.is_contiguous(), "cumulative seqlens must be contiguous")
    p = DenseParams()
    p.batch = cu_q.shape[0] - 1
    p.total_q, p.h_q, p.d_qk = q.shape
    p.total_k, p.h_k, p.d_v = v.shape
    _require(k.shape[0] == v.shape[0] and k.shape[1] == v.shape[1] and k.shape[2] == q.shape[2], "k shape mismatch")
    _require(tuple(o.shape) == (q.shape[0], q.shape[1], v.shape[2]), "o shape mismatch")
    _require(tuple(lse.shape) == (q.shape[0], q.shape[1]), "lse must be [total_q, h_q]")
    p.max_seqlen_q, p.max_seqlen_k = int(max_q), int(max_k)
    p.is_causal = 1 if mask_mode_code == 1 else 0
    p.softmax_scale = float(softmax_scale)
    p.q, p.q_stride_t, p.q_stride_h = q.data_ptr(), q.stride(0), q.stride(1)
    p.k, p.k_stride_t, p.k_stride_h = k.data_ptr(), k.stride(0), k.stride(1)
    p.v, p.v_stride_t, p.v_stride_h = v.data_ptr(), v.stride(0), v.stride(1)
    p.cu_seqlens_q, p.cu_seqlens_k = cu_q.data_ptr(), cu_k.data_ptr()
    p.o, p.o_stride_t, p.o_stride_h = o.data_ptr(), o.stride(0), o.stride(1)
    p.lse, p.lse_stride_t, p.lse_stride_h = lse.data_ptr(), lse.stride(0), lse.stride(1)
    return p


def dense_prefill_fwd(workspace_buffer, q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse,
                      mask_mode_code: int, softmax_scale: float, max_seqlen_q: int, max_seqlen_kv: int,
                      is_varlen: bool = True) -> None:
    """csrc/pybind.cpp:817-839.  Writes o and lse in place.  workspace_buffer is accepted and unused
    (the reference's forward does not use it either, fmha_cutlass_fwd_sm100.cuh:302-306)."""
    p = _dense_params(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse, mask_mode_code, softmax_scale,
                      max_seqlen_q, max_seqlen_kv)
    with torch.cuda.device(q.device):
        check(lib.fmla_dense_prefill_fwd(C.byref(p), _stream(q)))


def dense_prefill_bwd(workspace_buffer, d_o, q, k, v, o, lse, cumulative_seqlen_q, cumulative_seqlen_kv,
                      dq, dk, dv, mask_mode_code: int, softmax_scale: float, max_seqlen_q: int,
                      max_seqlen_kv: int, is_varlen: bool = True) -> None:
    """csrc/pybind.cpp:841-867.  Writes dq, dk, dv in place."""
    p = _dense_params(q, k, v, cumulative_seqlen_q, cumulative_seqlen_kv, o, lse, mask_mode_code, softmax_scale,
                      max_seqlen_q, max_seqlen_kv)
    for t, n in ((d_o, "d_o"), (dq, "dq"), (dk, "dk"), (dv, "dv"), (workspace_buffer, "workspace_buffer")):
        _cuda(t, n)
        _require(t.stride(-1) == 1, f"{n} must have contiguous last dimension")
    _require(all(t.dtype == torch.bfloat16 for t in (d_o, dq, dk, dv)), "d_o, dq, dk, dv must be bfloat16")
    _require(tuple(d_o.shape) == tuple(o.shape) and tuple(dq.shape) == tuple(q.shape) and
             tuple(dk.shape) == tuple(k.shape) and tuple(dv.shape) == tuple(v.shape), "gradient shape mismatch")
    p.d_o, p.do_stride_t, p.do_stride_h = d_o.data_ptr(), d_o.stride(0), d_o.stride(1)
    p.dq, p.dq_stride_t, p.dq_stride_h = dq.data_ptr(), dq.stride(0), dq.stride(1)
    p.dk, p.dk_stride_t, p.dk_stride_h = dk.data_ptr(), dk.stride(0), dk.stride(1)
    p.dv, p.dv_stride_t, p.dv_stride_h = dv.data_ptr(), dv.stride(0), dv.stride(1)
    need = lib.fmla_dense_bwd_workspace_bytes(p.total_q, p.h_q, p.d_qk)
    _require(workspace_buffer.numel() * workspace_buffer.element_size() >= need,
             f"workspace_buffer too small: need {need} bytes")
    p.workspace, p.workspace_bytes = workspace_buffer.data_ptr(), workspace_buffer.numel() * workspace_buffer.element_size()
    with torch.cuda.device(q.device):
        check(lib.fmla_dense_prefill_bwd(C.byref(p), _stream(q)))


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
