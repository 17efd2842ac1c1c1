// Native marshalling of the calls (decode, its split-KV plan, sparse prefill, dense path, FP8 cache writer): torch tensors
// in, one C-ABI call out.  A step of a small batch is bound by what the host does per call -- tensor checks,
// output allocation, filling the parameter block, the launches -- and the same work through Python attribute access and
// ctypes took 38 us of host time per decode call, against 20 to 30 us of GPU work.  (Dense path: 200 tokens, 8 heads 35.5 us
// per forward through ctypes, 18.8 here, 12.3 of GPU work; 3 sequences of 300 to 900 tokens, 16 heads, forward and backward
// 180 to 199 -> 115 us.  With the outputs allocated here too, instead of by torch.empty in Python: 2 sequences of 100 to 200 tokens, 8 heads
// 18.2 -> 16.3 us of host time, with the backward 116 -> 105.)  Everything that computes stays behind the C ABI (include/flashmla_b200.h); error texts are those of
// the extension module of the reference (csrc/pybind.cpp:383-867).
//
// CPython functions with vector calls instead of pybind11: an argument costs a type check and a pointer.
#include "../../include/flashmla_b200.h"

#include <ATen/ATen.h>
#include <c10/core/InferenceMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <Python.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

namespace {

struct PythonErrorSet {};      // thrown where a Python call has failed and set the error

void require(bool cond, const char* msg) {
  if (!cond) throw std::runtime_error(msg);
}
void require_cuda(const at::Tensor& t, const char* name) {
  if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be on CUDA");
}
void check(int status) {
  if (status != FMLA_OK)
    throw std::runtime_error(std::string("flashmla_b200: ") + fmla_status_string(status) + ": " + fmla_last_error_message());
}

const at::Tensor& tensor(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) throw std::runtime_error(std::string(name) + " must be a torch.Tensor");
  return THPVariable_Unpack(o);
}
int64_t integer(PyObject* o) {
  if (!PyLong_Check(o)) {                      // what int() takes: 16.0, a numpy or tensor scalar
    PyObject* whole = PyNumber_Long(o);
    if (!whole) throw PythonErrorSet();
    const int64_t v = PyLong_AsLongLong(whole);
    Py_DECREF(whole);
    if (v == -1 && PyErr_Occurred()) throw PythonErrorSet();
    return v;
  }
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PythonErrorSet();
  return v;
}
int as_int(PyObject* o) {
  const int64_t v = integer(o);
  if (v < INT32_MIN || v > INT32_MAX) throw std::runtime_error("integer argument out of range");
  return static_cast<int>(v);
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PythonErrorSet();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PythonErrorSet();
  return v != 0;
}

at::Tensor new_tensor(at::IntArrayRef shape, const at::Tensor& like, at::ScalarType dtype) {
  return at::empty(shape, at::TensorOptions().dtype(dtype).device(like.device()));
}
void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// Gives up the GIL for the allocations and launches of a call: an allocation may synchronise and a launch waits while the
// stream's queue is full, and what it waits for may be a host callback that needs the GIL.  Python objects are read before,
// and tensors are declared outside its scope (the last reference to one may go through Python).
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

PyObject* pair(at::Tensor a, at::Tensor b) {
  PyObject* list = PyList_New(2);
  PyList_SET_ITEM(list, 0, THPVariable_Wrap(std::move(a)));
  PyList_SET_ITEM(list, 1, THPVariable_Wrap(std::move(b)));
  return list;
}

// Runs `f`, turning a C++ exception into the Python one that torch makes of it: torch.OutOfMemoryError for a failed
// allocation, IndexError and the like for torch's own errors, RuntimeError for the messages above.
template <class F>
PyObject* guarded(Py_ssize_t nargs, Py_ssize_t want, F&& f) {
  if (nargs != want) {
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
    return nullptr;
  }
  try {
    return f();
  } catch (const PythonErrorSet&) {
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}

// Whether the schedule of csrc/scheduler.cu leaves every one of `b` requests of the same length in one partition: all
// cuts fall on request boundaries or into the overhead at the start of a request.  Costs and pitch as stated there.
bool uniform_schedule_splits_nothing(int64_t b, int64_t len, int64_t parts) {
  const int64_t overhead = 5, cost = std::max<int64_t>((len + 63) / 64, 1) + overhead, total = b * cost;
  const int64_t pitch = (total + parts - 1) / parts + (b <= parts ? overhead : 0);
  for (int64_t k = 1; k < parts && k * pitch < total; ++k)
    if (k * pitch % cost > overhead) return false;
  return true;
}

// the same for the test that holds it against the oracle's statement of the schedule: b, len, parts -> bool
PyObject* splits_nothing(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, 3, [&]() -> PyObject* {
    const int64_t b = integer(a[0]), len = integer(a[1]), parts = integer(a[2]);
    require(b > 0 && len >= 0 && parts > 0, "b and parts must be positive, len non-negative");
    return PyBool_FromLong(uniform_schedule_splits_nothing(b, len, parts));
  });
}

// seqlens_k, num_q_tokens_per_head_k, h_k, h_q | None, is_fp8, topk | None -> [metadata, num_splits, no request is split]
// (the last one None where it depends on lengths that only the device has)
PyObject* metadata(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, 6, [&]() -> PyObject* {
    const at::Tensor& lens = tensor(a[0], "seqlens_k");
    const bool sparse = a[5] != Py_None;
    require_cuda(lens, "seqlens_k");
    require(lens.is_contiguous(), "seqlens_k must be contiguous");
    require(lens.scalar_type() == at::kInt, "seqlens_k must have dtype int32");
    if (sparse) require(a[3] != Py_None, "num_heads_q must be provided when topk is provided");
    const int q_per_hk = as_int(a[1]), h_k = as_int(a[2]), h_q = a[3] != Py_None ? as_int(a[3]) : 0;
    const bool fp8 = truth(a[4]);
    const int topk = sparse ? as_int(a[5]) : -1;
    const int64_t b = lens.size(0);
    int parts = 0;
    at::Tensor md, ns;
    {
      const NoGil nogil;
      check(fmla_get_num_sm_parts(lens.get_device(), q_per_hk, h_k, h_q, fp8, sparse, &parts));
      const c10::cuda::CUDAGuard guard(lens.device());
      // ordinary tensors under torch.inference_mode() too: what is known of a plan holds until an in-place write to it, which
      // only their version counter tells
      const c10::InferenceMode ordinary(false);
      md = new_tensor({parts, 8}, lens, at::kInt);
      ns = new_tensor({b + 1}, lens, at::kInt);
      check(fmla_get_mla_metadata(static_cast<const int32_t*>(lens.const_data_ptr()), static_cast<int>(b), parts, topk,
                                  static_cast<int32_t*>(md.mutable_data_ptr()), static_cast<int32_t*>(ns.mutable_data_ptr()),
                                  stream_of(lens)));
    }
    PyObject* list = PyList_New(3);
    PyList_SET_ITEM(list, 0, THPVariable_Wrap(std::move(md)));
    PyList_SET_ITEM(list, 1, THPVariable_Wrap(std::move(ns)));
    PyObject* whole = !sparse ? Py_None : uniform_schedule_splits_nothing(b, topk, parts) ? Py_True : Py_False;
    Py_INCREF(whole);
    PyList_SET_ITEM(list, 2, whole);
    return list;
  });
}

// q, kcache, head_size_v, seqlens_k, block_table, softmax_scale, is_causal, metadata, num_splits, is_fp8, indices | None,
// event begin, event end, indices_logical, address of the arrival counters (0: none), no request is split -> [out, lse]
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, 16, [&]() -> PyObject* {
    const at::Tensor &q = tensor(a[0], "q"), &kc = tensor(a[1], "kcache"), &lens = tensor(a[3], "seqlens_k"),
                     &bt = tensor(a[4], "block_table"), &md = tensor(a[7], "tile_scheduler_metadata"), &ns = tensor(a[8], "num_splits");
    const bool fp8 = truth(a[9]), sparse = a[10] != Py_None;
    const at::Tensor* idx = sparse ? &tensor(a[10], "indices") : nullptr;
    const at::ScalarType qt = q.scalar_type();
    require(qt == at::kBFloat16 || qt == at::kHalf, "q must be bfloat16 or float16");
    if (!fp8) {
      require(kc.scalar_type() == qt, "query and key must have the same dtype");
    } else {
      require(kc.scalar_type() == at::kFloat8_e4m3fn || kc.scalar_type() == at::kChar || kc.scalar_type() == at::kByte,
              "key must have dtype fp8_e4m3fn or int8 or uint8");
    }
    require(lens.scalar_type() == at::kInt, "seqlens_k must have dtype int32");
    require(bt.scalar_type() == at::kInt, "block_table must have dtype torch.int32");
    require(md.scalar_type() == at::kInt, "tile_scheduler_metadata must have dtype int32");
    require(ns.scalar_type() == at::kInt, "num_splits must have dtype int32");
    require(!sparse || idx->scalar_type() == at::kInt, "indices must have dtype int32");
    require_cuda(q, "q");
    require_cuda(kc, "kcache");
    require_cuda(lens, "seqlens_k");
    require_cuda(bt, "block_table");
    require_cuda(md, "tile_scheduler_metadata");
    require_cuda(ns, "num_splits");
    if (sparse) require_cuda(*idx, "indices");
    require(q.dim() == 4 && kc.dim() == 4, "q and kcache must be 4-D");
    require(q.stride(3) == 1, "q must have contiguous last dimension");
    require(kc.stride(3) == 1, "kcache must have contiguous last dimension");
    require(lens.is_contiguous(), "seqlens_k must be contiguous");
    require(bt.stride(-1) == 1, "block_table must have contiguous last dimension");
    require(md.is_contiguous() && ns.is_contiguous(), "tile_scheduler_metadata and num_splits must be contiguous");
    require(!sparse || idx->stride(-1) == 1, "indices must have contiguous last dimension");

    const int64_t b = q.size(0), s_q = q.size(1), h_q = q.size(2), d = q.size(3), h_k = kc.size(2), dv = integer(a[2]);
    require(md.dim() == 2 && md.size(1) == 8, "tile_scheduler_metadata must be [num_sm_parts, 8]");
    require(lens.dim() == 1 && lens.size(0) == b, "seqlens_k must be [batch]");
    require(ns.dim() == 1 && ns.size(0) == b + 1, "num_splits must be [batch + 1]");
    require(bt.dim() == 2 && bt.size(0) == b, "block_table must be [batch, max_blocks]");
    if (fp8) require(kc.size(3) == 656, "FP8 kcache must have 656 bytes per token");
    else require(kc.size(3) == d, "kcache head dim must equal q head dim");
    if (sparse) require(idx->dim() == 3 && idx->size(0) == b && idx->size(1) == s_q, "indices must be [b, s_q, topk]");
    require(!(qt == at::kHalf && (sparse || fp8)),
            "flashmla_b200: unsupported configuration: float16 queries are supported for the dense (float16 cache) decode only");

    // scratch of the split requests: fp32 partial outputs, then their log-sum-exps
    const int64_t parts = md.size(0), rows = (b + parts) * s_q * h_q;
    fmla_decode_params p = {};
    p.b = static_cast<int32_t>(b); p.s_q = static_cast<int32_t>(s_q); p.h_q = static_cast<int32_t>(h_q);
    p.h_k = static_cast<int32_t>(h_k); p.d = static_cast<int32_t>(d); p.d_v = static_cast<int32_t>(dv);
    p.num_blocks = static_cast<int32_t>(kc.size(0)); p.page_block_size = static_cast<int32_t>(kc.size(1));
    p.is_causal = truth(a[6]); p.is_fp8 = fp8; p.topk = sparse ? static_cast<int32_t>(idx->size(2)) : -1;
    p.q_dtype = qt == at::kHalf ? FMLA_DTYPE_FP16 : FMLA_DTYPE_BF16;
    p.softmax_scale = static_cast<float>(real(a[5]));
    p.q = q.const_data_ptr(); p.q_stride_b = q.stride(0); p.q_stride_s = q.stride(1); p.q_stride_h = q.stride(2);
    p.kcache = kc.const_data_ptr();
    p.k_stride_block = kc.stride(0); p.k_stride_row = kc.stride(1); p.k_stride_head = kc.stride(2);
    p.block_table = static_cast<const int32_t*>(bt.const_data_ptr()); p.block_table_stride_b = bt.stride(0);
    p.seqlens_k = static_cast<const int32_t*>(lens.const_data_ptr());
    if (sparse) {
      p.indices = static_cast<const int32_t*>(idx->const_data_ptr());
      p.indices_stride_b = idx->stride(0); p.indices_stride_s = idx->stride(1);
      p.indices_logical = truth(a[13]);
    }
    p.tile_scheduler_metadata = static_cast<const int32_t*>(md.const_data_ptr()); p.num_sm_parts = static_cast<int32_t>(parts);
    p.num_splits = static_cast<const int32_t*>(ns.const_data_ptr());
    p.arrival_counters = reinterpret_cast<int32_t*>(integer(a[14]));
    p.no_split_hint = truth(a[15]);
    p.profile_event_begin = reinterpret_cast<void*>(integer(a[11]));
    p.profile_event_end = reinterpret_cast<void*>(integer(a[12]));
    at::Tensor out, lse, accum;
    {
      const NoGil nogil;
      const c10::cuda::CUDAGuard guard(q.device());
      out = new_tensor({b, s_q, h_q, dv}, q, qt);
      lse = new_tensor({b, h_q, s_q}, q, at::kFloat);
      accum = new_tensor({rows * (dv + 1)}, q, at::kFloat);
      p.out = out.mutable_data_ptr(); p.o_stride_b = out.stride(0); p.o_stride_s = out.stride(1); p.o_stride_h = out.stride(2);
      p.softmax_lse = static_cast<float*>(lse.mutable_data_ptr());
      p.o_accum = static_cast<float*>(accum.mutable_data_ptr()); p.lse_accum = p.o_accum + rows * dv;
      check(fmla_fwd_kvcache_mla(&p, stream_of(q)));
    }
    return pair(std::move(out), std::move(lse));
  });
}

// q, kv, indices, sm_scale, d_v -> [out, max_logits, lse]
PyObject* sparse_prefill(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, 5, [&]() -> PyObject* {
    const at::Tensor &q = tensor(a[0], "q"), &kv = tensor(a[1], "kv"), &idx = tensor(a[2], "indices");
    require_cuda(q, "q");
    require_cuda(kv, "kv");
    require_cuda(idx, "indices");
    require(q.scalar_type() == at::kBFloat16 && kv.scalar_type() == at::kBFloat16, "q and kv must be bfloat16");
    require(idx.scalar_type() == at::kInt, "indices must be int32");
    require(q.dim() == 3 && kv.dim() == 3 && idx.dim() == 3, "q, kv, indices must be 3-D");
    require(q.stride(2) == 1 && kv.stride(2) == 1 && idx.stride(2) == 1, "last dimensions must be contiguous");
    require(kv.size(2) == q.size(2), "q and kv head dims differ");
    require(idx.size(0) == q.size(0) && idx.size(1) == kv.size(1), "indices must be [s_q, h_kv, topk]");
    const int64_t s_q = q.size(0), h_q = q.size(1), dv = integer(a[4]);
    fmla_sparse_prefill_params p = {};
    p.s_q = static_cast<int32_t>(s_q); p.s_kv = static_cast<int32_t>(kv.size(0)); p.h_q = static_cast<int32_t>(h_q);
    p.h_kv = static_cast<int32_t>(kv.size(1)); p.d_qk = static_cast<int32_t>(q.size(2)); p.d_v = static_cast<int32_t>(dv);
    p.topk = static_cast<int32_t>(idx.size(2));
    p.sm_scale = static_cast<float>(real(a[3]));
    p.q = q.const_data_ptr(); p.q_stride_s = q.stride(0); p.q_stride_h = q.stride(1);
    p.kv = kv.const_data_ptr(); p.kv_stride_s = kv.stride(0); p.kv_stride_h = kv.stride(1);
    p.indices = static_cast<const int32_t*>(idx.const_data_ptr()); p.indices_stride_s = idx.stride(0); p.indices_stride_h = idx.stride(1);
    at::Tensor out, mx, lse, scratch;
    {
      const NoGil nogil;
      const c10::cuda::CUDAGuard guard(q.device());
      out = new_tensor({s_q, h_q, dv}, q, at::kBFloat16);
      mx = new_tensor({s_q, h_q}, q, at::kFloat);
      lse = new_tensor({s_q, h_q}, q, at::kFloat);
      p.out = out.mutable_data_ptr();
      p.max_logits = static_cast<float*>(mx.mutable_data_ptr());
      p.lse = static_cast<float*>(lse.mutable_data_ptr());
      size_t bytes = 0;
      check(fmla_sparse_prefill_scratch_bytes(p.s_q, p.h_q, p.topk, &bytes));
      if (bytes > 0) scratch = new_tensor({static_cast<int64_t>(bytes)}, q, at::kByte);
      check(fmla_sparse_prefill_fwd_scratch(&p, bytes > 0 ? scratch.mutable_data_ptr() : nullptr, bytes, stream_of(q)));
    }
    PyObject* list = pair(std::move(out), std::move(mx));
    PyObject* l = THPVariable_Wrap(std::move(lse));
    PyList_Append(list, l);
    Py_DECREF(l);
    return list;
  });
}

// The arguments that both directions of the dense path have: a[0] q, a[1] k, a[2] v, a[3] cu_q, a[4] cu_k, a[5] o, a[6] lse,
// a[7] mask mode code, a[8] softmax scale, a[9] max_seqlen_q, a[10] max_seqlen_k.
constexpr Py_ssize_t kDenseArgs = 11;
// all but o and lse, whose tensors follow (`given`: the caller's, which are looked at first as the others are)
fmla_dense_params dense_params(PyObject* const* a, bool given) {
  const char* names[] = {"q", "k", "v", "cumulative_seqlen_q", "cumulative_seqlen_kv", "o", "lse"};
  for (int i = 0; i < (given ? 7 : 5); ++i) require_cuda(tensor(a[i], names[i]), names[i]);
  const at::Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]), &cu_q = THPVariable_Unpack(a[3]),
                   &cu_k = THPVariable_Unpack(a[4]);
  const at::Tensor *o = given ? &THPVariable_Unpack(a[5]) : nullptr, *lse = given ? &THPVariable_Unpack(a[6]) : nullptr;
  require(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16 && (!o || o->scalar_type() == at::kBFloat16),
          "q, k, v, o must be bfloat16");
  require(!lse || lse->scalar_type() == at::kFloat, "lse must be float32");
  require(cu_q.scalar_type() == at::kInt && cu_k.scalar_type() == at::kInt, "cumulative seqlens must be int32");
  require(q.dim() == 3 && k.dim() == 3 && v.dim() == 3 && (!o || (o->dim() == 3 && lse->dim() == 2)), "bad ranks");
  require(q.stride(2) == 1 && k.stride(2) == 1 && v.stride(2) == 1 && (!o || o->stride(2) == 1), "last dimensions must be contiguous");
  require(cu_q.is_contiguous() && cu_k.is_contiguous(), "cumulative seqlens must be contiguous");
  fmla_dense_params p = {};
  p.batch = static_cast<int32_t>(cu_q.size(0) - 1);
  require(cu_k.numel() >= cu_q.size(0), "cumulative_seqlen_kv is shorter than cumulative_seqlen_q");      // the kernels read as many of both
  require(k.size(0) == v.size(0) && k.size(1) == v.size(1) && k.size(2) == q.size(2), "k shape mismatch");
  if (given) {
    require(o->size(0) == q.size(0) && o->size(1) == q.size(1) && o->size(2) == v.size(2), "o shape mismatch");
    require(lse->size(0) == q.size(0) && lse->size(1) == q.size(1), "lse must be [total_q, h_q]");
  }
  p.total_q = static_cast<int32_t>(q.size(0)); p.h_q = static_cast<int32_t>(q.size(1)); p.d_qk = static_cast<int32_t>(q.size(2));
  p.total_k = static_cast<int32_t>(v.size(0)); p.h_k = static_cast<int32_t>(v.size(1)); p.d_v = static_cast<int32_t>(v.size(2));
  p.max_seqlen_q = as_int(a[9]); p.max_seqlen_k = as_int(a[10]);
  PyObject* one = PyLong_FromLong(1);
  const int causal = PyObject_RichCompareBool(a[7], one, Py_EQ);
  Py_DECREF(one);
  if (causal < 0) throw PythonErrorSet();
  p.is_causal = causal;
  p.softmax_scale = static_cast<float>(real(a[8]));
  p.q = q.const_data_ptr(); p.q_stride_t = q.stride(0); p.q_stride_h = q.stride(1);
  p.k = k.const_data_ptr(); p.k_stride_t = k.stride(0); p.k_stride_h = k.stride(1);
  p.v = v.const_data_ptr(); p.v_stride_t = v.stride(0); p.v_stride_h = v.stride(1);
  p.cu_seqlens_q = static_cast<const int32_t*>(cu_q.const_data_ptr());
  p.cu_seqlens_k = static_cast<const int32_t*>(cu_k.const_data_ptr());
  return p;
}
void dense_output_strides(fmla_dense_params& p, const at::Tensor& o, const at::Tensor& lse) {
  p.o_stride_t = o.stride(0); p.o_stride_h = o.stride(1);
  p.lse_stride_t = lse.stride(0); p.lse_stride_h = lse.stride(1);
}

// the arguments above; writes o and lse, or returns new ones ([total_q, h_q, d_v], and [total_q, h_q] contiguous along tokens) where both
// are None
PyObject* dense_fwd(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, kDenseArgs, [&]() -> PyObject* {
    const bool given = a[5] != Py_None || a[6] != Py_None;
    fmla_dense_params p = dense_params(a, given);
    const at::Tensor& q = THPVariable_Unpack(a[0]);
    at::Tensor o, lse;
    if (given) {
      o = THPVariable_Unpack(a[5]);
      lse = THPVariable_Unpack(a[6]);
    }
    {
      const NoGil nogil;
      const c10::cuda::CUDAGuard guard(q.device());
      if (!given) {
        o = new_tensor({p.total_q, p.h_q, p.d_v}, q, at::kBFloat16);
        lse = new_tensor({p.h_q, p.total_q}, q, at::kFloat).t();
      }
      p.o = o.mutable_data_ptr();
      p.lse = static_cast<float*>(lse.mutable_data_ptr());
      dense_output_strides(p, o, lse);
      check(fmla_dense_prefill_fwd(&p, stream_of(q)));
    }
    if (given) Py_RETURN_NONE;
    return pair(std::move(o), std::move(lse));
  });
}

// the arguments above, then d_o, dq, dk, dv, workspace; writes dq, dk, dv, or returns new ones where all four are None
PyObject* dense_bwd(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, kDenseArgs + 5, [&]() -> PyObject* {
    fmla_dense_params p = dense_params(a, true);
    const char* names[] = {"d_o", "dq", "dk", "dv", "workspace_buffer"};
    const bool given = a[12] != Py_None || a[13] != Py_None || a[14] != Py_None || a[15] != Py_None;
    for (int i = 0; i < (given ? 5 : 1); ++i) {
      const at::Tensor& t = tensor(a[kDenseArgs + i], names[i]);
      require_cuda(t, names[i]);
      if (t.stride(-1) != 1) throw std::runtime_error(std::string(names[i]) + " must have contiguous last dimension");
    }
    const at::Tensor &q = THPVariable_Unpack(a[0]), &k = THPVariable_Unpack(a[1]), &v = THPVariable_Unpack(a[2]), &o = THPVariable_Unpack(a[5]),
                     &lse = THPVariable_Unpack(a[6]), &d_o = THPVariable_Unpack(a[11]);
    at::Tensor dq, dk, dv, work;
    if (given) {
      dq = THPVariable_Unpack(a[12]); dk = THPVariable_Unpack(a[13]); dv = THPVariable_Unpack(a[14]); work = THPVariable_Unpack(a[15]);
    }
    require(d_o.scalar_type() == at::kBFloat16 && (!given || (dq.scalar_type() == at::kBFloat16 && dk.scalar_type() == at::kBFloat16 &&
                                                              dv.scalar_type() == at::kBFloat16)),
            "d_o, dq, dk, dv must be bfloat16");
    require(d_o.sizes() == o.sizes() && (!given || (dq.sizes() == q.sizes() && dk.sizes() == k.sizes() && dv.sizes() == v.sizes())), "gradient shape mismatch");
    p.o = const_cast<void*>(o.const_data_ptr());               // o and lse are read by this direction
    p.lse = const_cast<float*>(static_cast<const float*>(lse.const_data_ptr()));
    dense_output_strides(p, o, lse);
    p.d_o = d_o.const_data_ptr(); p.do_stride_t = d_o.stride(0); p.do_stride_h = d_o.stride(1);
    const size_t need = fmla_dense_bwd_workspace_bytes(p.total_q, p.h_q, p.d_qk);
    {
      const NoGil nogil;
      const c10::cuda::CUDAGuard guard(q.device());
      if (!given) {
        dq = new_tensor(q.sizes(), q, at::kBFloat16);
        dk = new_tensor(k.sizes(), q, at::kBFloat16);
        dv = new_tensor(v.sizes(), q, at::kBFloat16);
        work = new_tensor({static_cast<int64_t>(need)}, q, at::kByte);
      }
      p.dq = dq.mutable_data_ptr(); p.dq_stride_t = dq.stride(0); p.dq_stride_h = dq.stride(1);
      p.dk = dk.mutable_data_ptr(); p.dk_stride_t = dk.stride(0); p.dk_stride_h = dk.stride(1);
      p.dv = dv.mutable_data_ptr(); p.dv_stride_t = dv.stride(0); p.dv_stride_h = dv.stride(1);
      p.workspace_bytes = work.numel() * work.element_size();
      if (p.workspace_bytes < need) throw std::runtime_error("workspace_buffer too small: need " + std::to_string(need) + " bytes");
      p.workspace = work.mutable_data_ptr();
      check(fmla_dense_prefill_bwd(&p, stream_of(q)));
    }
    if (given) Py_RETURN_NONE;
    PyObject* list = pair(std::move(dq), std::move(dk));
    PyObject* third = THPVariable_Wrap(std::move(dv));
    PyList_Append(list, third);
    Py_DECREF(third);
    return list;
  });
}

// kv [..., 576], cache | None, slots | None -> the cache (a fresh [..., 656] one where none is given)
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  return guarded(nargs, 3, [&]() -> PyObject* {
    const at::Tensor& kv = tensor(a[0], "kv");
    require(kv.is_cuda() && kv.scalar_type() == at::kBFloat16 && kv.dim() > 0 && kv.size(-1) == 576, "kv must be CUDA bf16 [..., 576]");
    const at::Tensor* given = a[1] != Py_None ? &tensor(a[1], "cache") : nullptr;
    const int32_t* slots = nullptr;
    if (a[2] != Py_None) {
      const at::Tensor& s = tensor(a[2], "dst_slots");
      require(s.is_cuda() && s.scalar_type() == at::kInt && s.is_contiguous(), "dst_slots must be a contiguous CUDA int32 tensor");
      slots = static_cast<const int32_t*>(s.const_data_ptr());
    }
    at::Tensor flat, cache, records;
    {
      const NoGil nogil;
      flat = kv.dim() == 2 ? kv : kv.reshape({-1, 576});
      require(flat.stride(1) == 1, "kv rows must be contiguous");
      const c10::cuda::CUDAGuard guard(kv.device());
      if (!given) {
        std::vector<int64_t> shape(kv.sizes().begin(), kv.sizes().end());
        shape.back() = 656;
        cache = new_tensor(shape, kv, at::kFloat8_e4m3fn);
      } else {
        cache = *given;
      }
      const bool plain = cache.element_size() == 1 && cache.is_contiguous() && cache.dim() > 0 && cache.size(-1) == 656;
      records = plain ? cache : cache.view(at::kByte).reshape({-1, 656});
      check(fmla_quantize_kv_fp8(flat.const_data_ptr(), flat.stride(0), static_cast<int>(flat.size(0)), slots, records.mutable_data_ptr(),
                                 plain ? 656 : records.stride(0), stream_of(kv)));
    }
    if (a[1] == Py_None) return THPVariable_Wrap(std::move(cache));
    Py_INCREF(a[1]);
    return a[1];
  });
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F));
}
PyMethodDef methods[] = {{"metadata", fast<metadata>(), METH_FASTCALL, nullptr},
                         {"splits_nothing", fast<splits_nothing>(), METH_FASTCALL, nullptr},
                         {"decode", fast<decode>(), METH_FASTCALL, nullptr},
                         {"sparse_prefill", fast<sparse_prefill>(), METH_FASTCALL, nullptr},
                         {"dense_fwd", fast<dense_fwd>(), METH_FASTCALL, nullptr},
                         {"dense_bwd", fast<dense_bwd>(), METH_FASTCALL, nullptr},
                         {"quantize", fast<quantize>(), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fmla_torch", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__fmla_torch() { return PyModule_Create(&module); }
