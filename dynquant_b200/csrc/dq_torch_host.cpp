// The host path of the Python entry points, in one C call each: dynquant_b200._host.
//
// A decode call is a few microseconds of GPU work, so what a user waits for is the host: building
// QuantTensor views, ctypes structures and geometry objects in Python took 14 us (one linear
// module), 69 us (a fused layer of three shards), 50 us (an embedding lookup: three gathers and a
// dequant).  Here the tensors' pointers and sizes go straight into the C ABI's descriptors.
//
// Every function returns None for whatever it does not take -- odd shapes or types, tensor
// subclasses, tracing, dispatch modes, autograd in either direction -- and the Python code that calls it then goes its
// long way, where all checks and messages live.  Called through the vectorcall protocol
// (METH_FASTCALL); the GIL is released around the allocation and the launch.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <optional>

#include "dynquant_b200.h"

namespace {

constexpr int kMaxShards = 16;

// One shard of a (fused) layer: where its words and scales start in the flat buffers.
// Field for field what FusedPackedGeometry packs into its `table` (plugin.py).
struct Shard {
  int64_t rows, words_per_row, num_groups, group_values, in_features, word_offset, scale_offset, bits;
};

int tag_of(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return DQ_F16;
    case at::kBFloat16: return DQ_BF16;
    case at::kFloat: return DQ_F32;
    default: return -1;
  }
}

// Nothing that watches or rewrites operator calls is active on this thread.
bool plain_context() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() && at::impl::PythonTorchFunctionTLS::stack_len() == 0 &&
         !torch::jit::tracer::isTracing();
}

const at::Tensor* tensor(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.unsafeGetTensorImpl()->is_python_dispatch() || !t.has_storage()) return nullptr;
  if (t.is_neg() || t._fw_grad(0).defined()) return nullptr;  // (a lazy negation; a forward-mode tangent)
  return &t;
}

const at::Tensor* activation(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor* t = tensor(o);
  if (t == nullptr || t->dim() < 1 || tag_of(t->scalar_type()) < 0) return nullptr;
  return (t->requires_grad() && at::GradMode::is_enabled()) ? nullptr : t;
}

// packed / scales / offsets of one descriptor, as the kernels need them.
bool packed_buffers(const at::Tensor* q, const at::Tensor* s, PyObject* offsets, const at::Tensor** o) {
  if (q == nullptr || s == nullptr || q->scalar_type() != at::kInt || tag_of(s->scalar_type()) < 0 || !q->is_contiguous() ||
      !s->is_contiguous() || s->device() != q->device()) {
    return false;
  }
  *o = nullptr;
  if (offsets == Py_None) return true;
  *o = tensor(offsets);
  return *o != nullptr && (*o)->scalar_type() == s->scalar_type() && (*o)->sizes() == s->sizes() && (*o)->is_contiguous() &&
         (*o)->device() == q->device();
}

// The geometry of a row: dynquant_b200/format.py::row_geometry.
bool row_shape(int64_t bits, int64_t group_size, int64_t in_features, int64_t* group_values, int64_t* groups, int64_t* words) {
  if (!(bits == 2 || bits == 3 || bits == 4 || bits == 8) || in_features <= 0) return false;
  if (group_size == -1) {
    *group_values = in_features, *groups = 1, *words = (in_features * bits + 31) / 32;
    return true;
  }
  if (group_size <= 0 || group_size % 32 != 0) return false;
  *group_values = group_size;
  *groups = (in_features + group_size - 1) / group_size;
  *words = *groups * (group_size * bits / 32);
  return true;
}

dq_weight weight_of(const at::Tensor& q, const at::Tensor& s, const at::Tensor* o, const Shard& p) {
  dq_weight w = {};
  const int64_t meta = p.scale_offset * s.element_size();
  w.packed = static_cast<const char*>(q.const_data_ptr()) + p.word_offset * 4;
  w.scales = static_cast<const char*>(s.const_data_ptr()) + meta;
  w.offsets = o == nullptr ? nullptr : static_cast<const char*>(o->const_data_ptr()) + meta;
  w.rows = p.rows;
  w.words_per_row = p.words_per_row;
  w.num_groups = p.num_groups;
  w.group_values = p.group_values;
  w.in_features = p.in_features;
  w.bits = static_cast<int32_t>(p.bits);
  w.meta_dtype = tag_of(s.scalar_type());
  return w;
}

// The descriptor of one 2-D packed matrix.
bool matrix_of(PyObject* qo, PyObject* so, PyObject* oo, PyObject* bits, PyObject* group, PyObject* k, const at::Tensor** q,
               const at::Tensor** s, dq_weight* w) {
  *q = tensor(qo), *s = tensor(so);
  const at::Tensor* o = nullptr;
  if (!packed_buffers(*q, *s, oo, &o) || (*q)->dim() != 2 || (*s)->dim() != 2) return false;
  Shard p = {};
  p.bits = PyLong_AsLongLong(bits);
  p.in_features = PyLong_AsLongLong(k);
  const int64_t group_size = PyLong_AsLongLong(group);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  if (!row_shape(p.bits, group_size, p.in_features, &p.group_values, &p.num_groups, &p.words_per_row)) return false;
  p.rows = (*q)->size(0);
  if ((*q)->size(1) != p.words_per_row || (*s)->size(0) != p.rows || (*s)->size(1) != p.num_groups) return false;
  *w = weight_of(**q, **s, o, p);
  return true;
}

PyObject* unhandled() { Py_RETURN_NONE; }

at::Tensor new_cuda(at::IntArrayRef sizes, at::ScalarType dtype, at::Device device) {
  return at::Tensor(at::detail::empty_cuda(sizes, dtype, device, std::nullopt));
}

struct LibraryError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
void check(int32_t rc) {
  if (rc != DQ_OK) throw LibraryError(dq_last_error());
}

// Runs `body` without the GIL on `device`; wraps the tensor it returns (undefined: not handled).  What
// the kernels of earlier calls on the device have reported by now is raised first.
template <typename Body>
PyObject* on_device(at::Device device, Body body) {
  try {
    at::Tensor out;
    {
      struct Release {
        PyThreadState* state = PyEval_SaveThread();
        ~Release() { PyEval_RestoreThread(state); }
      } release;
      const c10::cuda::CUDAGuard guard(device);
      check(dq_poll_status(device.index()));
      out = body(at::cuda::getCurrentCUDAStream().stream());
    }
    return out.defined() ? THPVariable_Wrap(std::move(out)) : unhandled();
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// x [.., K] against n shards side by side.
PyObject* multiply(const at::Tensor* x, const dq_weight* w, int n, const at::Tensor& q, PyObject* bias_o) {
  int64_t total = 0;
  for (int i = 0; i < n; ++i) total += w[i].rows;
  const int64_t k = w[0].in_features;
  if (x->device() != q.device() || x->size(-1) != k || x->numel() == 0 || total == 0) return unhandled();
  const int64_t m = x->numel() / k;
  if (m > DQ_GEMV_CHUNKED_MAX_ROWS && at::autocast::is_autocast_enabled(at::kCUDA)) return unhandled();  // (a dense matmul casts)
  const at::Tensor* bias = nullptr;
  if (bias_o != Py_None) {
    bias = tensor(bias_o);
    if (bias == nullptr || bias->dim() != 1 || bias->size(0) != total || bias->device() != q.device() ||
        (bias->requires_grad() && at::GradMode::is_enabled())) {
      return unhandled();
    }
  }
  return on_device(q.device(), [&](cudaStream_t stream) {
    const at::Tensor flat = x->is_contiguous() ? *x : x->contiguous();
    at::Tensor cast;
    if (bias != nullptr) {
      cast = bias->scalar_type() == x->scalar_type() ? *bias : bias->to(x->scalar_type());
      if (!cast.is_contiguous()) cast = cast.contiguous();
    }
    at::DimVector sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = total;
    at::Tensor out = new_cuda(sizes, x->scalar_type(), q.device());
    const int tag = tag_of(x->scalar_type());
    const int32_t rc = dq_matmul_shards(flat.const_data_ptr(), tag, m, w, n, bias == nullptr ? nullptr : cast.const_data_ptr(),
                                        out.data_ptr(), total, tag, stream);
    if (rc == DQ_ERR_UNSUPPORTED && m > DQ_GEMV_CHUNKED_MAX_ROWS) return at::Tensor();
    check(rc);
    return out;
  });
}

// matmul(x, packed, scales, offsets, bits, group_size, in_features, bias)
PyObject* py_matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 8 || !plain_context()) return unhandled();
  const at::Tensor* x = activation(args[0]);
  const at::Tensor *q, *s;
  dq_weight w;
  if (x == nullptr || !matrix_of(args[1], args[2], args[3], args[4], args[5], args[6], &q, &s, &w)) return unhandled();
  return multiply(x, &w, 1, *q, args[7]);
}

// fused(x, qweight, scales, offsets, table, bias): flat buffers, `table` the bytes of a Shard array
PyObject* py_fused(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6 || !plain_context() || !PyBytes_Check(args[4])) return unhandled();
  const at::Tensor* x = activation(args[0]);
  const at::Tensor *q = tensor(args[1]), *s = tensor(args[2]), *o = nullptr;
  const Py_ssize_t bytes = PyBytes_GET_SIZE(args[4]);
  const int count = static_cast<int>(bytes / static_cast<Py_ssize_t>(sizeof(Shard)));
  if (x == nullptr || !packed_buffers(q, s, args[3], &o) || count < 1 || count > kMaxShards ||
      bytes % static_cast<Py_ssize_t>(sizeof(Shard)) != 0) {
    return unhandled();
  }
  std::array<Shard, kMaxShards> table;
  std::memcpy(table.data(), PyBytes_AS_STRING(args[4]), static_cast<size_t>(bytes));
  std::array<dq_weight, kMaxShards> w;
  for (int i = 0; i < count; ++i) {
    const Shard& p = table[i];
    if (p.word_offset + p.rows * p.words_per_row > q->numel() || p.scale_offset + p.rows * p.num_groups > s->numel()) {
      return unhandled();
    }
    w[i] = weight_of(*q, *s, o, p);
  }
  return multiply(x, w.data(), count, *q, args[5]);
}

// A bank of packed rows, 2-D or [experts, rows, cols].
bool bank_of(PyObject* const* args, int64_t bits, int64_t group_size, int64_t k, int64_t rows, const at::Tensor** q, dq_weight* w) {
  *q = tensor(args[0]);
  const at::Tensor *s = tensor(args[1]), *o = nullptr;
  if (!packed_buffers(*q, s, args[2], &o)) return false;
  Shard p = {};
  p.bits = bits, p.in_features = k, p.rows = rows;
  if (!row_shape(bits, group_size, k, &p.group_values, &p.num_groups, &p.words_per_row)) return false;
  if ((*q)->numel() != rows * p.words_per_row || s->numel() != rows * p.num_groups || (*q)->size(-1) != p.words_per_row) return false;
  *w = weight_of(**q, *s, o, p);
  return true;
}

// Whether `tokens` go through dq_moe_gemm: when dq_moe_gemv, which reads an expert's weights once per eight
// of its tokens and call of at most `small` tokens, would make two mean passes over the experts or more --
// one pass of dq_moe_gemm costs about as much (128 experts, top-8: 100 / 128 / 256 tokens 198 / 217 / 437 us
// against 200 / 200 / 205; 8 experts, top-4: 16 / 32 tokens 32 / 50 us against 33 / 34).
bool moe_is_wide(int64_t tokens, int64_t topk, int64_t experts, int64_t small) {
  double passes = 0.0;
  for (int64_t at = 0; at < tokens && passes < 2.0; at += small) {
    const double mean = static_cast<double>(std::min(tokens - at, small) * topk) / static_cast<double>(experts);
    passes += std::max(1.0 - std::exp(-mean), mean > 1.0 ? mean / 8.0 + 0.5 : 0.0);  // (the experts with a token at least)
  }
  return passes >= 1.95;
}

// moe(x, ids, weights, w13 packed, scales, offsets, w2 packed, scales, offsets, (experts, hidden, inter), bits13, bits2, group_size)
PyObject* py_moe(PyObject*, PyObject* const* args, Py_ssize_t n) {
  constexpr int64_t kMaxChunk = 4096;  // tokens per call: bounds the scratch
  if (n != 13 || !plain_context() || !PyTuple_Check(args[9]) || PyTuple_GET_SIZE(args[9]) != 3) return unhandled();
  const at::Tensor *x = activation(args[0]), *ids = tensor(args[1]), *weights = tensor(args[2]);
  if (x == nullptr || ids == nullptr || weights == nullptr || x->scalar_type() == at::kFloat || x->numel() == 0) return unhandled();
  const int64_t experts = PyLong_AsLongLong(PyTuple_GET_ITEM(args[9], 0)), hidden = PyLong_AsLongLong(PyTuple_GET_ITEM(args[9], 1)),
                inter = PyLong_AsLongLong(PyTuple_GET_ITEM(args[9], 2)), bits13 = PyLong_AsLongLong(args[10]),
                bits2 = PyLong_AsLongLong(args[11]), group_size = PyLong_AsLongLong(args[12]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return unhandled();
  }
  const at::Tensor *q13, *q2;
  dq_weight w13, w2;
  if (!bank_of(args + 3, bits13, group_size, hidden, experts * 2 * inter, &q13, &w13) ||
      !bank_of(args + 6, bits2, group_size, inter, experts * hidden, &q2, &w2)) {
    return unhandled();
  }
  const at::Device device = q13->device();
  const int64_t tokens = x->size(-1) == hidden ? x->numel() / hidden : 0;
  if (tokens == 0 || ids->numel() % tokens != 0 || ids->numel() == 0 || weights->numel() != ids->numel() || x->device() != device ||
      q2->device() != device || ids->device() != device || weights->device() != device) {
    return unhandled();
  }
  const int64_t topk = ids->numel() / tokens;
  const int tag = tag_of(x->scalar_type());
  return on_device(device, [&](cudaStream_t stream) {
    const at::Tensor flat = x->is_contiguous() ? *x : x->contiguous();
    at::Tensor id = ids->scalar_type() == at::kInt ? *ids : ids->to(at::kInt);
    at::Tensor p = weights->scalar_type() == at::kFloat ? *weights : weights->to(at::kFloat);
    if (!id.is_contiguous()) id = id.contiguous();
    if (!p.is_contiguous()) p = p.contiguous();
    at::Tensor out = new_cuda(x->sizes(), x->scalar_type(), device);
    const int64_t row = hidden * x->element_size();
    const int64_t small = dq_moe_max_tokens();
    bool wide = moe_is_wide(tokens, topk, experts, small);
    at::Tensor scratch;
    for (int64_t at = 0; at < tokens;) {
      const int64_t count = std::min<int64_t>(tokens - at, wide ? kMaxChunk : small);
      int64_t need = 0;
      check(wide ? dq_moe_gemm_scratch_bytes(count, topk, hidden, inter, experts, tag, &need)
                 : dq_moe_scratch_bytes(count, topk, hidden, inter, experts, tag, &need));
      if (!scratch.defined() || scratch.numel() < need) scratch = new_cuda({need}, at::kByte, device);
      const auto call = wide ? dq_moe_gemm : dq_moe_gemv_shard;
      const int32_t rc = call(static_cast<const char*>(flat.const_data_ptr()) + at * row, tag, count,
                              static_cast<const int32_t*>(id.const_data_ptr()) + at * topk, static_cast<const float*>(p.const_data_ptr()) + at * topk,
                              topk, 0, experts, &w13, &w2, hidden, inter, static_cast<char*>(out.data_ptr()) + at * row, tag, scratch.data_ptr(),
                              scratch.numel(), stream);
      if (rc == DQ_ERR_UNSUPPORTED && wide) {
        wide = false;
        continue;
      }
      check(rc);
      at += count;
    }
    return out;
  });
}

// embedding(ids, packed, scales, offsets, bits, group_size, in_features)
PyObject* py_embedding(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7 || !plain_context()) return unhandled();
  const at::Tensor* ids = THPVariable_CheckExact(args[0]) ? tensor(args[0]) : nullptr;
  const at::Tensor *q, *s;
  dq_weight w;
  if (ids == nullptr || (ids->scalar_type() != at::kLong && ids->scalar_type() != at::kInt) || ids->numel() == 0 ||
      !matrix_of(args[1], args[2], args[3], args[4], args[5], args[6], &q, &s, &w) || ids->device() != q->device() || w.rows == 0) {
    return unhandled();
  }
  return on_device(q->device(), [&](cudaStream_t stream) {
    const at::Tensor flat = ids->is_contiguous() ? *ids : ids->contiguous();
    at::DimVector sizes(ids->sizes().begin(), ids->sizes().end());
    sizes.push_back(w.in_features);
    at::Tensor out = new_cuda(sizes, s->scalar_type(), q->device());
    check(dq_dequant_rows(&w, flat.const_data_ptr(), ids->scalar_type() == at::kInt, flat.numel(), out.data_ptr(), w.meta_dtype, stream));
    return out;
  });
}

// dequant(packed, scales, offsets, bits, group_size, in_features)
PyObject* py_dequant(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6 || !plain_context()) return unhandled();
  const at::Tensor *q, *s;
  dq_weight w;
  if (!matrix_of(args[0], args[1], args[2], args[3], args[4], args[5], &q, &s, &w) || w.rows == 0) return unhandled();
  return on_device(q->device(), [&](cudaStream_t stream) {
    at::Tensor out = new_cuda({w.rows, w.in_features}, s->scalar_type(), q->device());
    check(dq_dequant(&w, out.data_ptr(), w.meta_dtype, stream));
    return out;
  });
}

// encode(weight, bits, group_size, symmetric) -> (packed, scales, offsets), the metadata in the
// weight's own type if that has 16 bits, else fp16
PyObject* py_encode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || !plain_context()) return unhandled();
  const at::Tensor* w = tensor(args[0]);
  if (w == nullptr || w->dim() != 2 || tag_of(w->scalar_type()) < 0 || w->numel() == 0) return unhandled();
  const int64_t bits = PyLong_AsLongLong(args[1]), group_size = PyLong_AsLongLong(args[2]);
  const int symmetric = PyObject_IsTrue(args[3]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return unhandled();
  }
  int64_t group_values, groups, words;
  if (!row_shape(bits, group_size, w->size(1), &group_values, &groups, &words)) return unhandled();
  const at::ScalarType meta = w->scalar_type() == at::kFloat ? at::kHalf : w->scalar_type();
  at::Tensor scales, offsets;
  PyObject* packed = on_device(w->device(), [&](cudaStream_t stream) {
    const at::Tensor dense = w->is_contiguous() ? *w : w->contiguous();
    at::Tensor out = new_cuda({w->size(0), words}, at::kInt, w->device());
    scales = new_cuda({w->size(0), groups}, meta, w->device());
    offsets = new_cuda({w->size(0), groups}, meta, w->device());
    const int32_t rc = dq_encode(dense.const_data_ptr(), tag_of(w->scalar_type()), w->size(0), w->size(1), static_cast<int32_t>(bits),
                                 group_values, symmetric, out.data_ptr(), scales.data_ptr(), offsets.data_ptr(), tag_of(meta), stream);
    if (rc == DQ_ERR_UNSUPPORTED) return at::Tensor();
    check(rc);
    return out;
  });
  if (packed == nullptr || packed == Py_None) return packed;
  PyObject *so = THPVariable_Wrap(std::move(scales)), *oo = THPVariable_Wrap(std::move(offsets));
  PyObject* result = (so != nullptr && oo != nullptr) ? PyTuple_Pack(3, packed, so, oo) : nullptr;
  Py_XDECREF(so);
  Py_XDECREF(oo);
  Py_DECREF(packed);
  return result;
}

PyMethodDef kMethods[] = {
    {"matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_matmul)), METH_FASTCALL, nullptr},
    {"fused", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_fused)), METH_FASTCALL, nullptr},
    {"moe", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_moe)), METH_FASTCALL, nullptr},
    {"embedding", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_embedding)), METH_FASTCALL, nullptr},
    {"dequant", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_dequant)), METH_FASTCALL, nullptr},
    {"encode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_encode)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "The host path of the Python entry points.", -1, kMethods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host() { return PyModule_Create(&kModule); }
