// The host path of a call, from torch tensors to the C ABI of libtq_b200.so, as one native function per entry point.
//
// A decode loop issues two calls per layer (append, attend) whose kernels take 3-10 us at short contexts; argument
// checks, tensor views and an 18-argument foreign call written in Python took about 34 us per call, so a short step was
// bound by the host five times over.  Here a call is argument unpacking, the checks, one output allocation and the
// launch.  Arguments that are already in the form the kernels take (device, type, contiguous) are used as they are;
// anything else is converted through torch first, as the Python layer did.
#include <Python.h>
#include <pybind11/pybind11.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>

#include "tq_b200.h"
#include "tq_host_copy.h"

namespace {

PyObject* g_tq_error = nullptr;   // turboquant_plus_b200._native.TQError

// A Python exception with its message has been set: unwind to the entry point.
struct PyRaised {};

[[noreturn]] void raise(PyObject* type, const char* msg) {
  PyErr_SetString(type, msg);
  throw PyRaised{};
}

void check(int64_t rc) {
  if (rc >= 0) return;
  const char* last = tq_last_error();
  if (rc == TQ_ERR_INVALID) raise(PyExc_ValueError, last && *last ? last : tq_error_string((int)rc));
  PyErr_Format(g_tq_error ? g_tq_error : PyExc_RuntimeError, "%s: %s", tq_error_string((int)rc),
               last && *last ? last : tq_error_string((int)rc));
  throw PyRaised{};
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch tensor, got %s", what, Py_TYPE(o)->tp_name);
    throw PyRaised{};
  }
  return THPVariable_Unpack(o);
}

template <typename T = void>
T* address(PyObject* o) {
  if (o == Py_None) return nullptr;
  void* p = PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw PyRaised{};
  return reinterpret_cast<T*>(p);
}

int64_t integer(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyRaised{};
  return v;
}

double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyRaised{};
  return v;
}

int32_t dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return TQ_F32;
    case at::kHalf: return TQ_F16;
    case at::kDouble: return TQ_F64;
    case at::kBFloat16: return TQ_BF16;
    default: break;
  }
  PyErr_Format(PyExc_KeyError, "%s", c10::toString(t));
  throw PyRaised{};
}

// `t` on `dev` as contiguous `type`; the tensor itself when it is that already
at::Tensor as(const at::Tensor& t, c10::Device dev, at::ScalarType type) {
  if (t.device() == dev && t.scalar_type() == type) return t.is_contiguous() ? t : t.contiguous();
  return t.to(dev, type).contiguous();
}

// contiguous tensor on the device the launch will run on
at::Tensor rows(const at::Tensor& t, c10::Device dev, const char* what) {
  if (t.device() != dev) {
    PyErr_Format(PyExc_ValueError, "%s must be on %s, got %s", what, dev.str().c_str(), t.device().str().c_str());
    throw PyRaised{};
  }
  return t.is_contiguous() ? t : t.contiguous();
}

// the device of a call made current for its duration, and the stream torch has selected on it
struct On {
  c10::cuda::OptionalCUDAGuard guard;
  void* stream;
  explicit On(c10::Device dev) {
    if (c10::cuda::current_device() != dev.index()) guard.set_device(dev);
    stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  }
};

void need(Py_ssize_t got, Py_ssize_t want, const char* name) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, got);
    throw PyRaised{};
  }
}

template <typename F>
PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  try {
    return f();
  } catch (const PyRaised&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

PyObject* none() { Py_RETURN_NONE; }

// set_error(type): the exception raised for status codes other than TQ_ERR_INVALID
PyObject* set_error(PyObject*, PyObject* type) {
  Py_INCREF(type);
  Py_XSETREF(g_tq_error, type);
  Py_RETURN_NONE;
}

// same_bytes(buffer, bytes): whether a C-contiguous buffer holds exactly these bytes
PyObject* same_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "same_bytes");
    Py_buffer b;
    if (PyObject_GetBuffer(a[0], &b, PyBUF_C_CONTIGUOUS) != 0) throw PyRaised{};
    const bool same = PyBytes_Check(a[1]) && b.len == PyBytes_GET_SIZE(a[1]) &&
                      memcmp(b.buf, PyBytes_AS_STRING(a[1]), (size_t)b.len) == 0;
    PyBuffer_Release(&b);
    return PyBool_FromLong(same);
  });
}

// append(k quantizer, v quantizer, layout, pool, k, v, slots)
PyObject* append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 7, "append");
    const auto* L = address<const tq_cache_layout>(a[2]);
    const at::Tensor& pool = tensor(a[3], "pool");
    const c10::Device dev = pool.device();
    const at::Tensor &k0 = tensor(a[4], "k"), &v0 = tensor(a[5], "v");
    if (k0.dim() != 3 || k0.sizes() != v0.sizes() || k0.size(1) != L->num_kv_heads || k0.size(2) != L->d)
      raise(PyExc_AssertionError, "k and v must have the shape (n_tokens, num_kv_heads, head_dim)");
    if (k0.scalar_type() != v0.scalar_type()) raise(PyExc_AssertionError, "k and v must have the same dtype");
    const at::Tensor k = rows(k0, dev, "k"), v = rows(v0, dev, "v");
    const at::Tensor slots = as(tensor(a[6], "slot_mapping"), dev, at::kLong);
    const On on(dev);
    check(tq_cache_append(address<const tq_quantizer>(a[0]), address<const tq_quantizer>(a[1]), L,
                          static_cast<uint8_t*>(pool.data_ptr()), k.const_data_ptr(), v.const_data_ptr(),
                          dtype_code(k.scalar_type()), k.size(0), static_cast<const int64_t*>(slots.const_data_ptr()),
                          on.stream));
    return none();
  });
}

// attend(k quantizer, v quantizer, layout, pool, q, block_table, seq_lens, scale, out or None, workspace, phases,
//        want_lse) -> out or (out, lse)
PyObject* attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 12, "attend");
    const auto* L = address<const tq_cache_layout>(a[2]);
    const at::Tensor& pool = tensor(a[3], "pool");
    const c10::Device dev = pool.device();
    const at::Tensor& q0 = tensor(a[4], "q");
    if (q0.dim() != 3) raise(PyExc_ValueError, "q must have the shape (batch, num_q_heads, head_dim)");
    if (q0.size(2) != L->d) raise(PyExc_AssertionError, "the queries' last dimension is not the head dimension");
    const at::Tensor q = rows(q0, dev, "q");
    const at::Tensor bt = as(tensor(a[5], "block_table"), dev, at::kInt);
    const at::Tensor sl = as(tensor(a[6], "seq_lens"), dev, at::kInt);
    const at::Tensor& ws = tensor(a[9], "workspace");
    at::Tensor out = a[8] == Py_None ? at::empty_like(q) : tensor(a[8], "out");
    const int32_t batch = (int32_t)q.size(0), hq = (int32_t)q.size(1);
    const auto *kq = address<const tq_quantizer>(a[0]), *vq = address<const tq_quantizer>(a[1]);
    const float scale = (float)real(a[7]);
    const int32_t phases = (int32_t)integer(a[10]);
    const bool want_lse = PyObject_IsTrue(a[11]) == 1;
    at::Tensor lse;
    if (want_lse) lse = at::empty({batch, hq}, q.options().dtype(at::kFloat));
    const On on(dev);
    const auto* pool_p = static_cast<const uint8_t*>(pool.const_data_ptr());
    const auto *bt_p = static_cast<const int32_t*>(bt.const_data_ptr()), *sl_p = static_cast<const int32_t*>(sl.const_data_ptr());
    const int32_t pages = (int32_t)bt.size(1), qd = dtype_code(q.scalar_type()), od = dtype_code(out.scalar_type());
    if (want_lse)
      check(tq_decode_attn_lse(kq, vq, L, pool_p, bt_p, pages, sl_p, q.const_data_ptr(), qd, batch, hq, scale, ws.data_ptr(),
                               ws.numel(), out.data_ptr(), od, phases, static_cast<float*>(lse.data_ptr()), on.stream));
    else
      check(tq_decode_attn_phases(kq, vq, L, pool_p, bt_p, pages, sl_p, q.const_data_ptr(), qd, batch, hq, scale,
                                  ws.data_ptr(), ws.numel(), out.data_ptr(), od, phases, on.stream));
    PyObject* o = a[8] == Py_None ? THPVariable_Wrap(std::move(out)) : Py_NewRef(a[8]);
    if (!want_lse) return o;
    return Py_BuildValue("(NN)", o, THPVariable_Wrap(std::move(lse)));
  });
}

// prefill(k quantizer, v quantizer, layout, pool, q, block_table, kv_lens, scale, out or None, workspace) -> out
PyObject* prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 10, "prefill");
    const auto* L = address<const tq_cache_layout>(a[2]);
    const at::Tensor& pool = tensor(a[3], "pool");
    const c10::Device dev = pool.device();
    const at::Tensor& q0 = tensor(a[4], "q");
    if (q0.dim() != 4) raise(PyExc_ValueError, "q must have the shape (batch, chunk_tokens, num_q_heads, head_dim)");
    if (q0.size(3) != L->d) raise(PyExc_AssertionError, "the queries' last dimension is not the head dimension");
    const at::Tensor q = rows(q0, dev, "q");
    const at::Tensor bt = as(tensor(a[5], "block_table"), dev, at::kInt);
    const at::Tensor kl = as(tensor(a[6], "kv_lens"), dev, at::kInt);
    const at::Tensor& ws = tensor(a[9], "workspace");
    at::Tensor out = a[8] == Py_None ? at::empty_like(q) : tensor(a[8], "out");
    const On on(dev);
    check(tq_prefill_attn(address<const tq_quantizer>(a[0]), address<const tq_quantizer>(a[1]), L,
                          static_cast<const uint8_t*>(pool.const_data_ptr()), static_cast<const int32_t*>(bt.const_data_ptr()),
                          (int32_t)bt.size(1), static_cast<const int32_t*>(kl.const_data_ptr()), q.const_data_ptr(),
                          dtype_code(q.scalar_type()), (int32_t)q.size(0), (int32_t)q.size(1), (int32_t)q.size(2),
                          (float)real(a[7]), ws.data_ptr(), ws.numel(), out.data_ptr(), dtype_code(out.scalar_type()),
                          on.stream));
    return a[8] == Py_None ? THPVariable_Wrap(std::move(out)) : Py_NewRef(a[8]);
  });
}

// workspace_bytes(batch, q heads, kv heads, pages, chunk tokens or 0): scratch of a decode (0) or prefill call
PyObject* workspace_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5, "workspace_bytes");
    const int32_t b = (int32_t)integer(a[0]), hq = (int32_t)integer(a[1]), hkv = (int32_t)integer(a[2]);
    const int32_t pages = (int32_t)integer(a[3]), chunk = (int32_t)integer(a[4]);
    const int64_t w = chunk ? tq_prefill_workspace_bytes(b, chunk, hq, hkv, pages) : tq_decode_workspace_bytes(b, hq, hkv, pages);
    check(w);
    return PyLong_FromLongLong(w);
  });
}

// quantize(quantizer, x (n, d or more columns, of which the first d count), d, bits, packed, want_scale, want_qjl) -> (codes,
// norms, scales or None, sketch or None, residual norms or None), all on x's device
PyObject* quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 7, "quantize");
    const at::Tensor& x = tensor(a[1], "x");
    const c10::Device dev = x.device();
    const int64_t d = integer(a[2]), bits = integer(a[3]);
    if (!dev.is_cuda() || x.dim() != 2 || x.size(1) < d) raise(PyExc_ValueError, "x must be a CUDA tensor of shape (n, d)");
    const int64_t nv = x.size(0);
    const bool packed = PyObject_IsTrue(a[4]) == 1, scale = PyObject_IsTrue(a[5]) == 1, qjl = PyObject_IsTrue(a[6]) == 1;
    const auto u8 = x.options().dtype(at::kByte), f32 = x.options().dtype(at::kFloat);
    at::Tensor codes = at::empty({nv, packed ? d * bits / 8 : d}, u8), norms = at::empty({nv}, f32), scales, sketch, rnorms;
    if (scale) scales = at::empty({nv}, f32);
    if (qjl) {
      sketch = at::empty({nv, (d + 7) / 8}, u8);
      rnorms = at::empty({nv}, f32);
    }
    auto u8p = [](const at::Tensor& t) { return t.defined() ? static_cast<uint8_t*>(t.data_ptr()) : nullptr; };
    auto fp = [](const at::Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; };
    const On on(dev);
    check(tq_quantize(address<const tq_quantizer>(a[0]), x.const_data_ptr(), dtype_code(x.scalar_type()), x.stride(0), nv,
                      packed ? u8p(codes) : nullptr, packed ? nullptr : u8p(codes), fp(norms), fp(scales), u8p(sketch),
                      fp(rnorms), on.stream));
    auto wrap = [](at::Tensor& t) { return t.defined() ? THPVariable_Wrap(std::move(t)) : none(); };
    return Py_BuildValue("(NNNNN)", wrap(codes), wrap(norms), wrap(scales), wrap(sketch), wrap(rnorms));
  });
}

// dequantize(quantizer, codes (n, ...), packed, norms, sketch or None, residual norms or None, shrinkage, d, dtype code)
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 9, "dequantize");
    const at::Tensor &codes = tensor(a[1], "codes"), &norms = tensor(a[3], "norms");
    const c10::Device dev = codes.device();
    if (!dev.is_cuda() || !codes.is_contiguous() || !norms.is_contiguous())
      raise(PyExc_ValueError, "codes and norms must be contiguous CUDA tensors");
    const int64_t nv = codes.size(0), d = integer(a[7]);
    const bool packed = PyObject_IsTrue(a[2]) == 1, qjl = a[4] != Py_None;
    const int32_t od = (int32_t)integer(a[8]);
    at::Tensor out = at::empty({nv, d}, codes.options().dtype(od == TQ_F64 ? at::kDouble : od == TQ_F16 ? at::kHalf : at::kFloat));
    const auto* c = static_cast<const uint8_t*>(codes.const_data_ptr());
    const On on(dev);
    check(tq_dequantize(address<const tq_quantizer>(a[0]), packed ? c : nullptr, packed ? nullptr : c,
                        static_cast<const float*>(norms.const_data_ptr()),
                        qjl ? static_cast<const uint8_t*>(tensor(a[4], "sketch").const_data_ptr()) : nullptr,
                        qjl ? static_cast<const float*>(tensor(a[5], "residual norms").const_data_ptr()) : nullptr,
                        (float)real(a[6]), nv, out.data_ptr(), od, on.stream));
    return THPVariable_Wrap(std::move(out));
  });
}

// sign_bits(t, d, pack): rows of d int8 signs <-> rows of ceil(d / 8) bytes
PyObject* sign_bits(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "sign_bits");
    const at::Tensor& t = tensor(a[0], "signs");
    const int64_t nv = t.size(0), d = integer(a[1]);
    const bool pack = PyObject_IsTrue(a[2]) == 1;
    if (!t.is_cuda() || !t.is_contiguous()) raise(PyExc_ValueError, "signs must be a contiguous CUDA tensor");
    at::Tensor out = at::empty({nv, pack ? (d + 7) / 8 : d}, t.options().dtype(pack ? at::kByte : at::kChar));
    const On on(t.device());
    if (pack)
      check(tq_pack_bits(static_cast<const int8_t*>(t.const_data_ptr()), nv, (int32_t)d, static_cast<uint8_t*>(out.data_ptr()), on.stream));
    else
      check(tq_unpack_bits(static_cast<const uint8_t*>(t.const_data_ptr()), nv, (int32_t)d, static_cast<int8_t*>(out.data_ptr()), on.stream));
    return THPVariable_Wrap(std::move(out));
  });
}

// cut(t, layers, heads): views of a tensor's layers x heads equal runs of rows, as a list of lists.  (One dispatch for all of them: 0.35 us a
// view; 0.6 with one each, 1.3 as slices in Python.)
PyObject* cut(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "cut");
    const at::Tensor& t = tensor(a[0], "t");
    const int64_t layers = integer(a[1]), heads = integer(a[2]);
    if (t.dim() < 1 || layers < 1 || heads < 1 || t.size(0) % (layers * heads)) raise(PyExc_ValueError, "rows do not divide into the runs");
    const std::vector<at::Tensor> runs = t.unflatten(0, {layers * heads, t.size(0) / (layers * heads)}).unbind(0);
    PyObject* all = PyList_New(layers);
    if (!all) throw PyRaised{};
    for (int64_t l = 0; l < layers; ++l) {
      PyObject* one = PyList_New(heads);
      if (!one) {
        Py_DECREF(all);
        throw PyRaised{};
      }
      PyList_SET_ITEM(all, l, one);
      try {
        for (int64_t h = 0; h < heads; ++h) PyList_SET_ITEM(one, h, THPVariable_Wrap(runs[l * heads + h]));
      } catch (...) {
        Py_DECREF(all);
        throw;
      }
    }
    return all;
  });
}

// join(list of tensors): their rows one after the other.  Runs that lie so in memory, as cut made them, are one view: a copy and a launch
// less for each of six tensors (4 layers x 8 heads of 2,000 rows: 190 us a
// decompress, 140 of them now, with the pieces' way through Python 126 and 79 of the host); others are concatenated.
PyObject* join(PyObject*, PyObject* list) {
  return guarded([&]() -> PyObject* {
    if (!PyList_Check(list) || PyList_GET_SIZE(list) == 0) raise(PyExc_ValueError, "join needs a list of tensors");
    const Py_ssize_t n = PyList_GET_SIZE(list);
    const at::Tensor& first = tensor(PyList_GET_ITEM(list, 0), "piece");
    bool plain = first.layout() == at::kStrided && first.has_storage() && !first.requires_grad() && !first.is_conj() && !first.is_neg() &&
                 first.dim() >= 1 && reinterpret_cast<uintptr_t>(first.const_data_ptr()) % 16 == 0;
    int64_t rows = 0, at = plain ? first.storage_offset() : 0;
    for (Py_ssize_t i = 0; i < n && plain; ++i) {
      const at::Tensor& t = tensor(PyList_GET_ITEM(list, i), "piece");
      plain = t.is_contiguous() && t.scalar_type() == first.scalar_type() && t.dim() == first.dim() && t.sizes().slice(1) == first.sizes().slice(1) &&
              t.key_set() == first.key_set() && t.has_storage() && t.storage().unsafeGetStorageImpl() == first.storage().unsafeGetStorageImpl() &&
              t.storage_offset() == at && !t.requires_grad();
      if (plain) {
        rows += t.size(0);
        at += t.numel();
      }
    }
    if (plain && n == 1) return Py_NewRef(PyList_GET_ITEM(list, 0));
    if (plain) {
      std::vector<int64_t> sizes(first.sizes().begin(), first.sizes().end()), strides(sizes.size(), 1);
      sizes[0] = rows;
      for (size_t k = sizes.size() - 1; k > 0; --k) strides[k - 1] = strides[k] * std::max<int64_t>(sizes[k], 1);   // (a piece's own: any where it has one row)
      return THPVariable_Wrap(first.as_strided(sizes, strides, first.storage_offset()));
    }
    std::vector<at::Tensor> all;
    for (Py_ssize_t i = 0; i < n; ++i) all.push_back(tensor(PyList_GET_ITEM(list, i), "piece"));
    return THPVariable_Wrap(at::cat(all));
  });
}

// the elements of a C-contiguous buffer of a type the copies know; PyBuffer released by the caller
tqhost::HostArray host_array(Py_buffer* b) {
  char f = b->format ? b->format[0] : 'B';
  if (f == '<' || f == '=' || f == '@') f = b->format[1];
  using tqhost::Elem;
  Elem e = Elem::U8;
  if (f == 'd') e = Elem::F64;
  else if (f == 'f') e = Elem::F32;
  else if (f == 'e') e = Elem::F16;
  else if ((f == 'l' || f == 'q') && b->itemsize == 8) e = Elem::I64;
  else if ((f == 'i' || f == 'l') && b->itemsize == 4) e = Elem::I32;
  else if (f == 'b') e = Elem::I8;
  else if (f != 'B') raise(PyExc_TypeError, "array type without a host copy");
  return {b->buf, b->itemsize ? (int64_t)(b->len / b->itemsize) : 0, e};
}

struct Buffers {
  std::vector<Py_buffer> all;
  ~Buffers() {
    for (auto& b : all) PyBuffer_Release(&b);
  }
  tqhost::HostArray get(PyObject* o, int flags) {
    all.emplace_back();
    if (PyObject_GetBuffer(o, &all.back(), flags | PyBUF_C_CONTIGUOUS | PyBUF_FORMAT) != 0) {
      all.pop_back();
      throw PyRaised{};
    }
    return host_array(&all.back());
  }
};

// upload(array, device index, dtype code or -2 for bytes, -3 for signed bytes) -> CUDA tensor of the array's shape
PyObject* upload(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "upload");
    Buffers bufs;
    const tqhost::HostArray h = bufs.get(a[0], PyBUF_SIMPLE);
    const Py_buffer& b = bufs.all.back();
    std::vector<int64_t> shape(b.shape, b.shape + b.ndim);
    const int64_t code = integer(a[2]);
    const at::ScalarType type = code == -2 ? at::kByte : code == -3 ? at::kChar : code == TQ_F64 ? at::kDouble
                                : code == TQ_F16 ? at::kHalf : at::kFloat;
    const c10::Device dev(c10::DeviceType::CUDA, (c10::DeviceIndex)integer(a[1]));
    at::Tensor t;
    {
      pybind11::gil_scoped_release nogil;
      const On on(dev);
      t = at::empty(shape, at::TensorOptions().device(dev).dtype(type));
      tqhost::to_device(h, t);
    }
    return THPVariable_Wrap(std::move(t));
  });
}

// download(tensor, array, tensor, array, ...): fills the arrays, converted to their types
PyObject* download(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Buffers bufs;
    bufs.all.reserve(n);
    std::vector<std::pair<at::Tensor, tqhost::HostArray>> jobs;
    for (Py_ssize_t i = 0; i + 1 < n; i += 2) {
      const at::Tensor& t = tensor(a[i], "source");
      const tqhost::HostArray h = bufs.get(a[i + 1], PyBUF_WRITABLE);
      if (!t.is_cuda() || t.numel() != h.count) raise(PyExc_ValueError, "download needs CUDA tensors and arrays of their sizes");
      jobs.emplace_back(t.is_contiguous() ? t : t.contiguous(), h);
    }
    if (!jobs.empty()) {
      pybind11::gil_scoped_release nogil;
      const On on(jobs[0].first.device());
      tqhost::to_host(jobs);
    }
    return none();
  });
}

#define TQ_FAST(name, f, doc) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, doc}
PyMethodDef methods[] = {
    {"set_error", set_error, METH_O, "exception type of failed calls"},
    TQ_FAST("same_bytes", same_bytes, "whether a buffer holds these bytes"),
    TQ_FAST("append", append, "tq_cache_append on tensors"),
    TQ_FAST("attend", attend, "tq_decode_attn_phases / tq_decode_attn_lse on tensors"),
    TQ_FAST("prefill", prefill, "tq_prefill_attn on tensors"),
    TQ_FAST("workspace_bytes", workspace_bytes, "scratch bytes of a decode or prefill call"),
    TQ_FAST("quantize", quantize, "tq_quantize on tensors"),
    TQ_FAST("dequantize", dequantize, "tq_dequantize on tensors"),
    TQ_FAST("sign_bits", sign_bits, "tq_pack_bits / tq_unpack_bits on tensors"),
    TQ_FAST("cut", cut, "runs of a tensor's rows as views"),
    {"join", join, METH_O, "runs of rows as one tensor"},
    TQ_FAST("upload", upload, "host array to a CUDA tensor, converted"),
    TQ_FAST("download", download, "CUDA tensors into host arrays, converted"),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tq_host", "tensor front end of libtq_b200.so", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tq_host() { return PyModule_Create(&module); }
