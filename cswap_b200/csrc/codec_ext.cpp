// Tensor-level front end of the codecs as a CPython extension: argument checks,
// output allocation, stream lookup and the C ABI call of one codec call without
// going back through the interpreter.
//
// What bounds it: nothing but host time.  A call on a tensor of a few hundred
// KiB runs 3-6 us on the GPU, and the same steps through ctypes (five foreign
// calls, a device context manager, a torch.empty) took 11-13 us, so that the
// GPU waited for the host.  The wrappers in codec.py keep the documented
// signatures; these functions take every argument by position.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>

#include "../../include/cswap_b200.h"

namespace {

PyObject* g_check = nullptr;  // cswap_b200._lib.check: raises CswapError for a status

// false with a Python exception set
bool status_ok(csw_status st, const char* what) {
  if (st == CSW_OK) return true;
  PyObject* r = PyObject_CallFunction(g_check, "is", st, what);
  Py_XDECREF(r);
  return false;
}
bool value_error(const char* fmt, const char* name = nullptr) {
  PyErr_Format(PyExc_ValueError, fmt, name);  // `fmt` names one %s where `name` is given
  return false;
}
bool arg_count(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
  return false;
}

const at::Tensor* as_tensor(PyObject* o, const char* name) {
  if (THPVariable_Check(o)) return &THPVariable_Unpack(o);
  PyErr_Format(PyExc_TypeError, "%s must be a tensor", name);
  return nullptr;
}
bool require_cuda_f32(const at::Tensor& t, const char* name) {
  if (!t.is_cuda()) return value_error("%s must be a CUDA tensor (this path has no CPU implementation)", name);
  if (t.scalar_type() != at::kFloat) return value_error("%s must be float32", name);
  if (!t.is_contiguous()) return value_error("%s must be contiguous", name);
  return true;
}
bool as_size(PyObject* o, size_t* v) {
  const Py_ssize_t x = PyNumber_AsSsize_t(o, PyExc_OverflowError);
  if (x == -1 && PyErr_Occurred()) return false;
  *v = (size_t)x;
  return true;
}

struct Field {
  size_t nx = 0, ny = 0, nz = 0;
};
// An extent; one that is negative or beyond 63 bits fits no tensor.
bool as_extent(PyObject* o, size_t* v) {
  const Py_ssize_t x = PyNumber_AsSsize_t(o, nullptr);  // saturates, so that the product below cannot be met
  if (x == -1 && PyErr_Occurred()) return false;
  if (x < 0) return value_error("dims do not match the tensor's element count");
  *v = (size_t)x;
  return true;
}
// Whether the extents, 0 counting as 1 behind the first, multiply to numel.  A product that has
// passed numel (below 2^63) is not multiplied on, so nothing wraps.
bool covers(const Field& f, size_t numel) {
  unsigned __int128 p = f.nx;
  for (const size_t v : {f.ny, f.nz}) {
    if (p > numel) return false;
    p *= v ? v : 1;
  }
  return p == numel;
}
// (nx, ny, nz) of the call: the caller's, or the swap path's view
bool field_of(PyObject* dims, size_t numel, Field* f) {
  if (dims == Py_None) return status_ok(csw_zfp_view(numel, &f->nx, &f->ny, &f->nz), "csw_zfp_view");
  PyObject* seq = PySequence_Fast(dims, "dims must be (nx, ny, nz)");
  if (!seq) return false;
  bool ok = PySequence_Fast_GET_SIZE(seq) == 3;
  if (!ok) value_error("dims must be (nx, ny, nz)");
  ok = ok && as_extent(PySequence_Fast_GET_ITEM(seq, 0), &f->nx) &&
       as_extent(PySequence_Fast_GET_ITEM(seq, 1), &f->ny) && as_extent(PySequence_Fast_GET_ITEM(seq, 2), &f->nz);
  Py_DECREF(seq);
  if (ok && !covers(*f, numel))
    return value_error("dims do not match the tensor's element count");
  return ok;
}

at::Tensor new_on(const at::Tensor& like, int64_t n, at::ScalarType type) {
  return at::empty({n}, at::TensorOptions().dtype(type).device(like.device()));
}

// What every call ends with: the ABI call on the tensor's device and torch's
// current stream there, without the interpreter lock.
template <class F>
bool launch(const at::Tensor& t, const char* what, F&& call) {
  const c10::cuda::CUDAGuard on(t.device());
  const csw_stream_t stream = c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
  csw_status st;
  Py_BEGIN_ALLOW_THREADS;
  st = call(stream);
  Py_END_ALLOW_THREADS;
  return status_ok(st, what);
}

// C++ exceptions (an allocation that failed, say) become torch's Python ones
template <class F>
PyObject* guarded(F&& body) {
  HANDLE_TH_ERRORS
  return body();
  END_HANDLE_TH_ERRORS
}

// zfp_compress(t, maxbits, dims, out) -> stream
PyObject* zfp_compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    size_t maxbits, need;
    Field f;
    if (!arg_count(n, 4)) return nullptr;
    const at::Tensor* t = as_tensor(a[0], "t");
    if (!t || !require_cuda_f32(*t, "t") || !as_size(a[1], &maxbits) || !field_of(a[2], t->numel(), &f) ||
        !status_ok(csw_zfp_max_bytes(f.nx, f.ny, f.nz, (unsigned)maxbits, &need), "csw_zfp_max_bytes"))
      return nullptr;
    at::Tensor out;
    if (a[3] == Py_None) {
      out = new_on(*t, (int64_t)need, at::kByte);
    } else {
      const at::Tensor* o = as_tensor(a[3], "out");
      if (!o) return nullptr;
      if (o->nbytes() < need || !o->is_cuda()) {
        value_error("out is too small or not on the device");
        return nullptr;
      }
      out = *o;
    }
    const float* src = t->const_data_ptr<float>();
    void* dst = out.mutable_data_ptr();
    if (!launch(*t, "csw_zfp_compress", [&](csw_stream_t s) {
          return csw_zfp_compress(src, f.nx, f.ny, f.nz, (unsigned)maxbits, dst, out.nbytes(), nullptr, s);
        }))
      return nullptr;
    return THPVariable_Wrap(out);
  });
}

// zfp_decompress(stream, numel, maxbits, dims, out) -> tensor
PyObject* zfp_decompress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    size_t numel, maxbits;
    Field f;
    if (!arg_count(n, 5)) return nullptr;
    const at::Tensor* stream = as_tensor(a[0], "stream");
    if (!stream) return nullptr;
    if (!stream->is_cuda()) {
      value_error("stream must be a CUDA tensor");
      return nullptr;
    }
    if (!as_size(a[1], &numel) || !as_size(a[2], &maxbits)) return nullptr;
    at::Tensor out;
    if (a[4] == Py_None) {
      out = new_on(*stream, (int64_t)numel, at::kFloat);
    } else {
      const at::Tensor* o = as_tensor(a[4], "out");
      if (!o) return nullptr;
      out = *o;
    }
    if (!require_cuda_f32(out, "out") || !field_of(a[3], out.numel(), &f)) return nullptr;
    const void* src = stream->const_data_ptr();
    float* dst = out.mutable_data_ptr<float>();
    if (!launch(*stream, "csw_zfp_decompress", [&](csw_stream_t s) {
          return csw_zfp_decompress(src, stream->nbytes(), f.nx, f.ny, f.nz, (unsigned)maxbits, dst, s);
        }))
      return nullptr;
    return THPVariable_Wrap(out);
  });
}

// sparse_compress(t, out, nnz_out, onepass) -> (packed, nnz)
PyObject* sparse_compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (!arg_count(n, 4)) return nullptr;
    const at::Tensor* t = as_tensor(a[0], "t");
    csw_sparse_layout lay;
    if (!t || !require_cuda_f32(*t, "t") ||
        !status_ok(csw_sparse_layout_of((size_t)t->numel(), &lay), "csw_sparse_layout_of"))
      return nullptr;
    at::Tensor out, nnz;
    if (a[1] == Py_None) {
      out = new_on(*t, (int64_t)lay.bound, at::kByte);
    } else {
      const at::Tensor* o = as_tensor(a[1], "out");
      if (!o) return nullptr;
      out = *o;
    }
    if (a[2] == Py_None) {
      nnz = new_on(*t, 1, at::kInt);  // written by every call
    } else {
      const at::Tensor* o = as_tensor(a[2], "nnz_out");
      if (!o) return nullptr;
      nnz = *o;
    }
    const int onepass = PyObject_IsTrue(a[3]);
    if (onepass < 0) return nullptr;
    const auto entry = onepass ? csw_sparse_compress_onepass : csw_sparse_compress;
    const float* src = t->const_data_ptr<float>();
    void* dst = out.mutable_data_ptr();
    uint32_t* cnt = static_cast<uint32_t*>(nnz.mutable_data_ptr());
    if (!launch(*t, "csw_sparse_compress", [&](csw_stream_t s) {
          return entry(src, (size_t)t->numel(), dst, (size_t)out.numel(), cnt, s);
        }))
      return nullptr;
    PyObject* first = THPVariable_Wrap(out);
    PyObject* second = first ? THPVariable_Wrap(nnz) : nullptr;
    PyObject* both = second ? PyTuple_Pack(2, first, second) : nullptr;
    Py_XDECREF(first);
    Py_XDECREF(second);
    return both;
  });
}

// sparse_decompress(packed, n, out) -> tensor
PyObject* sparse_decompress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    size_t count;
    if (!arg_count(n, 3)) return nullptr;
    const at::Tensor* packed = as_tensor(a[0], "packed");
    if (!packed) return nullptr;
    if (!packed->is_cuda()) {
      value_error("packed must be a CUDA tensor");
      return nullptr;
    }
    if (!as_size(a[1], &count)) return nullptr;
    at::Tensor out;
    if (a[2] == Py_None) {
      out = new_on(*packed, (int64_t)count, at::kFloat);
    } else {
      const at::Tensor* o = as_tensor(a[2], "out");
      if (!o) return nullptr;
      out = *o;
    }
    if (!require_cuda_f32(out, "out")) return nullptr;
    const void* src = packed->const_data_ptr();
    float* dst = out.mutable_data_ptr<float>();
    if (!launch(*packed, "csw_sparse_decompress",
                [&](csw_stream_t s) { return csw_sparse_decompress(src, count, dst, s); }))
      return nullptr;
    return THPVariable_Wrap(out);
  });
}

PyMethodDef methods[] = {
    {"zfp_compress", (PyCFunction)(void (*)(void))zfp_compress, METH_FASTCALL, "(t, maxbits, dims, out) -> stream"},
    {"zfp_decompress", (PyCFunction)(void (*)(void))zfp_decompress, METH_FASTCALL,
     "(stream, numel, maxbits, dims, out) -> tensor"},
    {"sparse_compress", (PyCFunction)(void (*)(void))sparse_compress, METH_FASTCALL,
     "(t, out, nnz_out, onepass) -> (packed, nnz)"},
    {"sparse_decompress", (PyCFunction)(void (*)(void))sparse_decompress, METH_FASTCALL, "(packed, n, out) -> tensor"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_codec_ext", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__codec_ext() {
  PyObject* lib = PyImport_ImportModule("cswap_b200._lib");
  if (!lib) return nullptr;
  g_check = PyObject_GetAttrString(lib, "check");
  Py_DECREF(lib);
  return g_check ? PyModule_Create(&module) : nullptr;
}
