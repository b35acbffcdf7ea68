// The per-call half of the Python binding: the checks, pointers and stream of
// a collective on CUDA tensors, read from the tensors themselves instead of
// through a dozen Python attributes and ctypes conversions.
//
// Small messages are bound by the host: a 4 KiB world-size-1 allreduce spent
// 8 us per call, of which the launch itself is 2.3 us (an empty kernel, back
// to back) and the Python side most of the rest.  Everything that is not on
// the path of a collective (set-up, messaging, diagnostics) stays in ctypes.
//
// The functions raise the package's IbcommError and return None.  The GIL is
// released around the library call, as ctypes does.  Tensors without storage, a
// missing driver and the like are C++ exceptions in torch: the entry points turn
// them into the Python exceptions torch's own methods raise.
#include <Python.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "ibcomm/c_api.h"
#include "ibcomm/device_types.h"

namespace {

PyObject* g_error = nullptr;  // IbcommError(code, message)

constexpr int kInvalidArgument = 1, kNotSupported = 4;

PyObject* Raise(int code, const char* message) {
  PyObject* e = g_error != nullptr ? PyObject_CallFunction(g_error, "is", code, message) : nullptr;
  if (e != nullptr) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  } else if (!PyErr_Occurred()) {
    PyErr_SetString(PyExc_RuntimeError, message);
  }
  return nullptr;
}

PyObject* RaiseLast(int code) {
  std::string m = ibcomm_last_error();
  while (!m.empty() && (m.back() == '\n' || m.back() == ' ')) m.pop_back();
  return Raise(code, m.c_str());
}

// Code of the library's element type, or -1.
int DTypeCode(c10::ScalarType t) {
  switch (t) {
    case c10::ScalarType::Float: return 0;
    case c10::ScalarType::Double: return 1;
    case c10::ScalarType::Int: return 2;
    case c10::ScalarType::Long: return 3;
    case c10::ScalarType::Half: return 4;
    case c10::ScalarType::BFloat16: return 5;
    default: return -1;
  }
}

// The tensor behind `o`; null with an exception set when it is none, has an
// unsupported type, is not contiguous or out of the GPU's reach.
const at::Tensor* Tensor(PyObject* o, int* dtype) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "a torch.Tensor is expected");
    return nullptr;
  }
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_contiguous()) {
    Raise(kInvalidArgument, "tensors must be contiguous");
    return nullptr;
  }
  const int d = DTypeCode(t.scalar_type());
  if (d < 0) {
    Raise(kNotSupported, (std::string("unsupported dtype ") + c10::toString(t.scalar_type())).c_str());
    return nullptr;
  }
  // A kernel reads and writes it: memory of a GPU, or pinned host memory.
  if (!t.is_cuda() && !t.is_pinned()) {
    Raise(kInvalidArgument, "tensors must live on the GPU");
    return nullptr;
  }
  *dtype = d;
  return &t;
}

// Whether a kernel that runs on the GPU of `a` can be given `b` too.
bool SameGpu(const at::Tensor& a, const at::Tensor& b) { return !a.is_cuda() || !b.is_cuda() || a.device() == b.device(); }

template <typename Handle>
bool ToHandle(PyObject* o, Handle** h) {
  *h = o == Py_None ? nullptr : static_cast<Handle*>(PyLong_AsVoidPtr(o));
  return !PyErr_Occurred();
}

// `stream` (a raw stream as an integer) or, for None, the current one of `device`.
bool ToStream(PyObject* stream, c10::DeviceIndex device, void** out) {
  if (stream == Py_None) {
    *out = c10::cuda::getCurrentCUDAStream(device).stream();
    return true;
  }
  *out = PyLong_AsVoidPtr(stream);
  return !PyErr_Occurred();
}

bool WantArgs(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "%zd arguments are expected, got %zd", want, n);
  return false;
}

// The tensors of a sequence, one per rank.  It holds on to the sequence: one that
// makes its items as it is read (the rows of a tensor) has them live no longer
// than the list they were gathered in.
struct RankTensors {
  PyObject* list = nullptr;
  void* ptr[ibcomm::kMaxRanks] = {};
  const at::Tensor* first = nullptr;
  int dtype = 0;
  int64_t shortest = 0;  // fewest elements of one

  RankTensors() = default;
  RankTensors(const RankTensors&) = delete;
  RankTensors& operator=(const RankTensors&) = delete;
  ~RankTensors() { Py_XDECREF(list); }

  // `elements` fit into every tensor, and `o` is of the same type on the same GPU.
  bool Hold(int64_t elements, const RankTensors& o) const { return shortest >= elements && dtype == o.dtype && SameGpu(*first, *o.first); }

  // A short sequence leaves nulls, which the library refuses.
  bool Read(PyObject* seq, int ranks) {
    list = PySequence_Fast(seq, "a sequence of tensors is expected");
    if (list == nullptr) return false;
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(list);
    if (n > ranks || n == 0) {
      PyErr_SetString(PyExc_IndexError, "one tensor per rank is expected");
      return false;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
      int d;
      const at::Tensor* t = Tensor(PySequence_Fast_GET_ITEM(list, i), &d);
      if (t == nullptr) return false;
      if (i == 0) first = t, dtype = d, shortest = t->numel();
      if (d != dtype || !SameGpu(*first, *t)) {
        Raise(kInvalidArgument, "the ranks' tensors must match in dtype and live on one GPU");
        return false;
      }
      if (t->numel() < shortest) shortest = t->numel();
      ptr[i] = t->data_ptr();
    }
    return true;
  }
};

PyObject* Done(int code) {
  if (code != 0) return RaiseLast(code);
  Py_RETURN_NONE;
}

// set_error(IbcommError)
PyObject* SetError(PyObject*, PyObject* cls) {
  Py_XDECREF(g_error);
  g_error = Py_NewRef(cls);
  Py_RETURN_NONE;
}

// allreduce(handle, send, recv, algo, scale, wire, stream, flags); wire < 0: the tensors' type
PyObject* Allreduce(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!WantArgs(n, 8)) return nullptr;
  ibcomm_comm* c;
  if (!ToHandle(a[0], &c)) return nullptr;
  int d, rd;
  const at::Tensor* s = Tensor(a[1], &d);
  if (s == nullptr) return nullptr;
  const at::Tensor* r = Tensor(a[2], &rd);
  if (r == nullptr) return nullptr;
  if (d != rd || s->numel() != r->numel()) return Raise(kInvalidArgument, "sendbuf and recvbuf must match in dtype and size");
  if (!SameGpu(*s, *r)) return Raise(kInvalidArgument, "sendbuf and recvbuf must live on the same GPU");
  const int algo = static_cast<int>(PyLong_AsLong(a[3]));
  const double scale = PyFloat_AsDouble(a[4]);
  const int wire = static_cast<int>(PyLong_AsLong(a[5]));
  const int flags = static_cast<int>(PyLong_AsLong(a[7]));
  void* stream;
  if (PyErr_Occurred() || !ToStream(a[6], s->device().index(), &stream)) return nullptr;
  const void* in = s->data_ptr();
  void* out = r->data_ptr();
  const size_t len = static_cast<size_t>(s->numel());
  if (len != 0 && (in == nullptr || out == nullptr)) return Raise(kInvalidArgument, "tensors must have memory");
  int code;
  Py_BEGIN_ALLOW_THREADS;
  code = ibcomm_allreduce_cuda(c, algo, d, in, out, len, scale, wire < 0 ? d : wire, stream, flags);
  Py_END_ALLOW_THREADS;
  return Done(code);
  END_HANDLE_TH_ERRORS
}

// copy_scale(src, dst, scale)
PyObject* CopyScale(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!WantArgs(n, 3)) return nullptr;
  int di, dout;
  const at::Tensor* s = Tensor(a[0], &di);
  if (s == nullptr) return nullptr;
  const at::Tensor* d = Tensor(a[1], &dout);
  if (d == nullptr) return nullptr;
  if (!s->is_cuda()) return Raise(kInvalidArgument, "src must be a CUDA tensor");
  if (d->numel() < s->numel() || !SameGpu(*s, *d)) return Raise(kInvalidArgument, "dst must hold every element of src, on the same GPU");
  const double scale = PyFloat_AsDouble(a[2]);
  if (PyErr_Occurred()) return nullptr;
  const void* in = s->data_ptr();
  void* out = d->data_ptr();
  const size_t len = static_cast<size_t>(s->numel());
  if (len != 0 && (in == nullptr || out == nullptr)) return Raise(kInvalidArgument, "tensors must have memory");
  void* stream = c10::cuda::getCurrentCUDAStream(s->device().index()).stream();
  int code;
  Py_BEGIN_ALLOW_THREADS;
  code = ibcomm_copy_scale(in, out, len, di, dout, scale, stream);
  Py_END_ALLOW_THREADS;
  return Done(code);
  END_HANDLE_TH_ERRORS
}

// emu_allreduce(handle, ranks, sends, recvs, algo, scale, wire, channels, stream, async)
PyObject* EmuAllreduce(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!WantArgs(n, 10)) return nullptr;
  ibcomm_emu* w;
  if (!ToHandle(a[0], &w)) return nullptr;
  const int ranks = static_cast<int>(PyLong_AsLong(a[1]));
  RankTensors in, out;
  if (PyErr_Occurred()) return nullptr;
  if (ranks < 1 || ranks > ibcomm::kMaxRanks) return Raise(kNotSupported, "the number of ranks is out of range");
  if (!in.Read(a[2], ranks) || !out.Read(a[3], ranks)) return nullptr;
  const int64_t len = in.first->numel();
  if (!in.Hold(len, out) || !out.Hold(len, in))
    return Raise(kInvalidArgument, "every rank's tensors must match in dtype and hold as many elements as the first");
  const int algo = static_cast<int>(PyLong_AsLong(a[4]));
  const double scale = PyFloat_AsDouble(a[5]);
  const int wire = static_cast<int>(PyLong_AsLong(a[6]));
  const int channels = static_cast<int>(PyLong_AsLong(a[7]));
  const int async = static_cast<int>(PyLong_AsLong(a[9]));
  void* stream;
  if (PyErr_Occurred() || !ToStream(a[8], -1, &stream)) return nullptr;
  int code;
  Py_BEGIN_ALLOW_THREADS;
  code = ibcomm_emu_allreduce(w, algo, in.dtype, in.ptr, out.ptr, static_cast<size_t>(len), scale, wire < 0 ? in.dtype : wire, channels, stream, async);
  Py_END_ALLOW_THREADS;
  return Done(code);
  END_HANDLE_TH_ERRORS
}

// emu_rsag(handle, ranks, all_gather, sends, recvs, scale, channels)
PyObject* EmuRsAg(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!WantArgs(n, 7)) return nullptr;
  ibcomm_emu* w;
  if (!ToHandle(a[0], &w)) return nullptr;
  const int ranks = static_cast<int>(PyLong_AsLong(a[1]));
  const int all_gather = static_cast<int>(PyLong_AsLong(a[2]));
  RankTensors in, out;
  if (PyErr_Occurred()) return nullptr;
  if (ranks < 1 || ranks > ibcomm::kMaxRanks) return Raise(kNotSupported, "the number of ranks is out of range");
  if (!in.Read(a[3], ranks) || !out.Read(a[4], ranks)) return nullptr;
  const int64_t block = (all_gather ? in : out).first->numel();
  if (!in.Hold(all_gather ? block : block * ranks, out) || !out.Hold(all_gather ? block * ranks : block, in))
    return Raise(kInvalidArgument, "every rank's tensors must match in dtype and hold a block, or a block per rank");
  const double scale = PyFloat_AsDouble(a[5]);
  const int channels = static_cast<int>(PyLong_AsLong(a[6]));
  void* stream;
  if (PyErr_Occurred() || !ToStream(Py_None, -1, &stream)) return nullptr;
  int code;
  Py_BEGIN_ALLOW_THREADS;
  code = ibcomm_emu_rsag(w, all_gather, in.dtype, in.ptr, out.ptr, static_cast<size_t>(block), scale, channels, stream, 0);
  Py_END_ALLOW_THREADS;
  return Done(code);
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"set_error", SetError, METH_O, "set_error(exception_class)"},
    {"allreduce", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(Allreduce)), METH_FASTCALL, nullptr},
    {"copy_scale", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(CopyScale)), METH_FASTCALL, nullptr},
    {"emu_allreduce", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(EmuAllreduce)), METH_FASTCALL, nullptr},
    {"emu_rsag", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(EmuRsAg)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fastcall", "Collectives on CUDA tensors without ctypes.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&kModule); }
