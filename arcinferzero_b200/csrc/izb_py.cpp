// Native side of the Python binding: the calls a decode step or a prompt chunk makes by the dozen.
//
// A ctypes call through the public C ABI costs about 14 us of host time in Python (a dozen argument conversions, the
// stream lookup through torch.cuda, torch.empty per output), more than most decode kernels run: a layer of a small model
// (eight calls) took 114 us on the host and 35 us on the GPU.  Here a call takes the tensors as they are, reads pointers
// and strides from them, allocates its outputs from torch's caching allocator and calls the same C entry point with the
// current stream: about 1 us beside the launch itself.
//
// The module holds no state but the entry points' addresses: bind() receives them from the loaded libizb200.so, so the
// one library (also a build named by IZB200_LIB) serves both the ctypes and the native calls.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/izb200.h"

namespace {

#define IZB_PY_CALLS(X) \
  X(izb_quantize_act) X(izb_swiglu_quant) X(izb_rmsnorm_quant) X(izb_add_norm_quant) X(izb_softcap_rows) X(izb_matmul) X(izb_quant_matmul) \
  X(izb_gemv) X(izb_gemm) X(izb_moe_route_ex) X(izb_moe_sort_ex) X(izb_moe_gateup) X(izb_moe_down) X(izb_moe_combine_ex)

struct Calls {
#define X(name) decltype(&name) name##_ = nullptr;
  IZB_PY_CALLS(X)
#undef X
} g;
PyObject* g_fail = nullptr;     // Python callable(status): raises
PyObject* g_address = nullptr;  // Python callable(object): the address of what is no torch tensor (a numpy array over pinned memory, ...)

// ---- arguments
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw torch::TypeError(std::string("expected a torch tensor, got ") + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
template <class T>
T* ptr(PyObject* o) {  // None = NULL
  if (o == Py_None) return nullptr;
  if (THPVariable_Check(o)) return static_cast<T*>(THPVariable_Unpack(o).data_ptr());
  PyObject* v = PyObject_CallOneArg(g_address, o);
  if (!v) throw python_error();
  void* p = PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  if (!p && PyErr_Occurred()) throw python_error();
  return static_cast<T*>(p);
}
int extent(PyObject* o, int d) {  // o.shape[d]
  if (THPVariable_Check(o)) return (int)THPVariable_Unpack(o).size(d);
  PyObject* shape = PyObject_GetAttrString(o, "shape");
  PyObject* v = shape ? PySequence_GetItem(shape, d) : nullptr;
  Py_XDECREF(shape);
  if (!v) throw python_error();
  const long n = PyLong_AsLong(v);
  Py_DECREF(v);
  if (n == -1 && PyErr_Occurred()) throw python_error();
  return (int)n;
}
// rows and columns, as `rows, columns = x.shape` unpacks them: other numbers of dimensions are a ValueError
const at::Tensor& matrix(PyObject* o) {
  const at::Tensor& t = tensor(o);
  TORCH_CHECK_VALUE(t.dim() == 2, "expected two dimensions, got ", t.dim());
  return t;
}
int num(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  if (v != (int)v) throw torch::TypeError("integer argument out of range: " + std::to_string(v));
  return (int)v;
}
float real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return (float)v;
}
izb_weight* weight(PyObject* o) {  // the handle's address, None = NULL
  if (o == Py_None) return nullptr;
  void* p = PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw python_error();
  return static_cast<izb_weight*>(p);
}
void count(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) throw torch::TypeError(std::to_string(n) + " arguments, " + std::to_string(want) + " expected");
}

at::Tensor empty(std::initializer_list<int64_t> size, at::ScalarType type, c10::Device dev) {
  if (dev.is_cuda()) return at::detail::empty_cuda(at::IntArrayRef(size), type, dev, std::nullopt);
  return at::empty(at::IntArrayRef(size), at::TensorOptions().dtype(type).device(dev));
}
// rows of the reference engine's padding (zero/engine.h:521-522)
int pad_rows(int m) { return m >= 128 ? (m + 127) / 128 * 128 : (m + 15) / 16 * 16; }
int rows_or_pad(PyObject* o, int64_t m) {
  const int v = o == Py_None ? 0 : num(o);
  return v ? v : pad_rows((int)m);
}

// ---- the call itself: without the interpreter lock, on the current stream of the current device
template <class F, class... A>
void call(F f, A... args) {
  void* st = c10::cuda::getCurrentCUDAStream().stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f(args..., st);
  Py_END_ALLOW_THREADS
  if (rc != 0) {
    PyObject* r = PyObject_CallFunction(g_fail, "i", rc);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "izb200 status %d", rc);
    throw python_error();
  }
}

PyObject* own(PyObject* o) { Py_INCREF(o); return o; }
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* tuple(std::initializer_list<PyObject*> items) {  // takes the references over
  PyObject* t = PyTuple_New((Py_ssize_t)items.size());
  Py_ssize_t i = 0;
  for (PyObject* o : items) PyTuple_SET_ITEM(t, i++, o);
  return t;
}

struct Quantised {
  at::Tensor aq, asc;
  // (one allocation for both: an allocator round trip is half a microsecond of a call's four)
  Quantised(int Mp, int64_t K, c10::Device dev) {
    const int64_t q_bytes = (Mp * K + 15) / 16 * 16;
    const at::Tensor both = empty({q_bytes + K / 32 * Mp * 4}, at::kByte, dev);
    auto part = [&](caffe2::TypeMeta type, int64_t rows, int64_t cols, int64_t first) {
      at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(both.storage()), both.key_set(), type);
      t.unsafeGetTensorImpl()->set_storage_offset(first);
      t.unsafeGetTensorImpl()->set_sizes_contiguous({rows, cols});
      return t;
    };
    aq = part(caffe2::TypeMeta::Make<int8_t>(), Mp, K, 0);
    asc = part(caffe2::TypeMeta::Make<float>(), K / 32, Mp, q_bytes / 4);
  }
  int8_t* q() { return static_cast<int8_t*>(aq.data_ptr()); }
  float* s() { return static_cast<float*>(asc.data_ptr()); }
};

#define FN(name) PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n)

// (x, Mp, want_absum, aq, asc, absum): aq None = allocate
FN(quantize_act) {
  HANDLE_TH_ERRORS
  count(n, 6);
  const at::Tensor& x = matrix(a[0]);
  const int M = (int)x.size(0), K = (int)x.size(1), Mp = rows_or_pad(a[1], M);
  if (a[3] != Py_None) {
    call(g.izb_quantize_act_, ptr<float>(a[0]), (int)x.stride(0), M, Mp, K, ptr<int8_t>(a[3]), ptr<float>(a[4]), ptr<int16_t>(a[5]));
    return tuple({own(a[3]), own(a[4]), own(a[5])});
  }
  Quantised o(Mp, K, x.device());
  at::Tensor sums;
  if (PyObject_IsTrue(a[2])) sums = empty({K / 16, Mp}, at::kShort, x.device());
  int16_t* ps = sums.defined() ? static_cast<int16_t*>(sums.data_ptr()) : nullptr;
  call(g.izb_quantize_act_, ptr<float>(a[0]), (int)x.stride(0), M, Mp, K, o.q(), o.s(), ps);
  return tuple({wrap(o.aq), wrap(o.asc), ps ? wrap(sums) : own(Py_None)});
  END_HANDLE_TH_ERRORS
}

// (gu, F, Mp, want_h)
FN(swiglu_quant) {
  HANDLE_TH_ERRORS
  count(n, 4);
  const at::Tensor& gu = tensor(a[0]);
  const int M = (int)gu.size(0), F = num(a[1]), Mp = rows_or_pad(a[2], M);
  Quantised o(Mp, F, gu.device());
  at::Tensor h;
  if (PyObject_IsTrue(a[3])) h = empty({M, F}, at::kFloat, gu.device());
  float* ph = h.defined() ? static_cast<float*>(h.data_ptr()) : nullptr;
  call(g.izb_swiglu_quant_, ptr<float>(a[0]), (int)gu.stride(0), 1, M, Mp, F, ph, o.q(), o.s(), nullptr);
  return tuple({wrap(o.aq), wrap(o.asc), ph ? wrap(h) : own(Py_None)});
  END_HANDLE_TH_ERRORS
}

// (x, w, eps, Mp, want_h)
FN(rmsnorm_quant) {
  HANDLE_TH_ERRORS
  count(n, 5);
  const at::Tensor& x = matrix(a[0]);
  const int M = (int)x.size(0), K = (int)x.size(1), Mp = rows_or_pad(a[3], M);
  const float eps = real(a[2]);
  Quantised o(Mp, K, x.device());
  at::Tensor h;
  if (PyObject_IsTrue(a[4])) h = empty({M, K}, at::kFloat, x.device());
  float* ph = h.defined() ? static_cast<float*>(h.data_ptr()) : nullptr;
  call(g.izb_rmsnorm_quant_, ptr<float>(a[0]), (int)x.stride(0), ptr<float>(a[1]), eps, M, Mp, K, ph, o.q(), o.s(), nullptr);
  return tuple({wrap(o.aq), wrap(o.asc), ph ? wrap(h) : own(Py_None)});
  END_HANDLE_TH_ERRORS
}

// (x, t, w, eps, s, w2, Mp)
FN(add_norm_quant) {
  HANDLE_TH_ERRORS
  count(n, 7);
  const at::Tensor& x = matrix(a[0]);
  const int M = (int)x.size(0), K = (int)x.size(1), Mp = rows_or_pad(a[6], M);
  const float eps = real(a[3]), s = real(a[4]);
  Quantised o(Mp, K, x.device());
  call(g.izb_add_norm_quant_, ptr<float>(a[0]), ptr<float>(a[1]), ptr<float>(a[2]), eps, s, ptr<float>(a[5]), M, Mp, K, o.q(), o.s(), nullptr);
  return tuple({wrap(o.aq), wrap(o.asc)});
  END_HANDLE_TH_ERRORS
}

// (c, rows, N, cap, off)
FN(softcap_rows) {
  HANDLE_TH_ERRORS
  count(n, 5);
  const at::Tensor& c = tensor(a[0]);
  const int rows = num(a[1]), N = num(a[2]), off = num(a[4]);
  const float cap = real(a[3]);
  call(g.izb_softcap_rows_, ptr<float>(a[0]), rows, (int)c.stride(0), off, N, cap);
  return own(a[0]);
  END_HANDLE_TH_ERRORS
}

// the output of a product: the caller's, or a new one of `rows` x `cols`
struct Out {
  at::Tensor made;
  PyObject* given;
  float* p;
  int ld;
  Out(PyObject* o, int rows, int cols, PyObject* like) : given(o) {  // (`like`: on whose device)
    if (o == Py_None) {
      made = empty({rows, cols}, at::kFloat, tensor(like).device());
      p = static_cast<float*>(made.data_ptr());
      ld = cols;
    } else {
      const at::Tensor& t = tensor(o);
      p = static_cast<float*>(t.data_ptr());
      ld = (int)t.stride(0);
    }
  }
  PyObject* result() { return given == Py_None ? wrap(made) : own(given); }
};

// (weight, N, mat, aq, asc, T, out, c_off, acc)
FN(matmul) {
  HANDLE_TH_ERRORS
  count(n, 9);
  izb_weight* w = weight(a[0]);
  const int mat = num(a[2]), T = num(a[5]), c_off = num(a[7]), acc = num(a[8]), Mp = extent(a[4], 1);
  Out o(a[6], Mp, num(a[1]), a[3]);
  call(g.izb_matmul_, w, mat, ptr<int8_t>(a[3]), ptr<float>(a[4]), nullptr, T, Mp, o.p, o.ld, c_off, acc);
  return o.result();
  END_HANDLE_TH_ERRORS
}

// (weight, N_out, K, x, T, Mp, out, c_off, acc, mat, aq, asc): aq None = allocate
FN(quant_matmul) {
  HANDLE_TH_ERRORS
  count(n, 12);
  izb_weight* w = weight(a[0]);
  const at::Tensor& x = tensor(a[3]);
  const int K = num(a[2]), T = num(a[4]), Mp = rows_or_pad(a[5], T), c_off = num(a[7]), acc = num(a[8]), mat = num(a[9]);
  at::Tensor aq, asc;
  if (a[10] == Py_None) {
    Quantised q(Mp, K, x.device());
    aq = q.aq;
    asc = q.asc;
  }
  Out o(a[6], Mp, num(a[1]), a[3]);
  int8_t* pq = aq.defined() ? static_cast<int8_t*>(aq.data_ptr()) : ptr<int8_t>(a[10]);
  float* ps = asc.defined() ? static_cast<float*>(asc.data_ptr()) : ptr<float>(a[11]);
  call(g.izb_quant_matmul_, w, mat, ptr<float>(a[3]), (int)x.stride(0), T, Mp, pq, ps, o.p, o.ld, c_off, acc);
  return tuple({o.result(), a[10] == Py_None ? wrap(aq) : own(a[10]), a[10] == Py_None ? wrap(asc) : own(a[11])});
  END_HANDLE_TH_ERRORS
}

// (weight, N, mat, aq, asc, T, out, c_off, acc)
FN(gemv) {
  HANDLE_TH_ERRORS
  count(n, 9);
  izb_weight* w = weight(a[0]);
  const int mat = num(a[2]), T = num(a[5]), c_off = num(a[7]), acc = num(a[8]), Mp = extent(a[4], 1);
  Out o(a[6], T, num(a[1]), a[3]);
  call(g.izb_gemv_, w, mat, ptr<int8_t>(a[3]), ptr<float>(a[4]), T, Mp, o.p, o.ld, c_off, acc);
  return o.result();
  END_HANDLE_TH_ERRORS
}

// (weight, N_out, mat, aq, asc, M, out, c_off, acc, impl): M 0 = all padded rows
FN(gemm) {
  HANDLE_TH_ERRORS
  count(n, 10);
  izb_weight* w = weight(a[0]);
  const int mat = num(a[2]), c_off = num(a[7]), acc = num(a[8]), impl = num(a[9]), Mp = extent(a[4], 1);
  const int m = a[5] == Py_None ? 0 : num(a[5]), M = m ? m : Mp;
  Out o(a[6], Mp, num(a[1]), a[3]);
  call(g.izb_gemm_, w, mat, ptr<int8_t>(a[3]), ptr<float>(a[4]), M, Mp, o.p, o.ld, c_off, acc, impl);
  return o.result();
  END_HANDLE_TH_ERRORS
}

// (logits, NU, shared_gate)
FN(moe_route) {
  HANDLE_TH_ERRORS
  count(n, 3);
  const at::Tensor& l = tensor(a[0]);
  const bool shared = PyObject_IsTrue(a[2]);
  const int T = (int)l.size(0), NE = (int)l.size(1) - (shared ? 1 : 0), NU = num(a[1]);
  const c10::Device dev = l.device();
  at::Tensor ids = empty({T, NU}, at::kInt, dev), wts = empty({T, NU}, at::kFloat, dev), counts = empty({NE}, at::kInt, dev), gate;
  if (shared) gate = empty({T}, at::kFloat, dev);
  float* pg = shared ? static_cast<float*>(gate.data_ptr()) : nullptr;
  call(g.izb_moe_route_ex_, ptr<float>(a[0]), (int)l.stride(0), T, NE, NU, static_cast<int32_t*>(ids.data_ptr()), static_cast<float*>(wts.data_ptr()),
                               static_cast<int32_t*>(counts.data_ptr()), pg);
  if (shared) return tuple({wrap(ids), wrap(wts), wrap(counts), wrap(gate)});
  return tuple({wrap(ids), wrap(wts), wrap(counts)});
  END_HANDLE_TH_ERRORS
}

// (ids, wts, counts, TM, e0, e1)
FN(moe_sort) {
  HANDLE_TH_ERRORS
  count(n, 6);
  const at::Tensor& ids = matrix(a[0]);
  const c10::Device dev = ids.device();
  const int T = (int)ids.size(0), NU = (int)ids.size(1), NE = extent(a[2], 0), TM = num(a[3]), e0 = num(a[4]), e1 = num(a[5]);
  const int S = T * NU, max_tiles = (TM > 0 ? (S + TM - 1) / TM : 0) + NE;
  at::Tensor offs = empty({NE + 1}, at::kInt, dev), tiles = empty({1 + 3 * (int64_t)max_tiles}, at::kInt, dev), stok = empty({S}, at::kInt, dev),
             swt = empty({S}, at::kFloat, dev), inv = empty({S}, at::kInt, dev);
  auto pi = [](at::Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); };
  call(g.izb_moe_sort_ex_, ptr<int32_t>(a[0]), ptr<float>(a[1]), ptr<int32_t>(a[2]), T, NE, NU, TM, e0, e1, pi(offs), pi(tiles), max_tiles, pi(stok),
                              static_cast<float*>(swt.data_ptr()), pi(inv));
  return tuple({wrap(offs), wrap(tiles), PyLong_FromLong(max_tiles), wrap(stok), wrap(swt), wrap(inv)});
  END_HANDLE_TH_ERRORS
}

// (wg, wu, N_out, aq, asc, tiles, max_tiles, TM, stok, S)
FN(moe_gateup) {
  HANDLE_TH_ERRORS
  count(n, 10);
  izb_weight *wg = weight(a[0]), *wu = weight(a[1]);
  const int N = num(a[2]), Mp = extent(a[4], 1), max_tiles = num(a[6]), TM = num(a[7]), S = num(a[9]);
  at::Tensor h = empty({S, N}, at::kFloat, tensor(a[3]).device());
  float* ph = static_cast<float*>(h.data_ptr());
  call(g.izb_moe_gateup_, wg, wu, ptr<int8_t>(a[3]), ptr<float>(a[4]), Mp, ptr<int32_t>(a[5]), max_tiles, TM, ptr<int32_t>(a[8]), ph);
  return wrap(h);
  END_HANDLE_TH_ERRORS
}

// (wd, N, hq, hsc, tiles, max_tiles, TM, swt, S)
FN(moe_down) {
  HANDLE_TH_ERRORS
  count(n, 9);
  izb_weight* w = weight(a[0]);
  const int N = num(a[1]), Sp = extent(a[3], 1), max_tiles = num(a[5]), TM = num(a[6]), S = num(a[8]);
  at::Tensor y = empty({S, N}, at::kFloat, tensor(a[2]).device());
  float* py = static_cast<float*>(y.data_ptr());
  call(g.izb_moe_down_, w, ptr<int8_t>(a[2]), ptr<float>(a[3]), Sp, ptr<int32_t>(a[4]), max_tiles, TM, ptr<float>(a[7]), py);
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// (x, y, inv, NU, sh, sgate, partial)
FN(moe_combine) {
  HANDLE_TH_ERRORS
  count(n, 7);
  const at::Tensor& x = matrix(a[0]);
  const int T = (int)x.size(0), E = (int)x.size(1), NU = num(a[3]), partial = PyObject_IsTrue(a[6]) ? 1 : 0;
  call(g.izb_moe_combine_ex_, ptr<float>(a[0]), ptr<float>(a[1]), ptr<int32_t>(a[2]), T, NU, E, ptr<float>(a[4]), ptr<float>(a[5]), partial);
  return own(a[0]);
  END_HANDLE_TH_ERRORS
}

// bind(fail, address, {"izb_...": address})
FN(bind) {
  HANDLE_TH_ERRORS
  count(n, 3);
#define X(name)                                                                    \
  {                                                                                \
    PyObject* v = PyDict_GetItemString(a[2], #name);                               \
    if (!v) throw torch::TypeError("bind: no address for " #name);             \
    g.name##_ = reinterpret_cast<decltype(&name)>(PyLong_AsVoidPtr(v));            \
    if (!g.name##_) throw torch::TypeError("bind: null address for " #name);   \
  }
  IZB_PY_CALLS(X)
#undef X
  Py_INCREF(a[0]);
  Py_INCREF(a[1]);
  g_fail = a[0];
  g_address = a[1];
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// names(): the entry points bind() wants
PyObject* names(PyObject*, PyObject*) {
  PyObject* l = PyList_New(0);
#define X(name)                                   \
  {                                               \
    PyObject* s = PyUnicode_FromString(#name);    \
    PyList_Append(l, s);                          \
    Py_DECREF(s);                                 \
  }
  IZB_PY_CALLS(X)
#undef X
  return l;
}

#define M(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {M(bind), M(quantize_act), M(swiglu_quant), M(rmsnorm_quant), M(add_norm_quant), M(softcap_rows), M(matmul), M(quant_matmul), M(gemv),
                         M(gemm), M(moe_route), M(moe_sort), M(moe_gateup), M(moe_down), M(moe_combine), {"names", names, METH_NOARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_izb_py", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__izb_py(void) { return PyModule_Create(&module); }
