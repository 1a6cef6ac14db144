// Host side of the launches, native: a CPython module (`_b200_host.so`) that `ops/_lib.py` and `ops/kernels.py` use when it is there.
//
//   bind(table, last_error, fallback)   name -> (address, argument codes) of the launchers of the kernel library
//   call(name, *args)                   converts the arguments by their codes, calls the launcher with the GIL released and raises
//                                       RuntimeError on a code other than 0
//   gemm(...)                           ops.kernels.gemm for CUDA operands that need no copy: checks, output, split workspace, launch
//
// ctypes converts twenty arguments through as many Python objects and calls: 5 of the 20 us a launch of a small model took.  With
// it, the native GEMM operator and no autograd nodes where no gradient is wanted: a step of a two-layer model of width 512 2020 ->
// 1625 us, sampling with one double and two single MMDiT blocks 1668 -> 1012 us.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <unordered_map>

namespace {

constexpr int MAX_INTS = 40, MAX_FLOATS = 8;

struct Entry {
  void* fn;
  std::string codes;             // P pointer, I int, L long long, U unsigned long long, F float
};
std::unordered_map<PyObject*, Entry> g_table;        // by interned name
const char* (*g_last_error)() = nullptr;
PyObject* g_fallback = nullptr;                      // the ctypes call, for arguments this module does not convert

// x86-64 System V: integer and pointer arguments fill their registers and then the stack in order, float arguments their own
// registers, independently of how the two mix; surplus arguments are ignored by the callee.  So one signature calls every launcher.
#if !defined(__x86_64__) || defined(_WIN32)
#error "the launcher trampoline is written for the x86-64 System V calling convention"
#endif
using Fn = int (*)(float, float, float, float, float, float, float, float,
                   long long, long long, long long, long long, long long, long long, long long, long long, long long, long long,
                   long long, long long, long long, long long, long long, long long, long long, long long, long long, long long,
                   long long, long long, long long, long long, long long, long long, long long, long long, long long, long long,
                   long long, long long, long long, long long, long long, long long, long long, long long, long long, long long);

int invoke(void* fn, const float* f, const long long* a) {
  return reinterpret_cast<Fn>(fn)(f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7],
      a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15], a[16], a[17], a[18], a[19],
      a[20], a[21], a[22], a[23], a[24], a[25], a[26], a[27], a[28], a[29], a[30], a[31], a[32], a[33], a[34], a[35], a[36], a[37],
      a[38], a[39]);
}

PyObject* raise_code(const char* name, int rc) {
  PyErr_Format(PyExc_RuntimeError, "%s failed with code %d: %s", name, rc, g_last_error ? g_last_error() : "");
  return nullptr;
}

const Entry* find(PyObject* name) {
  auto it = g_table.find(name);
  if (it != g_table.end()) return &it->second;
  if (!PyUnicode_Check(name)) return nullptr;
  PyObject* s = name;
  Py_INCREF(s);
  PyUnicode_InternInPlace(&s);
  it = g_table.find(s);
  Py_DECREF(s);
  return it == g_table.end() ? nullptr : &it->second;
}

PyObject* py_call(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs < 1) { PyErr_SetString(PyExc_TypeError, "call(name, *args)"); return nullptr; }
  const Entry* e = find(args[0]);
  if (e == nullptr || (Py_ssize_t)e->codes.size() != nargs - 1) return PyObject_Vectorcall(g_fallback, args, nargs, nullptr);
  float f[MAX_FLOATS] = {};
  long long a[MAX_INTS] = {};
  int nf = 0, na = 0;
  for (Py_ssize_t i = 1; i < nargs; ++i) {
    PyObject* o = args[i];
    const char c = e->codes[i - 1];
    if (c == 'F') {
      const double v = PyFloat_AsDouble(o);
      if (v == -1.0 && PyErr_Occurred()) return nullptr;
      f[nf++] = (float)v;
    } else if (o == Py_None && c == 'P') {
      a[na++] = 0;
    } else if (PyLong_Check(o)) {                    // (bool is one)
      a[na] = (long long)PyLong_AsUnsignedLongLongMask(o);           // wraps, as ctypes does
      if (c == 'I') a[na] = (int)a[na];
      if (a[na] == -1 && PyErr_Occurred()) return nullptr;
      ++na;
    } else {
      return PyObject_Vectorcall(g_fallback, args, nargs, nullptr);  // arrays of pointers and the like
    }
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = invoke(e->fn, f, a);
  Py_END_ALLOW_THREADS
  if (rc != 0) return raise_code(PyUnicode_AsUTF8(args[0]), rc);
  Py_RETURN_NONE;
}

// bind({name: (address, codes)}, address of b200_last_error, fallback)
PyObject* py_bind(PyObject*, PyObject* args) {
  PyObject *table, *fallback;
  unsigned long long last;
  if (!PyArg_ParseTuple(args, "O!KO", &PyDict_Type, &table, &last, &fallback)) return nullptr;
  PyObject *key, *val;
  Py_ssize_t pos = 0;
  std::unordered_map<PyObject*, Entry> t;
  while (PyDict_Next(table, &pos, &key, &val)) {
    unsigned long long addr;
    const char* codes;
    if (!PyArg_ParseTuple(val, "Ks", &addr, &codes)) return nullptr;
    int nf = 0, na = 0;
    for (const char* c = codes; *c; ++c) (*c == 'F' ? nf : na)++;
    if (nf > MAX_FLOATS || na > MAX_INTS) continue;                  // left to the fallback
    Py_INCREF(key);
    PyUnicode_InternInPlace(&key);
    t[key] = Entry{reinterpret_cast<void*>(addr), codes};
  }
  g_table = std::move(t);
  g_last_error = reinterpret_cast<const char* (*)()>(last);
  Py_INCREF(fallback);
  Py_XDECREF(g_fallback);
  g_fallback = fallback;
  Py_RETURN_NONE;
}

using GemmFn = int (*)(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, int, const void*,
                       const void*, long long, float, void*, long long, void*);
using WorkFn = long long (*)(int, int, int);
GemmFn g_gemm = nullptr;
WorkFn g_gemm_ws = nullptr;
thread_local std::unordered_map<unsigned long long, long long> t_ws;   // (device, M, N, K) -> bytes; bounded below

// rows that the GEMM's tensor maps take as they are
bool plain(const at::Tensor& t) {
  return t.dim() == 2 && t.stride(1) == 1 && (t.stride(0) & 7) == 0 && t.stride(0) >= t.size(1) &&
         (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}

// gemm(a, b, a_mn_major, b_mn_major, out, out_fp32, accumulate, bias, residual, alpha): the result, or None where the general
// path has to look at the operands (copies, errors).
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 10 || g_gemm == nullptr) Py_RETURN_NONE;
  for (int i : {0, 1})
    if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
  const at::Tensor &a = THPVariable_Unpack(args[0]), &b = THPVariable_Unpack(args[1]);
  const bool a_mn = PyObject_IsTrue(args[2]) == 1, b_mn = PyObject_IsTrue(args[3]) == 1, acc = PyObject_IsTrue(args[6]) == 1;
  bool f32 = PyObject_IsTrue(args[5]) == 1;
  if (PyErr_Occurred()) return nullptr;
  if (!a.is_cuda() || !b.is_cuda() || a.scalar_type() != at::kBFloat16 || b.scalar_type() != at::kBFloat16 || !plain(a) || !plain(b) ||
      a.device() != b.device())
    Py_RETURN_NONE;
  const int64_t M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0);
  if (K != b.size(b_mn ? 0 : 1) || M <= 0 || N <= 0 || K <= 0 || M > 0x7fffffff || N > 0x7fffffff || K > 0x7fffffff) Py_RETURN_NONE;
  const int dev = a.device().index();
  if (c10::cuda::current_device() != dev) Py_RETURN_NONE;
  const bool has_out = args[4] != Py_None;
  at::Tensor out;
  if (has_out) {
    if (!THPVariable_Check(args[4])) Py_RETURN_NONE;
    out = THPVariable_Unpack(args[4]);
    const auto ty = out.scalar_type();
    if (!out.is_cuda() || out.dim() != 2 || out.size(0) != M || out.size(1) != N || out.stride(1) != 1 ||
        (ty != at::kBFloat16 && ty != at::kFloat) || (out.stride(0) * (int64_t)out.element_size()) % 16 != 0 ||
        (reinterpret_cast<uintptr_t>(out.data_ptr()) & 15) != 0)
      Py_RETURN_NONE;
    f32 = ty == at::kFloat;
  } else if (acc || N * (f32 ? 4 : 2) % 16 != 0) {
    Py_RETURN_NONE;
  }
  const void *bias = nullptr, *res = nullptr;
  long long ldr = 0;
  if (args[7] != Py_None) {
    if (!THPVariable_Check(args[7])) Py_RETURN_NONE;
    const at::Tensor& t = THPVariable_Unpack(args[7]);
    if (!t.is_cuda() || t.scalar_type() != at::kBFloat16 || !t.is_contiguous()) Py_RETURN_NONE;
    bias = t.data_ptr();
  }
  if (args[8] != Py_None) {
    if (!THPVariable_Check(args[8])) Py_RETURN_NONE;
    const at::Tensor& t = THPVariable_Unpack(args[8]);
    if (!t.is_cuda() || t.dim() != 2 || t.scalar_type() != at::kBFloat16 || t.stride(1) != 1) Py_RETURN_NONE;
    res = t.data_ptr();
    ldr = t.stride(0);
  }
  const double alpha = PyFloat_AsDouble(args[9]);
  if (alpha == -1.0 && PyErr_Occurred()) return nullptr;
  long long ws_bytes;
  if (M < (1 << 20) && N < (1 << 20) && K < (1 << 20) && dev < 16) {
    // (the answer depends on the shape and the device alone)
    const unsigned long long key = ((unsigned long long)dev << 60) | ((unsigned long long)M << 40) | ((unsigned long long)N << 20) | (unsigned long long)K;
    auto it = t_ws.find(key);
    if (it == t_ws.end()) {
      if (t_ws.size() > 4096) t_ws.clear();
      it = t_ws.emplace(key, g_gemm_ws((int)M, (int)N, (int)K)).first;
    }
    ws_bytes = it->second;
  } else {
    ws_bytes = g_gemm_ws((int)M, (int)N, (int)K);
  }
  int rc;
  {
    pybind11::gil_scoped_release nogil;
    if (!has_out) out = at::empty({M, N}, a.options().dtype(f32 ? at::kFloat : at::kBFloat16).requires_grad(false));
    at::Tensor ws;
    if (ws_bytes > 0) ws = at::empty({ws_bytes}, a.options().dtype(at::kByte).requires_grad(false));
    rc = g_gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), (int)M, (int)N, (int)K, a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn,
                f32, acc, bias, res, ldr, (float)alpha, ws_bytes > 0 ? ws.data_ptr() : nullptr, ws_bytes,
                c10::cuda::getCurrentCUDAStream(dev).stream());
  }
  if (rc != 0) return raise_code("b200_gemm_bf16", rc);
  if (has_out) { Py_INCREF(args[4]); return args[4]; }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind_gemm(address of b200_gemm_bf16, address of b200_gemm_bf16_workspace)
PyObject* py_bind_gemm(PyObject*, PyObject* args) {
  unsigned long long g, w;
  if (!PyArg_ParseTuple(args, "KK", &g, &w)) return nullptr;
  g_gemm = reinterpret_cast<GemmFn>(g);
  g_gemm_ws = reinterpret_cast<WorkFn>(w);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, nullptr},
    {"bind_gemm", py_bind_gemm, METH_VARARGS, nullptr},
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_call)), METH_FASTCALL, nullptr},
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_gemm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200_host(void) { return PyModule_Create(&module); }
