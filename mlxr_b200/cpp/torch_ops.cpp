// The operators of mlxr_b200/ops.py for the arguments they are called with in a loop: one native call from
// Python objects to the C ABI.  At decode sizes a kernel takes 5 to 30 us and the interpreted wrapper
// (attribute checks, shape tuples, ctypes marshalling: 19 to 31 us a call) was what a stream of calls
// waited for.
//
// Every function returns the result, or the C ABI's status as an int, or None when an argument is not
// plainly valid (wrong type, shape, device, not contiguous): the caller then runs the interpreted
// wrapper, which owns the error messages.  Nothing is computed here.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <climits>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/mlxr_b200.h"

namespace {

// the entry points, bound to the library that the package has loaded
decltype(&mlxr_quantized_weight_size) p_weight_size;
decltype(&mlxr_mlp_block) p_mlp_block;
decltype(&mlxr_q_gemm_dequant) p_q_gemm;
decltype(&mlxr_qkv_rope) p_qkv_rope;
decltype(&mlxr_rmsnorm) p_rmsnorm;
decltype(&mlxr_rope_apply) p_rope;
decltype(&mlxr_swiglu) p_swiglu;

struct Bad {};   // not plainly valid: leave it to the interpreted wrapper

// A plain tensor with memory on the current device.  Subclasses (whose type the wrapper's results keep) and the
// wrappers of vmap, torch.func.grad and fake tensors (which have no memory to point at) are not plain.
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) throw Bad();
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || !t.is_contiguous() || t.get_device() != c10::cuda::current_device()) throw Bad();
  return t;
}
const at::Tensor* optional(PyObject* o) { return o == Py_None ? nullptr : &tensor(o); }
const void* data(const at::Tensor* t) { return t ? t->const_data_ptr() : nullptr; }
int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return MLXR_F16;
    case at::kBFloat16: return MLXR_BF16;
    case at::kFloat: return MLXR_F32;
    default: throw Bad();
  }
}
int integer(PyObject* o) {
  if (!PyLong_Check(o)) throw Bad();   // QuantType members are ints
  int over = 0;
  const long v = PyLong_AsLongAndOverflow(o, &over);
  if (over || v != (int)v) throw Bad();
  return (int)v;
}
float real(PyObject* o) {
  if (PyFloat_Check(o)) return (float)PyFloat_AS_DOUBLE(o);
  return (float)integer(o);
}
size_t bytes(const at::Tensor& t) { return (size_t)t.numel() * t.element_size(); }
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
void want(bool ok) { if (!ok) throw Bad(); }

// Pointers are taken before: nothing that can throw runs without the interpreter lock.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};
template <typename F> int without_gil(F&& f) {
  NoGil released;
  return f();
}
// torch's own translation of C++ exceptions (an allocation that fails stays a torch.OutOfMemoryError)
template <typename F> PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  try {
    return f();
  } catch (const Bad&) {
    Py_RETURN_NONE;
  }
  END_HANDLE_TH_ERRORS
}
PyObject* result(int rc, const at::Tensor& y) { return rc == MLXR_OK ? THPVariable_Wrap(y) : PyLong_FromLong(rc); }

// mlp_block(x, norm_weight, w_gate, w_up, w_down, inter, quant_type, eps)
PyObject* mlp_block(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 8);
    const at::Tensor &x = tensor(a[0]), &wg = tensor(a[2]), &wu = tensor(a[3]), &wd = tensor(a[4]);
    const int inter = integer(a[5]), qt = integer(a[6]), dt = dtype_code(x);
    want(x.dim() == 2);
    const int M = (int)x.size(0), hidden = (int)x.size(1);
    const at::Tensor* norm = optional(a[1]);
    if (norm) want(norm->dim() == 1 && norm->numel() == hidden && norm->scalar_type() == x.scalar_type());
    const size_t gu = p_weight_size(inter, hidden, qt), dn = p_weight_size(hidden, inter, qt);
    want(gu && dn && bytes(wg) == gu && bytes(wu) == gu && bytes(wd) == dn);
    const float eps = real(a[7]);
    const at::Tensor y = at::empty(x.sizes(), x.options());
    void* st = stream();
    const void *xp = data(&x), *np = data(norm), *gp = data(&wg), *up = data(&wu), *dp = data(&wd);
    void* yp = y.data_ptr();
    return result(without_gil([&] { return p_mlp_block(xp, np, gp, up, dp, yp, M, hidden, inter, qt, eps, dt, st); }), y);
  });
}

// q_gemm_dequant(input, weights, M, N, K, quant_type, group_size, bias)
PyObject* q_gemm_dequant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 8);
    const at::Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    const int M = integer(a[2]), N = integer(a[3]), K = integer(a[4]), qt = integer(a[5]), gs = integer(a[6]), dt = dtype_code(x);
    want(x.dim() == 2 && x.size(0) == M && x.size(1) == K);
    const at::Tensor* bias = optional(a[7]);
    if (bias) want(bias->dim() == 1 && bias->size(0) == N && bias->scalar_type() == x.scalar_type());
    const size_t need = p_weight_size(N, K, qt);
    want(need && bytes(w) >= need);
    const at::Tensor y = at::empty({M, N}, x.options());
    void* st = stream();
    const void *xp = data(&x), *wp = data(&w), *bp = data(bias);
    void* yp = y.data_ptr();
    return result(without_gil([&] { return p_q_gemm(xp, wp, bp, yp, M, N, K, qt, gs, dt, st); }), y);
  });
}

// qkv_rope(x, norm_weight, wq, wk, wv, cos, sin, positions, q_heads, kv_heads, head_dim, quant_type, eps, position_offset)
PyObject* qkv_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 14);
    const at::Tensor &x = tensor(a[0]), &wq = tensor(a[2]), &wk = tensor(a[3]), &wv = tensor(a[4]), &cs = tensor(a[5]), &sn = tensor(a[6]), &pos = tensor(a[7]);
    const int qh = integer(a[8]), kh = integer(a[9]), hd = integer(a[10]), qt = integer(a[11]), off = integer(a[13]), dt = dtype_code(x);
    want(x.dim() == 2 && qh > 0 && kh > 0 && hd > 0 && cs.dim() == 2 && pos.scalar_type() == at::kInt && pos.numel() == x.size(0));
    const int M = (int)x.size(0), hidden = (int)x.size(1);
    const at::Tensor* norm = optional(a[1]);
    if (norm) want(norm->numel() >= hidden && norm->scalar_type() == x.scalar_type());
    want(hd % 2 == 0 && (long long)qh * hd <= INT_MAX && (long long)kh * hd <= INT_MAX);
    for (const at::Tensor* t : {&cs, &sn}) want(t->dim() == 2 && t->size(1) == hd / 2 && t->size(0) >= cs.size(0) && t->scalar_type() == at::kHalf);
    const size_t nq = p_weight_size(qh * hd, hidden, qt), nkv = p_weight_size(kh * hd, hidden, qt);
    want(nq && nkv && bytes(wq) >= nq && bytes(wk) >= nkv && bytes(wv) >= nkv);
    const float eps = real(a[12]);
    const at::Tensor q = at::empty({M, qh, hd}, x.options()), k = at::empty({M, kh, hd}, x.options()), v = at::empty({M, kh, hd}, x.options());
    void* st = stream();
    const void *xp = data(&x), *np = data(norm), *qw = data(&wq), *kw = data(&wk), *vw = data(&wv);
    const uint16_t *cp = (const uint16_t*)data(&cs), *sp = (const uint16_t*)data(&sn);
    const int32_t* pp = (const int32_t*)data(&pos);
    void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr();
    const int max_seq = (int)cs.size(0);
    const int rc = without_gil([&] { return p_qkv_rope(xp, np, qw, kw, vw, cp, sp, pp, qp, kp, vp, M, hidden, qh, kh, hd, max_seq, qt, eps, off, dt, st); });
    if (rc != MLXR_OK) return PyLong_FromLong(rc);
    PyObject* t = PyTuple_New(3);
    if (!t) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(q));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(k));
    PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(v));
    return t;
  });
}

// rmsnorm_fused(input, weight, eps, residual)
PyObject* rmsnorm_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 4);
    const at::Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    const int dt = dtype_code(x);
    want(x.dim() >= 1 && w.dim() == 1 && x.size(-1) == w.numel() && w.numel() > 0 && w.scalar_type() == x.scalar_type());
    const at::Tensor* res = optional(a[3]);
    if (res) want(res->numel() >= x.numel() && res->scalar_type() == x.scalar_type());
    const float eps = real(a[2]);
    const int hidden = (int)w.numel(), rows = (int)(x.numel() / hidden);
    const at::Tensor y = at::empty(x.sizes(), x.options());
    void* st = stream();
    const void *xp = data(&x), *wp = data(&w), *rp = data(res);
    void* yp = y.data_ptr();
    return result(without_gil([&] { return p_rmsnorm(xp, wp, rp, yp, rows, hidden, eps, dt, st); }), y);
  });
}

// swiglu(gate, up)
PyObject* swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 2);
    const at::Tensor &g = tensor(a[0]), &u = tensor(a[1]);
    const int dt = dtype_code(g);
    want(g.sizes() == u.sizes() && g.scalar_type() == u.scalar_type());
    const at::Tensor y = at::empty(g.sizes(), g.options());
    void* st = stream();
    const void *gp = data(&g), *up = data(&u);
    void* yp = y.data_ptr();
    const size_t count = (size_t)g.numel();
    return result(without_gil([&] { return p_swiglu(gp, up, yp, count, dt, st); }), y);
  });
}

// rope_apply(input, cos, sin, positions, scaling_mode, scale_factor, position_offset, inplace, check_positions)
PyObject* rope_apply(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 9);
    const at::Tensor &x = tensor(a[0]), &cs = tensor(a[1]), &sn = tensor(a[2]), &pos = tensor(a[3]);
    const int mode = integer(a[4]), off = integer(a[6]), dt = dtype_code(x);
    const float scale = real(a[5]);
    want(PyBool_Check(a[7]) && PyBool_Check(a[8]));
    const bool inplace = a[7] == Py_True, check = a[8] == Py_True;
    want(x.dim() == 3 || x.dim() == 4);
    const int batch = (int)x.size(0), seq = x.dim() == 4 ? (int)x.size(1) : 1, heads = (int)x.size(-2), hd = (int)x.size(-1);
    want(hd > 0 && hd % 2 == 0);
    for (const at::Tensor* t : {&cs, &sn}) want(t->dim() == 2 && t->size(1) == hd / 2 && t->size(0) >= cs.size(0) && t->scalar_type() == at::kHalf);
    if (seq == 1) want(pos.dim() == 1 && pos.size(0) == batch);
    else want(pos.dim() == 2 && pos.size(0) == batch && pos.size(1) == seq);
    want(pos.scalar_type() == at::kInt);
    const at::Tensor y = inplace ? x : at::empty(x.sizes(), x.options());
    void* st = stream();
    void* yp = y.data_ptr();           // in place: before x's, since it may give a lazily copied tensor memory of its own
    const void* xp = data(&x);
    const uint16_t *cp = (const uint16_t*)data(&cs), *sp = (const uint16_t*)data(&sn);
    const int32_t* pp = (const int32_t*)data(&pos);
    const int max_seq = (int)cs.size(0);
    return result(without_gil([&] { return p_rope(xp, cp, sp, pp, yp, batch, seq, heads, hd, max_seq, mode, scale, off, dt, check ? 1 : 0, st); }), y);
  });
}

// bind({name: address}): the C ABI's functions in the library the package has loaded
PyObject* bind(PyObject*, PyObject* d) {
  auto get = [&](const char* name) -> void* {
    PyObject* v = PyDict_Check(d) ? PyDict_GetItemString(d, name) : nullptr;
    return v ? PyLong_AsVoidPtr(v) : nullptr;
  };
  p_weight_size = (decltype(p_weight_size))get("mlxr_quantized_weight_size");
  p_mlp_block = (decltype(p_mlp_block))get("mlxr_mlp_block");
  p_q_gemm = (decltype(p_q_gemm))get("mlxr_q_gemm_dequant");
  p_qkv_rope = (decltype(p_qkv_rope))get("mlxr_qkv_rope");
  p_rmsnorm = (decltype(p_rmsnorm))get("mlxr_rmsnorm");
  p_rope = (decltype(p_rope))get("mlxr_rope_apply");
  p_swiglu = (decltype(p_swiglu))get("mlxr_swiglu");
  if (!p_weight_size || !p_mlp_block || !p_q_gemm || !p_qkv_rope || !p_rmsnorm || !p_rope || !p_swiglu) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "an entry point is missing");
    return nullptr;
  }
  Py_RETURN_NONE;
}

#define FAST(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(mlp_block), FAST(q_gemm_dequant), FAST(qkv_rope), FAST(rmsnorm_fused), FAST(swiglu), FAST(rope_apply),
                         {"bind", (PyCFunction)bind, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "mlxr_torch_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_mlxr_torch_ops(void) { return PyModule_Create(&module); }
