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

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
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

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw Bad();
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.is_contiguous()) throw Bad();
  return t;
}
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

template <typename F> int without_gil(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  return rc;
}
template <typename F> PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const Bad&) {
    Py_RETURN_NONE;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
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
    const void* nw = nullptr;
    if (a[1] != Py_None) {
      const at::Tensor& t = tensor(a[1]);
      want(t.dim() == 1 && t.numel() == hidden && t.scalar_type() == x.scalar_type());
      nw = t.data_ptr();
    }
    const size_t gu = p_weight_size(inter, hidden, qt), dn = p_weight_size(hidden, inter, qt);
    want(gu && dn && bytes(wg) == gu && bytes(wu) == gu && bytes(wd) == dn);
    const float eps = real(a[7]);
    const at::Tensor y = at::empty(x.sizes(), x.options());
    void* st = stream();
    return result(without_gil([&] { return p_mlp_block(x.data_ptr(), nw, wg.data_ptr(), wu.data_ptr(), wd.data_ptr(), y.data_ptr(), M, hidden, inter, qt, eps, dt, st); }), y);
  });
}

// q_gemm_dequant(input, weights, M, N, K, quant_type, group_size, bias)
PyObject* q_gemm_dequant(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want(n == 8);
    const at::Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    const int M = integer(a[2]), N = integer(a[3]), K = integer(a[4]), qt = integer(a[5]), gs = integer(a[6]), dt = dtype_code(x);
    want(x.dim() == 2 && x.size(0) == M && x.size(1) == K);
    const void* b = nullptr;
    if (a[7] != Py_None) {
      const at::Tensor& t = tensor(a[7]);
      want(t.dim() == 1 && t.size(0) == N && t.scalar_type() == x.scalar_type());
      b = t.data_ptr();
    }
    const size_t need = p_weight_size(N, K, qt);
    want(need && bytes(w) >= need);
    const at::Tensor y = at::empty({M, N}, x.options());
    void* st = stream();
    return result(without_gil([&] { return p_q_gemm(x.data_ptr(), w.data_ptr(), b, y.data_ptr(), M, N, K, qt, gs, dt, st); }), y);
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
    const void* nw = a[1] == Py_None ? nullptr : tensor(a[1]).data_ptr();
    const float eps = real(a[12]);
    const at::Tensor q = at::empty({M, qh, hd}, x.options()), k = at::empty({M, kh, hd}, x.options()), v = at::empty({M, kh, hd}, x.options());
    void* st = stream();
    const int rc = without_gil([&] {
      return p_qkv_rope(x.data_ptr(), nw, wq.data_ptr(), wk.data_ptr(), wv.data_ptr(), (const uint16_t*)cs.data_ptr(), (const uint16_t*)sn.data_ptr(),
                        (const int32_t*)pos.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), M, hidden, qh, kh, hd, (int)cs.size(0), qt, eps, off, dt, st);
    });
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
    const void* r = a[3] == Py_None ? nullptr : tensor(a[3]).data_ptr();
    const float eps = real(a[2]);
    const int hidden = (int)w.numel(), rows = (int)(x.numel() / hidden);
    const at::Tensor y = at::empty(x.sizes(), x.options());
    void* st = stream();
    return result(without_gil([&] { return p_rmsnorm(x.data_ptr(), w.data_ptr(), r, y.data_ptr(), rows, hidden, eps, dt, st); }), y);
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
    return result(without_gil([&] { return p_swiglu(g.data_ptr(), u.data_ptr(), y.data_ptr(), (size_t)g.numel(), dt, st); }), y);
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
    for (const at::Tensor* t : {&cs, &sn}) want(t->dim() == 2 && t->size(1) == hd / 2 && t->scalar_type() == at::kHalf);
    if (seq == 1) want(pos.dim() == 1 && pos.size(0) == batch);
    else want(pos.dim() == 2 && pos.size(0) == batch && pos.size(1) == seq);
    want(pos.scalar_type() == at::kInt);
    const at::Tensor y = inplace ? x : at::empty(x.sizes(), x.options());
    void* st = stream();
    return result(without_gil([&] {
                    return p_rope(x.data_ptr(), (const uint16_t*)cs.data_ptr(), (const uint16_t*)sn.data_ptr(), (const int32_t*)pos.data_ptr(), y.data_ptr(), batch, seq,
                                  heads, hd, (int)cs.size(0), mode, scale, off, dt, check ? 1 : 0, st);
                  }), y);
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
