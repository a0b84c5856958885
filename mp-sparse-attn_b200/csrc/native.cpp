// The short way from torch tensors into libmpsa.so: checks, output allocation and the C call of the three entry points that programs
// call most, in one step.  Up to the C call that took 8 - 11 us of the host's time through ctypes and struct, here 3: back to back, a pair
// of quantizers over 4500 tokens 16.5 -> 11.0 us, causal attention over 128 tokens 17.0 -> 11.0.  Outputs and workspaces come from torch's allocator through its dispatcher, as
// torch.empty does, and like there the interpreter's lock is released from the first of them to the end of the C call: an allocation may
// wait for the device, and a launch for room in its queue.  Operands that the one-launch paths do not take make a function return
// None, and the caller goes the long way; an error code of the C entry is returned as an int.
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <exception>
#include <optional>

#include "../../include/mpsa.h"

namespace {

decltype(&mpsa_attention_workspace) workspace_fn;
decltype(&mpsa_attention) attention_fn;
decltype(&mpsa_quant_pair) quant_pair_fn;
decltype(&mpsa_gemm_block_scaled) gemm_fn;
PyObject* out_of_memory = PyExc_MemoryError;              // torch.OutOfMemoryError

const at::ScalarType kOut[] = {at::kFloat, at::kHalf, at::kBFloat16, at::kFloat8_e5m2};

// Plain tensors only: a subclass may stand for something without memory of its own.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && t.has_storage() && t.layout() == at::kStrided ? &t : nullptr;
}

// 4-D, 16 bits, rows of the last dimension dense, everything 16-byte aligned
bool aligned16(const at::Tensor& t) {
  if (t.dim() != 4) return false;
  const auto s = t.strides();
  return s[3] == 1 && !((s[0] | s[1] | s[2]) & 7) && !(reinterpret_cast<uintptr_t>(t.data_ptr()) & 15);
}

int in_dtype(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16 ? 0 : t.scalar_type() == at::kHalf ? 1 : -1; }

at::Tensor dense(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor& like) { return at::empty(sizes, like.options().dtype(type).requires_grad(false)); }

// Other Python threads run while this lives.  (The caller's argument array keeps the tensors.)
struct Unlocked {
  PyThreadState* const state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// The operands' device for the time of a call: the usual case costs one look.
struct OnDevice {
  std::optional<c10::cuda::CUDAGuard> guard;
  explicit OnDevice(c10::DeviceIndex i) { if (c10::cuda::current_device() != i) guard.emplace(i); }
};

long long as_ll(PyObject* o) { return PyLong_AsLongLong(o); }

template <typename F>
PyObject* guarded(F f) {
  try {
    PyObject* r = f();
    if (r && PyErr_Occurred()) { Py_DECREF(r); return nullptr; }
    return r;
  } catch (const c10::OutOfMemoryError& e) {
    PyErr_SetString(out_of_memory, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  } catch (...) {
    PyErr_SetString(PyExc_RuntimeError, "mpsa: unknown error");
  }
  return nullptr;
}

bool counted(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n != want) PyErr_Format(PyExc_TypeError, "%s takes %zd arguments", name, want);
  return n == want;
}

PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!counted(n, 5, "init")) return nullptr;
  workspace_fn = reinterpret_cast<decltype(workspace_fn)>(PyLong_AsVoidPtr(a[0]));
  attention_fn = reinterpret_cast<decltype(attention_fn)>(PyLong_AsVoidPtr(a[1]));
  quant_pair_fn = reinterpret_cast<decltype(quant_pair_fn)>(PyLong_AsVoidPtr(a[2]));
  gemm_fn = reinterpret_cast<decltype(gemm_fn)>(PyLong_AsVoidPtr(a[3]));
  if (PyErr_Occurred()) return nullptr;
  Py_INCREF(a[4]);
  out_of_memory = a[4];
  Py_RETURN_NONE;
}

// attention(q, k, v, prepared, range_flag, status, out_dtype, causal, band, uniform, route, pv_mode, fp8_fmt, smooth_k, fp4_kind, q_scale, tau)
// k and v may be None: then prepared = (Hkv, Skv, Skv_pad, k8, k8_sf, k4, k4_sf, vt, vt8, v8_sf, vt4, v4_sf).
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!counted(n, 17, "attention")) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor* q = plain(a[0]);
    if (!q || !aligned16(*q)) Py_RETURN_NONE;
    mpsa_attention_args c = {};
    c.in_dtype = in_dtype(*q);
    if (c.in_dtype < 0) Py_RETURN_NONE;
    const auto size = q->sizes(), qs = q->strides();
    c.q = q->data_ptr();
    c.q_sb = qs[0]; c.q_sh = qs[1]; c.q_sl = qs[2];
    long long hkv, skv;
    if (a[1] == Py_None) {
      if (!PyTuple_CheckExact(a[3]) || PyTuple_GET_SIZE(a[3]) != 12) { PyErr_SetString(PyExc_TypeError, "attention: prepared operands missing"); return nullptr; }
      long long w[12];
      for (int i = 0; i < 12; ++i) w[i] = as_ll(PyTuple_GET_ITEM(a[3], i));
      hkv = w[0]; skv = w[1]; c.Skv_pad = (int)w[2];
      const void** p[] = {&c.k8, &c.k8_sf, &c.k4, &c.k4_sf, &c.vt, &c.vt8, &c.v8_sf, &c.vt4, &c.v4_sf};
      for (int i = 0; i < 9; ++i) *p[i] = reinterpret_cast<const void*>(w[3 + i]);
    } else {
      const at::Tensor *k = plain(a[1]), *v = plain(a[2]);
      if (!k || !v || k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || !aligned16(*k) || !aligned16(*v) ||
          k->sizes() != v->sizes() || k->size(0) != size[0] || k->size(3) != size[3] || k->get_device() != q->get_device() ||
          v->get_device() != q->get_device())
        Py_RETURN_NONE;
      const auto ks = k->strides(), vs = v->strides();
      c.k = k->data_ptr(); c.v = v->data_ptr();
      c.k_sb = ks[0]; c.k_sh = ks[1]; c.k_sl = ks[2];
      c.v_sb = vs[0]; c.v_sh = vs[1]; c.v_sl = vs[2];
      hkv = k->size(1); skv = k->size(2);
    }
    if (PyErr_Occurred()) return nullptr;
    const long long most = 0x7fffffff;
    for (const long long x : {(long long)size[0], (long long)size[1], (long long)size[2], (long long)size[3], hkv, skv})
      if (x > most) Py_RETURN_NONE;
    c.B = (int)size[0]; c.Hq = (int)size[1]; c.S = (int)size[2]; c.D = (int)size[3]; c.Hkv = (int)hkv; c.Skv = (int)skv;
    c.causal = (int)as_ll(a[7]);
    if ((c.Hkv > 0 && c.Hq % c.Hkv) || (c.causal && c.Skv < c.S)) Py_RETURN_NONE;
    c.status = static_cast<int*>(PyLong_AsVoidPtr(a[5]));
    c.out_dtype = (int)as_ll(a[6]);
    c.band = (int)as_ll(a[8]); c.uniform = (int)as_ll(a[9]); c.route = (int)as_ll(a[10]); c.pv_mode = (int)as_ll(a[11]);
    c.fp8_fmt = (int)as_ll(a[12]); c.smooth_k = (int)as_ll(a[13]); c.fp4_kind = (int)as_ll(a[14]);
    c.q_scale = (float)PyFloat_AsDouble(a[15]); c.tau = (float)PyFloat_AsDouble(a[16]);
    if (PyErr_Occurred()) return nullptr;
    if (c.out_dtype < 0 || c.out_dtype > 2) Py_RETURN_NONE;
    if (a[4] != Py_None) {
      if (!THPVariable_Check(a[4])) { PyErr_SetString(PyExc_TypeError, "attention: range_flag must be a tensor"); return nullptr; }
      c.range_flag = static_cast<int*>(THPVariable_Unpack(a[4]).data_ptr());
    }
    at::Tensor out;
    long long rc;
    {
      const Unlocked unlocked;
      const OnDevice device(q->device().index());
      rc = workspace_fn(&c);                            // (refuses empty operands)
      if (rc >= 0) {
        const at::Tensor ws = dense({(int64_t)rc}, at::kByte, *q);
        out = dense(size, kOut[c.out_dtype], *q);
        c.out = out.data_ptr(); c.workspace = ws.data_ptr(); c.workspace_bytes = rc;
        rc = attention_fn(&c, c10::cuda::getCurrentCUDAStream(q->device().index()).stream());
      }
    }
    return rc ? PyLong_FromLongLong(rc) : THPVariable_Wrap(std::move(out));
  });
}

// quant_pair(q, k, q_scale, k_scale, fmt, hnd) -> (q codes, q scales, k codes, k scales)
PyObject* quant_pair(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!counted(n, 6, "quant_pair")) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor* x[2] = {plain(a[0]), plain(a[1])};
    if (!x[0] || !x[1] || !aligned16(*x[0]) || !aligned16(*x[1]) || x[0]->scalar_type() != x[1]->scalar_type() || x[0]->size(0) != x[1]->size(0) ||
        x[0]->size(3) != x[1]->size(3) || x[0]->get_device() != x[1]->get_device())
      Py_RETURN_NONE;
    mpsa_quant_pair_args c = {};
    c.in_dtype = in_dtype(*x[0]);
    const int64_t B = x[0]->size(0), D = x[0]->size(3);
    c.s[0] = (float)PyFloat_AsDouble(a[2]); c.s[1] = (float)PyFloat_AsDouble(a[3]);
    c.fp8_fmt = (int)as_ll(a[4]);
    const int hnd = PyObject_IsTrue(a[5]);
    if (PyErr_Occurred()) return nullptr;
    if (c.in_dtype < 0 || !(D == 64 || (D > 0 && D % 128 == 0)) || D > 0x7fffffff || B > 0x7fffffff || !(c.s[0] > 0.0f) || !(c.s[1] > 0.0f) ||
        c.fp8_fmt < 0 || c.fp8_fmt > 2)
      Py_RETURN_NONE;
    c.B = (int)B; c.D = (int)D;
    for (const at::Tensor* t : x)
      if (t->size(1) > 0x7fffffff || t->size(2) > 0x7fffffff) Py_RETURN_NONE;
    at::Tensor codes[2], scales[2];
    int rc;
    {
      const Unlocked unlocked;
      const OnDevice device(x[0]->device().index());
      const at::ScalarType type = c.fp8_fmt == 0 ? at::kByte : c.fp8_fmt == 1 ? at::kFloat8_e5m2 : at::kFloat8_e4m3fn;
      for (int i = 0; i < 2; ++i) {
        const auto z = x[i]->sizes(), st = x[i]->strides();
        const int h = hnd ? 1 : 2, l = hnd ? 2 : 1;       // where heads and length are
        codes[i] = dense(z, type, *x[i]);
        scales[i] = dense({B, z[h], z[l], D / 32}, at::kByte, *x[i]);
        const auto cs = codes[i].strides();
        c.x[i] = x[i]->data_ptr(); c.codes[i] = codes[i].data_ptr(); c.scales[i] = scales[i].data_ptr();
        c.H[i] = (int)z[h]; c.L[i] = (int)z[l];
        c.x_sb[i] = st[0]; c.x_sh[i] = st[h]; c.x_sl[i] = st[l];
        c.c_sb[i] = cs[0]; c.c_sh[i] = cs[h]; c.c_sl[i] = cs[l];
      }
      rc = quant_pair_fn(&c, c10::cuda::getCurrentCUDAStream(x[0]->device().index()).stream());
    }
    if (rc) return PyLong_FromLong(rc);
    PyObject* r = PyTuple_New(4);
    if (!r) return nullptr;
    for (int i = 0; i < 2; ++i) {
      PyTuple_SET_ITEM(r, 2 * i, THPVariable_Wrap(std::move(codes[i])));
      PyTuple_SET_ITEM(r, 2 * i + 1, THPVariable_Wrap(std::move(scales[i])));
    }
    return r;
  });
}

// gemm(a, a_scale, b, b_scale, M, N, K, mode, a_fmt, b_fmt, out_dtype, alpha, status)
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!counted(n, 13, "gemm")) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor *x = plain(a[0]), *xs = plain(a[1]), *y = plain(a[2]), *ys = plain(a[3]);
    if (!x || !xs || !y || !ys || x->dim() < 2 || y->dim() < 2 || x->stride(-1) != 1 || y->stride(-1) != 1 || !xs->is_contiguous() || !ys->is_contiguous())
      Py_RETURN_NONE;
    long long w[7];
    for (int i = 0; i < 7; ++i) w[i] = as_ll(a[4 + i]);
    const double alpha = PyFloat_AsDouble(a[11]);
    int* const status = static_cast<int*>(PyLong_AsVoidPtr(a[12]));
    if (PyErr_Occurred()) return nullptr;
    for (int i = 0; i < 3; ++i)
      if (w[i] <= 0 || w[i] > 0x7fffffff) Py_RETURN_NONE;
    if (w[6] < 0 || w[6] > 3) Py_RETURN_NONE;
    at::Tensor c;
    int rc;
    {
      const Unlocked unlocked;
      const OnDevice device(x->device().index());
      c = dense({(int64_t)w[0], (int64_t)w[1]}, kOut[w[6]], *x);
      rc = gemm_fn(x->data_ptr(), xs->data_ptr(), y->data_ptr(), ys->data_ptr(), c.data_ptr(), (int)w[0], (int)w[1], (int)w[2],
                   x->stride(0) * x->element_size(), y->stride(0) * y->element_size(), w[1], (int)w[3], (int)w[4], (int)w[5], (int)w[6],
                   (float)alpha, status, c10::cuda::getCurrentCUDAStream(x->device().index()).stream());
    }
    return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(c));
  });
}

PyMethodDef methods[] = {
    {"init", (PyCFunction)(void*)init, METH_FASTCALL, "addresses of mpsa_attention_workspace, mpsa_attention, mpsa_quant_pair, mpsa_gemm_block_scaled; torch.OutOfMemoryError"},
    {"attention", (PyCFunction)(void*)attention, METH_FASTCALL, "one attention call: output tensor, None (operands not taken) or an error code"},
    {"quant_pair", (PyCFunction)(void*)quant_pair, METH_FASTCALL, "two operands quantised: four tensors, None or an error code"},
    {"gemm", (PyCFunction)(void*)gemm, METH_FASTCALL, "block-scaled product: output tensor, None or an error code"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "torch tensors into libmpsa.so", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
