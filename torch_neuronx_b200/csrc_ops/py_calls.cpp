// Direct Python entry points: the calls of a generation loop (attention over key lengths, decode against a dense or
// paged cache, a chunk behind a cached prefix) go from Python into the C ABI in one foreign call.
//
// The small calls of this package take 10-20 us on the GPU; through the ctypes binding the host needed 24 us
// (sdpa_forward) to 52 us (scaled_dot_product_attention with kv_lens) to enqueue one, so the GPU waited.  Here the
// whole call -- checks, output and scratch allocation, parameter block, launch -- is native.
//
// Every function returns None when the call is not one of the plain ones it serves (subclasses, active modes and
// transforms, tracing, forward-mode tangents, gradients, other dtypes, anything malformed); the Python layer then takes its own path, which serves the rest and
// raises the errors.  So nothing here raises for a bad argument.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/grad_mode.h>
#include <ATen/ops/_scaled_dot_product_fused_attention_overrideable.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>

#include "ops_common.h"

namespace {

using namespace b200_ops;

struct NoGil {   // the interpreter lock is released for the lifetime of the object
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// The record of the last forward's plan: the dict of the Python layer, filled under the interpreter lock.
PyObject* g_plan_record = nullptr;

bool record_plan(const B200SdpaPlan& plan) {
  if (g_plan_record == nullptr) return true;
  static PyObject* const names[] = {
      PyUnicode_InternFromString("path"),      PyUnicode_InternFromString("block_m"),    PyUnicode_InternFromString("block_n"),
      PyUnicode_InternFromString("grid"),      PyUnicode_InternFromString("threads"),    PyUnicode_InternFromString("smem_bytes"),
      PyUnicode_InternFromString("kv_splits"), PyUnicode_InternFromString("launches"),   PyUnicode_InternFromString("workspace_bytes")};
  static PyObject* const paths[] = {PyUnicode_InternFromString("auto"), PyUnicode_InternFromString("generic"),
                                    PyUnicode_InternFromString("prefill"), PyUnicode_InternFromString("decode")};
  PyObject* const values[] = {Py_NewRef(paths[plan.path & 3]),
                              PyLong_FromLong(plan.block_m),
                              PyLong_FromLong(plan.block_n),
                              Py_BuildValue("(iii)", plan.grid_x, plan.grid_y, plan.grid_z),
                              PyLong_FromLong(plan.threads),
                              PyLong_FromLong(plan.smem_bytes),
                              PyLong_FromLong(plan.kv_splits),
                              PyLong_FromLong(plan.launches),
                              PyLong_FromUnsignedLongLong(plan.workspace_bytes)};
  PyDict_Clear(g_plan_record);
  bool ok = true;
  for (int i = 0; i < 9; ++i) {
    ok = ok && values[i] != nullptr && PyDict_SetItem(g_plan_record, names[i], values[i]) == 0;
    Py_XDECREF(values[i]);
  }
  return ok;
}

// A plain strided CUDA tensor with nothing between it and the kernels; a dual tensor of forward-mode differentiation
// has the same keys but carries a tangent, which only the dispatcher's formulas see (and refuse).
bool plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  static const uint64_t expected = c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA,
                                                        c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutocastCUDA})
                                       .raw_repr();
  return t.is_cuda() && (t.key_set().raw_repr() & ~expected) == 0 && !t._fw_grad(/*level=*/0).defined();
}
// Nothing on this thread stands between a call and the CUDA kernels.  The modes written in Python have stacks of their
// own; whatever else wants to see every call (the tracer, functorch's transforms, functionalization) includes a
// dispatch key.  Those included by default and autocast's, which these operations do not listen to, may be there.
bool no_modes() {
  static const c10::DispatchKeySet harmless = c10::default_included_set | c10::autocast_dispatch_keyset;
  return !at::impl::torch_function_mode_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         (c10::impl::tls_local_dispatch_key_set().included_ - harmless).empty();
}
bool wants_grad(const at::Tensor& t) { return t.requires_grad(); }

// out := the tensor of `o`, or an undefined one for None; false when `o` is something else.
bool optional_plain(PyObject* o, at::Tensor* out) {
  if (o == Py_None) return true;
  if (!plain(o)) return false;
  *out = THPVariable_Unpack(o);
  return true;
}
bool as_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
bool as_bool(PyObject* o, bool* v) {
  if (!PyBool_Check(o)) return false;
  *v = o == Py_True;
  return true;
}
bool as_scale(PyObject* o, int64_t head_dim, float* v) {
  if (o == Py_None) {
    *v = static_cast<float>(1.0 / std::sqrt(static_cast<double>(head_dim)));
    return true;
  }
  if (!PyFloat_CheckExact(o)) return false;
  *v = static_cast<float>(PyFloat_AS_DOUBLE(o));
  return true;
}

// The rules of the Python layer's validation for one forward call.
bool shapes_ok(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v) {
  return q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && dtype_code(q.scalar_type()) >= 0 &&
         q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type() && q.device() == k.device() &&
         q.device() == v.device() && q.size(0) == k.size(0) && q.size(0) == v.size(0) && k.size(1) == v.size(1) &&
         k.size(2) == v.size(2) && q.size(3) == k.size(3) && k.size(1) != 0 && q.size(1) % k.size(1) == 0 &&
         q.numel() != 0 && k.size(3) != 0 && v.size(3) != 0;
}
bool lens_ok(const at::Tensor& lens, const at::Tensor& q) {
  return lens.scalar_type() == at::kInt && lens.device() == q.device() && lens.dim() == 1 && lens.size(0) == q.size(0) &&
         lens.is_contiguous();
}

void fill_common(B200SdpaParams& p, const at::Tensor& q, const at::Tensor& out, const at::Tensor& lse, int dev) {
  p.struct_size = sizeof(B200SdpaParams);
  p.dtype = dtype_code(q.scalar_type());
  p.device = dev;
  p.q = q.data_ptr();
  p.out = out.data_ptr();
  copy_strides(q, p.q_stride);
  copy_strides(out, p.out_stride);
  if (lse.defined()) {
    p.lse = lse.data_ptr<float>();
    copy_strides(lse, p.lse_stride);
  }
  p.B = static_cast<int32_t>(q.size(0));
  p.Hq = static_cast<int32_t>(q.size(1));
  p.L = static_cast<int32_t>(q.size(2));
  p.E = static_cast<int32_t>(q.size(3));
  p.status = device_state(dev).status.data_ptr<int32_t>();
}

// Plan, scratch, launch; the interpreter lock is not held.
void launch(B200SdpaParams& p, int dev, bool decode_only, B200SdpaPlan& plan) {
  at::Tensor ws;   // freed (stream-ordered) when the launch has been queued
  NoGil nogil;
  plan.struct_size = sizeof(B200SdpaPlan);
  int rc = b200_sdpa_query_plan(&p, &plan);
  TORCH_CHECK(rc == B200_SDPA_OK, "b200_sdpa_query_plan: ", b200_sdpa_strerror(rc));
  if (plan.workspace_bytes != 0) {
    ws = scratch(dev, plan.workspace_bytes);
    p.workspace = ws.data_ptr();
    p.workspace_bytes = static_cast<uint64_t>(ws.numel());
  }
  const auto stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  rc = decode_only ? b200_sdpa_decode(&p, stream) : b200_sdpa_fwd(&p, stream);
  TORCH_CHECK(rc == B200_SDPA_OK, decode_only ? "b200_sdpa_decode: " : "b200_sdpa_fwd: ", b200_sdpa_strerror(rc));
}

struct ForwardArgs {
  bool causal = false;
  float scale = 0.f;
  int64_t q_offset = 0, k_offset = 0, force_path = 0, kv_chunk = 0;
  at::Tensor lens;
};

// False: a Python error is set.
bool forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const ForwardArgs& a, const at::Tensor& out,
             const at::Tensor& lse) {
  const int dev = q.device().index();
  B200SdpaParams p{};
  fill_common(p, q, out, lse, dev);
  p.force_path = static_cast<int32_t>(a.force_path);
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  copy_strides(k, p.k_stride);
  copy_strides(v, p.v_stride);
  p.Hkv = static_cast<int32_t>(k.size(1));
  p.S = static_cast<int32_t>(k.size(2));
  p.Dv = static_cast<int32_t>(v.size(3));
  p.scale = a.scale;
  p.is_causal = a.causal ? 1 : 0;
  p.q_offset = a.q_offset;
  p.k_offset = a.k_offset;
  p.kv_chunk = static_cast<int32_t>(a.kv_chunk);
  if (a.lens.defined()) p.kv_lens = a.lens.data_ptr<int32_t>();
  B200SdpaPlan plan{};
  launch(p, dev, false, plan);
  return record_plan(plan);
}

#define NOT_SERVED() do { if (PyErr_Occurred()) PyErr_Clear(); Py_RETURN_NONE; } while (0)

// attention(query, key, value, is_causal, scale, enable_gqa, kv_lens) -> output or None
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ForwardArgs a;
  bool gqa = false;
  if (n != 7 || !plain(args[0]) || !plain(args[1]) || !plain(args[2]) || !as_bool(args[3], &a.causal) ||
      !as_bool(args[5], &gqa) || !optional_plain(args[6], &a.lens) || !no_modes())
    NOT_SERVED();
  const at::Tensor& q = THPVariable_Unpack(args[0]);
  const at::Tensor& k = THPVariable_Unpack(args[1]);
  const at::Tensor& v = THPVariable_Unpack(args[2]);
  if (!shapes_ok(q, k, v) || !as_scale(args[4], q.size(3), &a.scale)) NOT_SERVED();
  if (!gqa && q.size(1) != k.size(1)) NOT_SERVED();
  if (a.lens.defined() && !lens_ok(a.lens, q)) NOT_SERVED();
  at::Tensor out;
  if (at::GradMode::is_enabled() && (wants_grad(q) || wants_grad(k) || wants_grad(v))) {
    if (a.lens.defined()) NOT_SERVED();
    NoGil nogil;
    c10::optional<double> scale;
    if (args[4] != Py_None) scale = PyFloat_AS_DOUBLE(args[4]);
    out = std::get<0>(at::_scaled_dot_product_fused_attention_overrideable(q, k, v, c10::nullopt, 0.0, a.causal, false, scale));
  } else {
    const c10::cuda::CUDAGuard guard(q.device());
    out = alloc_like_query(q, {q.size(0), q.size(1), q.size(2), v.size(3)});
    if (!forward(q, k, v, a, out, at::Tensor())) return nullptr;
  }
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// forward(query, key, value, is_causal, scale, kv_lens, q_offset, k_offset, need_lse, out, lse, force_path, kv_chunk)
//   -> (out, lse or None), or None
PyObject* py_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  ForwardArgs a;
  bool need_lse = false;
  at::Tensor out, lse;
  if (n != 13 || !plain(args[0]) || !plain(args[1]) || !plain(args[2]) || !as_bool(args[3], &a.causal) ||
      !optional_plain(args[5], &a.lens) || !as_int(args[6], &a.q_offset) || !as_int(args[7], &a.k_offset) ||
      !as_bool(args[8], &need_lse) || !optional_plain(args[9], &out) || !optional_plain(args[10], &lse) ||
      !as_int(args[11], &a.force_path) || !as_int(args[12], &a.kv_chunk) || !no_modes())
    NOT_SERVED();
  const at::Tensor& q = THPVariable_Unpack(args[0]);
  const at::Tensor& k = THPVariable_Unpack(args[1]);
  const at::Tensor& v = THPVariable_Unpack(args[2]);
  if (!shapes_ok(q, k, v) || !as_scale(args[4], q.size(3), &a.scale)) NOT_SERVED();
  if (a.lens.defined() && !lens_ok(a.lens, q)) NOT_SERVED();
  const int64_t B = q.size(0), H = q.size(1), L = q.size(2), Dv = v.size(3);
  if (out.defined() && (out.dim() != 4 || out.size(0) != B || out.size(1) != H || out.size(2) != L || out.size(3) != Dv ||
                        out.scalar_type() != q.scalar_type() || out.device() != q.device()))
    NOT_SERVED();
  if (lse.defined() && (lse.dim() != 3 || lse.size(0) != B || lse.size(1) != H || lse.size(2) != L ||
                        lse.scalar_type() != at::kFloat || lse.device() != q.device()))
    NOT_SERVED();
  const c10::cuda::CUDAGuard guard(q.device());
  if (!out.defined()) out = alloc_like_query(q, {B, H, L, Dv});
  if (!lse.defined() && need_lse) lse = at::empty({B, H, L}, q.options().dtype(at::kFloat));
  if (!forward(q, k, v, a, out, lse)) return nullptr;
  PyObject* po = THPVariable_Wrap(out);
  PyObject* pl = lse.defined() ? THPVariable_Wrap(lse) : Py_NewRef(Py_None);
  return Py_BuildValue("(NN)", po, pl);
  END_HANDLE_TH_ERRORS
}

// decode(query, k_cache, v_cache, block_table, kv_lens, scale, layout, out, lse, need_lse, kv_chunk, k_new, v_new,
//        rope_cos, rope_sin, rope_interleaved) -> (out, lse or None, new_lens or None), or None
// layout: 0 a dense (B, Hkv, S, D) cache, 1 pages (pages, rows, Hkv, D), 2 pages (pages, Hkv, rows, D)
PyObject* py_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  at::Tensor table, out, lse, k_new, v_new, cos, sin;
  int64_t layout = 0, kv_chunk = 0;
  bool need_lse = false, interleaved = false;
  if (n != 16 || !plain(args[0]) || !plain(args[1]) || !plain(args[2]) || !optional_plain(args[3], &table) ||
      !plain(args[4]) || !as_int(args[6], &layout) || !optional_plain(args[7], &out) || !optional_plain(args[8], &lse) ||
      !as_bool(args[9], &need_lse) || !as_int(args[10], &kv_chunk) || !optional_plain(args[11], &k_new) ||
      !optional_plain(args[12], &v_new) || !optional_plain(args[13], &cos) || !optional_plain(args[14], &sin) ||
      !as_bool(args[15], &interleaved) || !no_modes() || layout < 0 || layout > 2)
    NOT_SERVED();
  const at::Tensor& q = THPVariable_Unpack(args[0]);
  const at::Tensor& k = THPVariable_Unpack(args[1]);
  const at::Tensor& v = THPVariable_Unpack(args[2]);
  const at::Tensor& lens = THPVariable_Unpack(args[4]);
  const auto dt = q.scalar_type();
  if (q.dim() != 4 || q.size(2) != 1 || k.dim() != 4 || v.dim() != 4 || (dt != at::kHalf && dt != at::kBFloat16) ||
      k.scalar_type() != dt || v.scalar_type() != dt || k.device() != q.device() || v.device() != q.device() ||
      k.sizes() != v.sizes() || q.numel() == 0)
    NOT_SERVED();
  const bool paged = layout != 0;
  const int hd = layout == 1 ? 2 : 1, rd = layout == 1 ? 1 : 2;
  const int64_t B = q.size(0), Hq = q.size(1), E = q.size(3), Hkv = k.size(hd);
  if (Hkv == 0 || Hq % Hkv != 0 || k.size(3) != E || !lens_ok(lens, q)) NOT_SERVED();
  if (paged != table.defined() || (!paged && k.size(0) != B)) NOT_SERVED();
  if (paged && (table.scalar_type() != at::kInt || table.dim() != 2 || table.size(0) != B || table.device() != q.device() ||
                !table.is_contiguous()))
    NOT_SERVED();
  float scale = 0.f;
  if (!as_scale(args[5], E, &scale)) NOT_SERVED();
  const int64_t S = paged ? table.size(1) * k.size(rd) : k.size(2);
  if (k_new.defined() != v_new.defined() || cos.defined() != sin.defined() || (cos.defined() && !k_new.defined())) NOT_SERVED();
  for (const at::Tensor* t : {&k_new, &v_new}) {
    if (t->defined() && (t->dim() != 3 || t->size(0) != B || t->size(1) != Hkv || t->size(2) != E || t->scalar_type() != dt ||
                         t->device() != q.device() || t->stride(2) != 1))
      NOT_SERVED();
  }
  for (const at::Tensor* t : {&cos, &sin}) {
    if (t->defined() && (t->scalar_type() != at::kFloat || t->dim() != 2 || t->size(1) < E / 2 || t->stride(1) != 1 ||
                         t->device() != q.device() || t->size(0) < 1 || t->size(0) < S))
      NOT_SERVED();
  }
  if (cos.defined() && (cos.stride(0) != sin.stride(0) || cos.size(0) != sin.size(0))) NOT_SERVED();
  if (out.defined() && (out.sizes() != q.sizes() || out.scalar_type() != dt || out.device() != q.device())) NOT_SERVED();
  if (lse.defined() && (lse.dim() != 3 || lse.size(0) != B || lse.size(1) != Hq || lse.size(2) != 1 ||
                        lse.scalar_type() != at::kFloat || lse.device() != q.device()))
    NOT_SERVED();

  const c10::cuda::CUDAGuard guard(q.device());
  const int dev = q.device().index();
  if (!out.defined()) out = at::empty_like(q);
  if (!lse.defined() && need_lse) lse = at::empty({B, Hq, 1}, q.options().dtype(at::kFloat));
  at::Tensor new_lens;
  B200SdpaParams p{};
  fill_common(p, q, out, lse, dev);
  p.force_path = B200_SDPA_PATH_DECODE;
  p.k = k.data_ptr();
  p.v = v.data_ptr();
  const int order[4] = {0, hd, rd, 3};
  for (int i = 0; i < 4; ++i) {
    p.k_stride[i] = k.stride(order[i]);
    p.v_stride[i] = v.stride(order[i]);
  }
  p.Hkv = static_cast<int32_t>(Hkv);
  p.S = static_cast<int32_t>(S);
  p.Dv = static_cast<int32_t>(E);
  p.scale = scale;
  p.kv_lens = lens.data_ptr<int32_t>();
  p.kv_chunk = static_cast<int32_t>(kv_chunk);
  if (paged) {
    p.block_table = table.data_ptr<int32_t>();
    p.block_table_stride = static_cast<int32_t>(table.size(1));
    p.page_size = static_cast<int32_t>(k.size(rd));
  }
  if (k_new.defined()) {
    p.k_new = k_new.data_ptr();
    p.v_new = v_new.data_ptr();
    for (int i = 0; i < 2; ++i) {
      p.k_new_stride[i] = k_new.stride(i);
      p.v_new_stride[i] = v_new.stride(i);
    }
    if (cos.defined()) {
      p.rope_cos = cos.data_ptr<float>();
      p.rope_sin = sin.data_ptr<float>();
      p.rope_positions = static_cast<int32_t>(cos.size(0));
      p.rope_stride = static_cast<int32_t>(cos.stride(0));
      p.rope_interleaved = interleaved ? 1 : 0;
    }
    new_lens = at::empty_like(lens);
    p.kv_lens_out = new_lens.data_ptr<int32_t>();
  }
  B200SdpaPlan plan{};
  launch(p, dev, true, plan);
  PyObject* po = THPVariable_Wrap(out);
  PyObject* pl = lse.defined() ? THPVariable_Wrap(lse) : Py_NewRef(Py_None);
  PyObject* pn = new_lens.defined() ? THPVariable_Wrap(new_lens) : Py_NewRef(Py_None);
  return Py_BuildValue("(NNN)", po, pl, pn);
  END_HANDLE_TH_ERRORS
}

// set_plan_record(dict): where every forward made here leaves its plan
PyObject* py_set_plan_record(PyObject*, PyObject* record) {
  if (!PyDict_CheckExact(record)) {
    PyErr_SetString(PyExc_TypeError, "set_plan_record: a dict");
    return nullptr;
  }
  PyObject* old = g_plan_record;
  g_plan_record = Py_NewRef(record);
  Py_XDECREF(old);
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_attention)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_forward)), METH_FASTCALL, nullptr},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_decode)), METH_FASTCALL, nullptr},
    {"set_plan_record", py_set_plan_record, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
