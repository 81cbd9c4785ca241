// The per-call host work of the operators that decoding and short prompts call most, in native code: what ops.py and ops_seq.py do around one entry of
// the C ABI - looking at the tensors, allocating the result, finding the workspace and the stream - and the call itself, without ctypes.
//
// Every function here serves the ordinary call only.  Whatever is not ordinary (another type, device or layout, an entry that returns an error, an
// allocation that fails) makes it return None before anything is enqueued, or with an error that the entry repeats, and the Python operator goes on as it would
// without this file: it raises, or takes the general path.  So the operators' checks and errors live in one place.
//
// Measured on a B200 host, us a call: int4 and fp16 linears 10.1 -> 6.1 (the launch 3, nn.Module 2), bfloat16 products 9.7 -> 4.0, decode attention (two
// launches) 13.4 -> 6.2, prompt attention 11.1 -> 4.2.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <unordered_map>
#include <vector>

// which Python and torch this file is built for (build.py looks for it in the built file)
extern "C" __attribute__((used, visibility("default"))) const char b200_host_tag[] = B200_HOST_TAG;

namespace {

struct Entries {   // the C ABI (include/b200_tgis.h, include/b200_seq.h)
  int64_t (*gemm_workspace_bytes_max)(int64_t, int64_t);
  int (*gemm_w4a16_ex)(const void*, const void*, const void*, void*, int64_t, int64_t, int64_t, int, int, int, void*, void*);
  int (*gemm_f16)(const void*, const void*, const void*, void*, int64_t, int64_t, int64_t, void*, void*);
  int (*gemm_bf16)(const void*, const void*, const void*, void*, int, int64_t, int64_t, int64_t, void*, void*);
  int64_t (*attn_decode_workspace_bytes)(int, int, int, int);
  int (*attn_decode_paged)(const void*, int64_t, const void*, const void*, const int32_t*, int64_t, const int32_t*, void*, int64_t, void*, int64_t, int, int, int,
                           int, int, float, void*);
  int (*attn_prefill_paged)(const void*, int64_t, int64_t, const void*, const void*, int64_t, const int32_t*, int64_t, const int32_t*, const int32_t*, void*, int64_t,
                            int, int, int, int, int, float, void*);
};

// One of the two libraries (they may be loaded side by side, each with workspaces of its own): its entries, and the workspaces that Python handed out for it
struct Library {
  Entries f = {};
  PyObject* gemm_workspace = nullptr;   // (tensor, N, K) -> workspace for products on its device
  PyObject* attn_workspace = nullptr;   // (tensor, bytes) -> workspace for decode attention on its device
  std::unordered_map<uint64_t, int64_t> gemm_bytes;   // by N and K
  std::vector<at::Tensor> gemm_ws, attn_ws;           // by device
};
Library &g_tgis = *new Library, &g_seq = *new Library;   // never destroyed: at exit their tensors would be freed behind the CUDA driver

bool tensor(PyObject* o, const at::Tensor*& t) {
  if (!THPVariable_Check(o)) return false;
  t = &THPVariable_Unpack(o);
  return t->is_cuda();
}
bool maybe_tensor(PyObject* o, const at::Tensor*& t) {   // or None
  t = nullptr;
  return o == Py_None || tensor(o, t);
}
void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
bool integer(PyObject* o, int64_t& v) {
  if (!PyLong_Check(o)) return false;
  v = PyLong_AsLongLong(o);
  return v != -1 || !PyErr_Occurred();
}
bool real(PyObject* o, double& v) {
  v = PyFloat_AsDouble(o);
  return v != -1.0 || !PyErr_Occurred();
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// The device's workspace of at least `need` bytes, from Python when there is none yet or it is too small; undefined where there is none to be had.  The caller
// holds it until its entry has returned: other threads run meanwhile, and one that needs more replaces it here and in Python.  What is made while
// the stream is captured belongs to the graph and is not kept.
at::Tensor workspace(std::vector<at::Tensor>& have, PyObject* make, PyObject* like, const at::Tensor& t, int64_t need, PyObject* a, PyObject* b) {
  const size_t dev = (size_t)t.get_device();
  if (have.size() <= dev) have.resize(dev + 1);
  if (!have[dev].defined() || have[dev].numel() < need) {
    PyObject* got = b ? PyObject_CallFunctionObjArgs(make, like, a, b, nullptr) : PyObject_CallFunctionObjArgs(make, like, a, nullptr);
    const at::Tensor* w = nullptr;
    if (!got || !tensor(got, w) || w->numel() < need) {
      Py_XDECREF(got);
      return {};
    }
    at::Tensor made = *w;
    Py_DECREF(got);
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return made;
    have[dev] = made;
  }
  return have[dev];
}
at::Tensor gemm_workspace(Library& lib, PyObject* like, const at::Tensor& t, int64_t N, int64_t K) {
  const uint64_t key = (uint64_t)N << 32 ^ (uint64_t)K;
  if (N >> 31 || K >> 31) return {};
  auto it = lib.gemm_bytes.find(key);
  if (it == lib.gemm_bytes.end()) {
    if (lib.gemm_bytes.size() >= 4096) lib.gemm_bytes.clear();
    it = lib.gemm_bytes.emplace(key, lib.f.gemm_workspace_bytes_max(N, K)).first;
  }
  PyObject *n = PyLong_FromLongLong(N), *k = PyLong_FromLongLong(K);
  const int64_t need = it->second;
  at::Tensor w;
  if (n && k) w = workspace(lib.gemm_ws, lib.gemm_workspace, like, t, need, n, k);
  Py_XDECREF(n);
  Py_XDECREF(k);
  return w;
}

// runs `call`; None where it cannot serve the call, also after an exception of C++ or Python
template <typename F>
PyObject* serve(F&& call) {
  PyObject* r = nullptr;
  try {
    r = call();
  } catch (...) {
    r = nullptr;
  }
  if (!r) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  return r;
}
// the entry itself, other Python threads running meanwhile
template <typename F>
bool enqueue(F&& entry) {
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = entry();
  Py_END_ALLOW_THREADS
  return status == 0;
}
PyObject* give(PyObject* out, const at::Tensor* given, const at::Tensor& made) {
  if (!given) return THPVariable_Wrap(made);
  Py_INCREF(out);
  return out;
}

// x, packed, N, groupsize, bias, out, workspace, layout, silu_mul
PyObject* gemm_w4a16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return serve([&]() -> PyObject* {
    const at::Tensor *x, *packed, *bias, *out, *ws;
    int64_t N, group, layout, silu;
    if (n != 9 || !tensor(a[0], x) || !tensor(a[1], packed) || !integer(a[2], N) || !integer(a[3], group) || !maybe_tensor(a[4], bias) || !maybe_tensor(a[5], out) ||
        !maybe_tensor(a[6], ws) || !integer(a[7], layout) || !integer(a[8], silu))
      return nullptr;
    if (x->scalar_type() != at::kHalf || packed->scalar_type() != at::kByte || x->dim() != 2 || !x->is_contiguous() || !packed->is_contiguous() || N <= 0) return nullptr;
    const int64_t T = x->size(0), K = x->size(1);
    at::Tensor made, held;
    if (!ws) {
      held = gemm_workspace(g_tgis, a[0], *x, N, K);
      if (!held.defined()) return nullptr;
      ws = &held;
    }
    if (!out) made = at::empty({T, silu ? N / 2 : N}, x->options());
    const at::Tensor& y = out ? *out : made;
    void *px = x->data_ptr(), *pp = packed->data_ptr(), *pb = ptr(bias), *py = y.data_ptr(), *pw = ws->data_ptr(), *st = stream();
    if (!enqueue([&] { return g_tgis.f.gemm_w4a16_ex(px, pp, pb, py, T, N, K, (int)group, (int)layout, silu != 0, pw, st); })) return nullptr;
    return give(a[5], out, made);
  });
}

// x, w, bias, out, workspace
PyObject* gemm_f16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return serve([&]() -> PyObject* {
    const at::Tensor *x, *w, *bias, *out, *ws;
    if (n != 5 || !tensor(a[0], x) || !tensor(a[1], w) || !maybe_tensor(a[2], bias) || !maybe_tensor(a[3], out) || !maybe_tensor(a[4], ws)) return nullptr;
    if (x->scalar_type() != at::kHalf || w->scalar_type() != at::kHalf || x->dim() != 2 || w->dim() != 2 || !x->is_contiguous() || !w->is_contiguous()) return nullptr;
    const int64_t T = x->size(0), K = x->size(1), N = w->size(0);
    at::Tensor made, held;
    if (!ws) {
      held = gemm_workspace(g_tgis, a[0], *x, N, K);
      if (!held.defined()) return nullptr;
      ws = &held;
    }
    if (!out) made = at::empty({T, N}, x->options());
    const at::Tensor& y = out ? *out : made;
    void *px = x->data_ptr(), *pm = w->data_ptr(), *pb = ptr(bias), *py = y.data_ptr(), *pw = ws->data_ptr(), *st = stream();
    if (!enqueue([&] { return g_tgis.f.gemm_f16(px, pm, pb, py, T, N, K, pw, st); })) return nullptr;
    return give(a[3], out, made);
  });
}

// x, w, bias, out in fp32: bfloat16 operands, new result in bfloat16 or fp32, no activation
PyObject* linear_bf16(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return serve([&]() -> PyObject* {
    const at::Tensor *x, *w, *bias;
    int64_t f32;
    if (n != 4 || !tensor(a[0], x) || !tensor(a[1], w) || !maybe_tensor(a[2], bias) || !integer(a[3], f32)) return nullptr;
    if (x->scalar_type() != at::kBFloat16 || w->scalar_type() != at::kBFloat16 || (bias && bias->scalar_type() != at::kBFloat16) || x->dim() != 2 || w->dim() != 2 ||
        !x->is_contiguous() || !w->is_contiguous())
      return nullptr;
    const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
    if (w->size(1) != K || K % 8 != 0 || K < 64 || M == 0 || N == 0 || ((uintptr_t)x->data_ptr() | (uintptr_t)w->data_ptr()) % 16 != 0) return nullptr;
    const at::Tensor ws = gemm_workspace(g_seq, a[0], *x, N, K);
    if (!ws.defined()) return nullptr;
    at::Tensor y = at::empty({M, N}, x->options().dtype(f32 ? at::kFloat : at::kBFloat16));
    void *px = x->data_ptr(), *pm = w->data_ptr(), *pb = ptr(bias), *py = y.data_ptr(), *pw = ws.data_ptr(), *st = stream();
    if (!enqueue([&] { return g_seq.f.gemm_bf16(px, pm, pb, py, f32 != 0, M, N, K, pw, st); })) return nullptr;
    return THPVariable_Wrap(y);
  });
}

// a [rows, heads, dim] fp16 tensor whose last two dimensions are dense
bool heads_rows(const at::Tensor& q) { return q.scalar_type() == at::kHalf && q.dim() == 3 && q.stride(2) == 1 && q.stride(1) == q.size(2); }

// q, k_pool, v_pool, block_table, context_lens, max_context_len, scale, n_kv_heads, out, workspace
PyObject* attn_decode_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return serve([&]() -> PyObject* {
    const at::Tensor *q, *k, *v, *table, *lens, *out, *ws;
    int64_t most, kv;
    double scale;
    if (n != 10 || !tensor(a[0], q) || !tensor(a[1], k) || !tensor(a[2], v) || !tensor(a[3], table) || !tensor(a[4], lens) || !integer(a[5], most) || !real(a[6], scale) ||
        !integer(a[7], kv) || !maybe_tensor(a[8], out) || !maybe_tensor(a[9], ws))
      return nullptr;
    if (!heads_rows(*q) || table->scalar_type() != at::kInt || lens->scalar_type() != at::kInt || table->dim() < 1 || (out && out->dim() < 1)) return nullptr;
    const int64_t B = q->size(0), h = q->size(1), d = q->size(2);
    const int64_t need = g_tgis.f.attn_decode_workspace_bytes((int)B, (int)h, (int)d, (int)most);
    at::Tensor made, held;
    if (ws) {
      if ((int64_t)(ws->numel() * ws->element_size()) < need) return nullptr;
    } else {
      PyObject* bytes = PyLong_FromLongLong(need);
      if (bytes) held = workspace(g_tgis.attn_ws, g_tgis.attn_workspace, a[0], *q, need, bytes, nullptr);
      Py_XDECREF(bytes);
      if (!held.defined()) return nullptr;
      ws = &held;
    }
    if (!out) made = at::empty({B, h, d}, q->options());
    const at::Tensor& y = out ? *out : made;
    void *pq = q->data_ptr(), *pk = k->data_ptr(), *pv = v->data_ptr(), *py = y.data_ptr(), *pw = ws->data_ptr(), *st = stream();
    const int32_t *pt = (const int32_t*)table->data_ptr(), *pl = (const int32_t*)lens->data_ptr();
    const int64_t qs = q->stride(0), ts = table->stride(0), ys = y.stride(0), wb = ws->numel() * ws->element_size();
    if (!enqueue([&] { return g_tgis.f.attn_decode_paged(pq, qs, pk, pv, pt, ts, pl, py, ys, pw, wb, (int)B, (int)h, (int)kv, (int)d, (int)most, (float)scale, st); }))
      return nullptr;
    return give(a[8], out, made);
  });
}

// q, k_pool, v_pool, block_table, context_lens, cu_seqlens_q, max_q, scale, out
PyObject* attn_prefill_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return serve([&]() -> PyObject* {
    const at::Tensor *q, *k, *v, *table, *lens, *cu, *out;
    int64_t most;
    double scale;
    if (n != 9 || !tensor(a[0], q) || !tensor(a[1], k) || !tensor(a[2], v) || !tensor(a[3], table) || !tensor(a[4], lens) || !tensor(a[5], cu) || !integer(a[6], most) ||
        !real(a[7], scale) || !maybe_tensor(a[8], out))
      return nullptr;
    if (!heads_rows(*q) || table->scalar_type() != at::kInt || lens->scalar_type() != at::kInt || cu->scalar_type() != at::kInt || !k->is_contiguous() || !v->is_contiguous() ||
        k->dim() < 2 || table->dim() < 1 || cu->dim() < 1 || (out && out->dim() < 1))
      return nullptr;
    const int64_t T = q->size(0), h = q->size(1), d = q->size(2), B = cu->size(0) - 1, blocks = k->size(0), kv = k->size(1);
    at::Tensor made;
    if (!out) made = at::empty({T, h, d}, q->options());
    const at::Tensor& y = out ? *out : made;
    void *pq = q->data_ptr(), *pk = k->data_ptr(), *pv = v->data_ptr(), *py = y.data_ptr(), *st = stream();
    const int32_t *pt = (const int32_t*)table->data_ptr(), *pl = (const int32_t*)lens->data_ptr(), *pc = (const int32_t*)cu->data_ptr();
    const int64_t qs = q->stride(0), ts = table->stride(0), ys = y.stride(0);
    if (!enqueue([&] {
          return g_tgis.f.attn_prefill_paged(pq, qs, T, pk, pv, blocks, pt, ts, pl, pc, py, ys, (int)B, (int)most, (int)h, (int)kv, (int)d, (float)scale, st);
        }))
      return nullptr;
    return give(a[8], out, made);
  });
}

// (which: 0 the flash families' library, 1 the hybrid families'; {entry: address}; workspace callables)
PyObject* bind(PyObject*, PyObject* args) {
  int which;
  PyObject *entries, *gemm, *attn;
  if (!PyArg_ParseTuple(args, "iO!OO", &which, &PyDict_Type, &entries, &gemm, &attn)) return nullptr;
  Library& lib = which ? g_seq : g_tgis;
  auto set = [&](const char* name, auto& f) {
    PyObject* o = PyDict_GetItemString(entries, name);
    if (o) f = reinterpret_cast<std::decay_t<decltype(f)>>(PyLong_AsVoidPtr(o));
  };
  set("b200_gemm_workspace_bytes_max", lib.f.gemm_workspace_bytes_max);
  set("b200_gemm_w4a16_ex", lib.f.gemm_w4a16_ex);
  set("b200_gemm_f16", lib.f.gemm_f16);
  set("b200_gemm_bf16", lib.f.gemm_bf16);
  set("b200_attn_decode_workspace_bytes", lib.f.attn_decode_workspace_bytes);
  set("b200_attn_decode_paged", lib.f.attn_decode_paged);
  set("b200_attn_prefill_paged", lib.f.attn_prefill_paged);
  Py_XDECREF(lib.gemm_workspace);
  Py_XDECREF(lib.attn_workspace);
  Py_INCREF(gemm);
  Py_INCREF(attn);
  lib.gemm_workspace = gemm;
  lib.attn_workspace = attn;
  lib.gemm_bytes.clear();
  lib.gemm_ws.clear();   // what earlier callables handed out is theirs
  lib.attn_ws.clear();
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr},
                         {"gemm_w4a16", (PyCFunction)(void*)gemm_w4a16, METH_FASTCALL, nullptr},
                         {"gemm_f16", (PyCFunction)(void*)gemm_f16, METH_FASTCALL, nullptr},
                         {"linear_bf16", (PyCFunction)(void*)linear_bf16, METH_FASTCALL, nullptr},
                         {"attn_decode_paged", (PyCFunction)(void*)attn_decode_paged, METH_FASTCALL, nullptr},
                         {"attn_prefill_paged", (PyCFunction)(void*)attn_prefill_paged, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200_host() { return PyModule_Create(&module); }
