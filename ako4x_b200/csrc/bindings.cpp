// Python bindings of the operators' `run(...)`: argument checks, output and workspace allocation
// and the C-ABI call (include/ako4x_b200.h) in one native call per operator.
//
// Why it is native: the small calls of this library run 2 to 20 us on the GPU, and the same host
// path written in Python over ctypes cost 12 us (RMSNorm) to 60 us (indexer + sparse attention) of
// host time per call, so a stream of such calls was bound by the host. Here a call costs the
// parsing of its tensors, one caching-allocator request per output and workspace, and the kernel
// launches. Nothing is kept between calls: outputs and workspaces come from PyTorch's caching
// allocator on the current stream, as they did before. Measured per call in a stream of calls: RMSNorm
// of 64 rows 12.1 -> 3.8 us, GDN decode of 16 sequences 21.6 -> 5.5 us, GQA decode of one sequence
// 26.0 -> 12.6 us (now bound by its two kernels).
//
// Every function is METH_FASTCALL and takes the positional arguments of the Python wrapper of the
// same operator (ako4x_b200/<op>.py). The GIL is released around the launches, which may block when
// the stream's queue is full.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <string>

#include "ako4x_b200.h"

namespace {

using at::IntArrayRef;
using at::ScalarType;
using at::Tensor;

PyObject* g_error = nullptr;  // ako4x_b200._cabi.Ako4xError

[[noreturn]] void fail(const std::string& msg) {
  PyErr_SetString(g_error, msg.c_str());
  throw python_error();
}
void need(bool ok, const char* msg) {
  if (!ok) fail(msg);
}
void check_status(int st, const char* what) {
  if (st == AKO4X_OK) return;
  const char* name = st == AKO4X_EINVAL              ? "AKO4X_EINVAL"
                     : st == AKO4X_EUNSUPPORTED_SHAPE ? "AKO4X_EUNSUPPORTED_SHAPE"
                     : st == AKO4X_ELAUNCH            ? "AKO4X_ELAUNCH"
                     : st == AKO4X_EWORKSPACE         ? "AKO4X_EWORKSPACE"
                     : st == AKO4X_ETOOLARGE          ? "AKO4X_ETOOLARGE"
                                                      : "unknown status";
  fail(std::string(what) + " failed: " + name);
}

const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "tensor expected, got %s", Py_TYPE(o)->tp_name);
    throw python_error();
  }
  return THPVariable_Unpack(o);
}
double number(PyObject* o) {  // a Python number, or a one-element tensor (which is then read)
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
int64_t integer(PyObject* o) {
  if (PyLong_CheckExact(o)) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  PyObject* as_int = PyNumber_Long(o);
  if (!as_int) throw python_error();
  const long long v = PyLong_AsLongLong(as_int);
  Py_DECREF(as_int);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
void count(Py_ssize_t n, Py_ssize_t expected, const char* op) {
  if (n != expected) {
    PyErr_Format(PyExc_TypeError, "%s: %zd arguments expected, got %zd", op, expected, n);
    throw python_error();
  }
}

bool shape_is(const Tensor& t, std::initializer_list<int64_t> s) {
  const IntArrayRef sz = t.sizes();
  if (sz.size() != s.size()) return false;
  size_t i = 0;
  for (int64_t v : s)
    if (sz[i++] != v) return false;
  return true;
}

// Device address of a contiguous CUDA tensor.
void* ptr(const Tensor& t) {
  need(t.is_cuda(), "ako4x_b200 operators take CUDA tensors only (there is no CPU path)");
  need(t.is_contiguous(), "tensor must be contiguous");
  return t.data_ptr();
}
// A contiguous copy where the tensor is not contiguous already; the caller keeps it alive until
// the launches are enqueued.
Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
Tensor dense(const Tensor& t, ScalarType dt) { return t.scalar_type() == dt ? dense(t) : t.to(dt).contiguous(); }

Tensor empty(IntArrayRef sizes, ScalarType dt, const Tensor& like) {
  need(like.is_cuda(), "ako4x_b200 operators take CUDA tensors only (there is no CPU path)");
  return at::detail::empty_cuda(sizes, dt, like.device(), std::nullopt);
}
struct Workspace {
  Tensor t;
  void* p = nullptr;
  size_t bytes = 0;
  Workspace(size_t n, const Tensor& like) : bytes(n) {
    if (n > 0) {
      t = empty({(int64_t)n}, at::kByte, like);
      p = t.data_ptr();
    }
  }
};

void* current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

struct NoGil {
  PyThreadState* s;
  NoGil() : s(PyEval_SaveThread()) {}
  ~NoGil() { PyEval_RestoreThread(s); }
};
template <class F>
int without_gil(F&& f) {
  NoGil g;
  return f();
}

PyObject* pack(Tensor a) { return THPVariable_Wrap(std::move(a)); }
template <class... T>
PyObject* pack_tuple(T... ts) {
  PyObject* out = PyTuple_New(sizeof...(T));
  if (!out) throw python_error();
  Py_ssize_t i = 0;
  bool ok = true;
  auto put = [&](Tensor t) {
    PyObject* o = THPVariable_Wrap(std::move(t));
    if (!o) ok = false;
    PyTuple_SET_ITEM(out, i++, o);
  };
  (put(std::move(ts)), ...);
  if (!ok) {
    Py_DECREF(out);
    throw python_error();
  }
  return out;
}

// ---- RMSNorm -----------------------------------------------------------------------------------

PyObject* rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 2, "rmsnorm");
  c10::NoGradGuard ng;
  const Tensor &h = tensor(a[0]), &w = tensor(a[1]);
  need(h.dim() == 2 && h.size(1) == 128, "rmsnorm: hidden_states must be [rows, 128]");
  need(h.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16, "rmsnorm: bf16 tensors expected");
  need(w.numel() == 128, "rmsnorm: weight must have 128 elements");
  const Tensor x = dense(h), wc = dense(w);
  const int64_t rows = x.size(0);
  Tensor out = empty(x.sizes(), at::kBFloat16, x);
  void *xp = ptr(x), *wp = ptr(wc), *op = ptr(out), *st = current_stream();
  check_status(without_gil([&] { return ako4x_rmsnorm_h128(xp, wp, op, rows, st); }), "ako4x_rmsnorm_h128");
  return pack(std::move(out));
  END_HANDLE_TH_ERRORS
}

// ---- attention ---------------------------------------------------------------------------------

PyObject* gqa_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 6, "gqa_decode");
  c10::NoGradGuard ng;
  const Tensor &q0 = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]), &indptr = tensor(a[3]), &indices = tensor(a[4]);
  const float scale = (float)number(a[5]);
  need(q0.dim() == 3 && q0.size(1) == 32 && q0.size(2) == 128, "gqa_decode: q must be [batch, 32, 128]");
  need(k.dim() == 4 && k.size(2) == 8 && k.size(3) == 128 && v.sizes() == k.sizes(),
       "gqa_decode: caches must be [pages, page_size, 8, 128]");
  need(q0.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16,
       "gqa_decode: bf16 tensors expected");
  need(indptr.scalar_type() == at::kInt && indices.scalar_type() == at::kInt,
       "gqa_decode: kv_indptr / kv_indices must be int32");
  const int64_t batch = q0.size(0), page_size = k.size(1), n_idx = indices.numel();
  need(indptr.numel() == batch + 1, "gqa_decode: kv_indptr must have batch + 1 entries");
  const Tensor q = dense(q0);
  Tensor o = empty(q.sizes(), at::kBFloat16, q), lse = empty({batch, 32}, at::kFloat, q);
  Workspace ws(ako4x_gqa_paged_decode_workspace_bytes(batch, n_idx, page_size), q);
  void *qp = ptr(q), *kp = ptr(k), *vp = ptr(v), *ip = ptr(indptr), *xp = ptr(indices), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_gqa_paged_decode(qp, kp, vp, (const int32_t*)ip, (const int32_t*)xp, scale, o.data_ptr(),
                                               (float*)lse.data_ptr(), batch, n_idx, page_size, ws.p, ws.bytes, st);
               }),
               "ako4x_gqa_paged_decode");
  return pack_tuple(std::move(o), std::move(lse));
  END_HANDLE_TH_ERRORS
}

void check_mla(const std::string& op, const Tensor& qn, const Tensor& qp, const Tensor& ckv, const Tensor& kpe) {
  if (!(qn.dim() == 3 && qn.size(1) == 16 && qn.size(2) == 512 && shape_is(qp, {qn.size(0), 16, 64})))
    fail(op + ": q_nope must be [n,16,512] and q_pe [n,16,64]");
  if (!(ckv.dim() == 3 && ckv.size(2) == 512 && shape_is(kpe, {ckv.size(0), ckv.size(1), 64})))
    fail(op + ": caches must be [pages,page_size,512] and [pages,page_size,64]");
  if (qn.scalar_type() != at::kBFloat16 || qp.scalar_type() != at::kBFloat16 || ckv.scalar_type() != at::kBFloat16 ||
      kpe.scalar_type() != at::kBFloat16)
    fail(op + ": bf16 tensors expected");
}

PyObject* mla_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 7, "mla_decode");
  c10::NoGradGuard ng;
  const Tensor &qn0 = tensor(a[0]), &qp0 = tensor(a[1]), &ckv = tensor(a[2]), &kpe = tensor(a[3]), &indptr = tensor(a[4]),
               &indices = tensor(a[5]);
  const float scale = (float)number(a[6]);
  check_mla("mla_decode", qn0, qp0, ckv, kpe);
  need(indptr.scalar_type() == at::kInt && indices.scalar_type() == at::kInt,
       "mla_decode: kv_indptr / kv_indices must be int32");
  const int64_t batch = qn0.size(0), page_size = ckv.size(1), n_idx = indices.numel();
  need(indptr.numel() == batch + 1, "mla_decode: kv_indptr must have batch + 1 entries");
  const Tensor qn = dense(qn0), qp = dense(qp0);
  Tensor o = empty(qn.sizes(), at::kBFloat16, qn), lse = empty({batch, 16}, at::kFloat, qn);
  Workspace ws(ako4x_mla_paged_decode_workspace_bytes(batch, n_idx, page_size), qn);
  void *p0 = ptr(qn), *p1 = ptr(qp), *p2 = ptr(ckv), *p3 = ptr(kpe), *p4 = ptr(indptr), *p5 = ptr(indices), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_mla_paged_decode(p0, p1, p2, p3, (const int32_t*)p4, (const int32_t*)p5, scale, o.data_ptr(),
                                               (float*)lse.data_ptr(), batch, n_idx, page_size, ws.p, ws.bytes, st);
               }),
               "ako4x_mla_paged_decode");
  return pack_tuple(std::move(o), std::move(lse));
  END_HANDLE_TH_ERRORS
}

PyObject* mla_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 8, "mla_prefill");
  c10::NoGradGuard ng;
  const Tensor &qn0 = tensor(a[0]), &qp0 = tensor(a[1]), &ckv = tensor(a[2]), &kpe = tensor(a[3]), &qoi = tensor(a[4]),
               &kvi = tensor(a[5]), &indices = tensor(a[6]);
  const float scale = (float)number(a[7]);
  check_mla("mla_prefill", qn0, qp0, ckv, kpe);
  need(qoi.scalar_type() == at::kInt && kvi.scalar_type() == at::kInt && indices.scalar_type() == at::kInt,
       "mla_prefill: indptr / indices must be int32");
  need(qoi.numel() == kvi.numel(), "mla_prefill: qo_indptr and kv_indptr must have the same length");
  const int64_t total_q = qn0.size(0), batch = qoi.numel() - 1, page_size = ckv.size(1), n_idx = indices.numel();
  const Tensor qn = dense(qn0), qp = dense(qp0);
  Tensor o = empty(qn.sizes(), at::kBFloat16, qn), lse = empty({total_q, 16}, at::kFloat, qn);
  Workspace ws(ako4x_mla_paged_prefill_workspace_bytes(total_q, batch, n_idx, page_size), qn);
  void *p0 = ptr(qn), *p1 = ptr(qp), *p2 = ptr(ckv), *p3 = ptr(kpe), *p4 = ptr(qoi), *p5 = ptr(kvi), *p6 = ptr(indices),
       *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_mla_paged_prefill(p0, p1, p2, p3, (const int32_t*)p4, (const int32_t*)p5, (const int32_t*)p6,
                                                scale, o.data_ptr(), (float*)lse.data_ptr(), total_q, batch, n_idx, page_size,
                                                ws.p, ws.bytes, st);
               }),
               "ako4x_mla_paged_prefill");
  return pack_tuple(std::move(o), std::move(lse));
  END_HANDLE_TH_ERRORS
}

PyObject* dsa_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 6, "dsa_attention");
  c10::NoGradGuard ng;
  const Tensor &qn0 = tensor(a[0]), &qp0 = tensor(a[1]), &ckv = tensor(a[2]), &kpe = tensor(a[3]), &si = tensor(a[4]);
  const float scale = (float)number(a[5]);
  check_mla("dsa_attention", qn0, qp0, ckv, kpe);
  const int64_t tokens = qn0.size(0);
  need(si.scalar_type() == at::kInt && si.dim() == 2 && si.size(0) == tokens,
       "dsa_attention: sparse_indices must be int32 [tokens, topk]");
  const int64_t topk = si.size(1), rows = ckv.size(0) * ckv.size(1);
  const Tensor qn = dense(qn0), qp = dense(qp0), idx = dense(si);
  Tensor o = empty(qn.sizes(), at::kBFloat16, qn), lse = empty({tokens, 16}, at::kFloat, qn);
  Workspace ws(ako4x_dsa_sparse_attention_workspace_bytes(tokens, topk), qn);
  void *p0 = ptr(qn), *p1 = ptr(qp), *p2 = ptr(ckv), *p3 = ptr(kpe), *p4 = ptr(idx), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_dsa_sparse_attention(p0, p1, p2, p3, (const int32_t*)p4, scale, o.data_ptr(),
                                                   (float*)lse.data_ptr(), tokens, topk, rows, ws.p, ws.bytes, st);
               }),
               "ako4x_dsa_sparse_attention");
  return pack_tuple(std::move(o), std::move(lse));
  END_HANDLE_TH_ERRORS
}

// ---- DSA indexer -------------------------------------------------------------------------------

constexpr int64_t kIndexPageBytes = 8448, kTopk = 2048;

struct IndexerArgs {
  Tensor q, cache, w, lens, table;
  int64_t rows, npages, max_pages;
  explicit IndexerArgs(PyObject* const* a) {
    const Tensor &q0 = tensor(a[0]), &c0 = tensor(a[1]), &w0 = tensor(a[2]), &l0 = tensor(a[3]), &t0 = tensor(a[4]);
    need(q0.dim() == 3 && q0.size(1) == 64 && q0.size(2) == 128 && q0.element_size() == 1,
         "dsa_indexer: q_index_fp8 must be e4m3 [rows, 64, 128]");
    rows = q0.size(0);
    need(c0.dim() >= 1 && c0.numel() * (int64_t)c0.element_size() == c0.size(0) * kIndexPageBytes,
         "dsa_indexer: cache must hold 8448 bytes per page");
    npages = c0.size(0);
    need(w0.scalar_type() == at::kFloat && shape_is(w0, {rows, 64}), "dsa_indexer: weights must be fp32 [rows, 64]");
    need(l0.scalar_type() == at::kInt && t0.scalar_type() == at::kInt && l0.numel() == rows && t0.dim() == 2 && t0.size(0) == rows,
         "dsa_indexer: seq_lens int32 [rows], block_table int32 [rows, pages]");
    max_pages = t0.size(1);
    q = dense(q0);
    cache = dense(c0);
    w = dense(w0);
    lens = dense(l0);
    table = dense(t0);
  }
};

PyObject* dsa_indexer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 5, "dsa_indexer");
  c10::NoGradGuard ng;
  const IndexerArgs x(a);
  Tensor out = empty({x.rows, kTopk}, at::kInt, x.q);
  Workspace ws(ako4x_dsa_topk_indexer_workspace_bytes(x.rows, x.max_pages), x.q);
  void *p0 = ptr(x.q), *p1 = ptr(x.cache), *p2 = ptr(x.w), *p3 = ptr(x.lens), *p4 = ptr(x.table), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_dsa_topk_indexer(p0, p1, (const float*)p2, (const int32_t*)p3, (const int32_t*)p4,
                                               (int32_t*)out.data_ptr(), x.rows, x.max_pages, x.npages, ws.p, ws.bytes, st);
               }),
               "ako4x_dsa_topk_indexer");
  return pack_tuple(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyObject* dsa_indexer_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 10, "dsa_indexer_attention");
  c10::NoGradGuard ng;
  const IndexerArgs x(a);
  const Tensor &qn0 = tensor(a[5]), &qp0 = tensor(a[6]), &ckv = tensor(a[7]), &kpe = tensor(a[8]);
  const float scale = (float)number(a[9]);
  check_mla("dsa_indexer_attention", qn0, qp0, ckv, kpe);
  need(qn0.size(0) == x.rows && ckv.size(0) == x.npages && ckv.size(1) == 64,
       "dsa_indexer_attention: one query row per indexer row, caches of [pages, 64, .]");
  const Tensor qn = dense(qn0), qp = dense(qp0);
  Tensor topk = empty({x.rows, kTopk}, at::kInt, x.q), o = empty(qn.sizes(), at::kBFloat16, x.q),
         lse = empty({x.rows, 16}, at::kFloat, x.q);
  Workspace ws(ako4x_dsa_indexer_attention_workspace_bytes(x.rows, x.max_pages), x.q);
  void *p0 = ptr(x.q), *p1 = ptr(x.cache), *p2 = ptr(x.w), *p3 = ptr(x.lens), *p4 = ptr(x.table), *p5 = ptr(qn), *p6 = ptr(qp),
       *p7 = ptr(ckv), *p8 = ptr(kpe), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_dsa_indexer_attention(p0, p1, (const float*)p2, (const int32_t*)p3, (const int32_t*)p4, p5, p6,
                                                    p7, p8, scale, (int32_t*)topk.data_ptr(), o.data_ptr(),
                                                    (float*)lse.data_ptr(), x.rows, x.max_pages, x.npages, ws.p, ws.bytes, st);
               }),
               "ako4x_dsa_indexer_attention");
  return pack_tuple(std::move(o), std::move(lse), std::move(topk));
  END_HANDLE_TH_ERRORS
}

// ---- FP8 producers and MoE ---------------------------------------------------------------------

PyObject* quantize_1x128(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 1, "quantize_1x128");
  c10::NoGradGuard ng;
  const Tensor& x0 = tensor(a[0]);
  need(x0.dim() == 2 && x0.scalar_type() == at::kBFloat16 && x0.size(1) % 128 == 0,
       "quantize_1x128: bf16 [rows, cols] with cols a multiple of 128");
  const int64_t rows = x0.size(0), cols = x0.size(1);
  const Tensor x = dense(x0);
  Tensor q = empty({rows, cols}, at::kFloat8_e4m3fn, x), scale = empty({cols / 128, rows}, at::kFloat, x);
  void *xp = ptr(x), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_fp8_quantize_1x128(xp, q.data_ptr(), (float*)scale.data_ptr(), rows, cols, st);
               }),
               "ako4x_fp8_quantize_1x128");
  return pack_tuple(std::move(q), std::move(scale));
  END_HANDLE_TH_ERRORS
}

// (k, slot_mapping, k_index_cache): in place, returns None
PyObject* index_k_cache_write(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 3, "index_k_cache_write");
  c10::NoGradGuard ng;
  const Tensor &k0 = tensor(a[0]), &s0 = tensor(a[1]), &cache = tensor(a[2]);
  need(k0.dim() == 2 && k0.size(1) == 128 && k0.scalar_type() == at::kBFloat16,
       "index_k_cache_write: k must be bf16 [tokens, 128]");
  need(s0.scalar_type() == at::kInt && s0.numel() == k0.size(0), "index_k_cache_write: slot_mapping must be int32 [tokens]");
  need(cache.dim() >= 1 && cache.numel() * (int64_t)cache.element_size() == cache.size(0) * kIndexPageBytes && cache.is_contiguous(),
       "index_k_cache_write: the cache must be contiguous with 8448 bytes per page");
  const int64_t tokens = k0.size(0), npages = cache.size(0);
  const Tensor k = dense(k0), slots = dense(s0);
  void *kp = ptr(k), *sp = ptr(slots), *cp = ptr(cache), *st = current_stream();
  check_status(without_gil([&] { return ako4x_dsa_index_k_cache_write(kp, (const int32_t*)sp, cp, tokens, npages, st); }),
               "ako4x_dsa_index_k_cache_write");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// The ten arguments of moe.run, then a flag: true returns (out, workspace) for a read of the
// device status word, false returns out.
PyObject* moe(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  constexpr int64_t H = 7168, I = 2048, E = 256;
  count(n, 11, "moe");
  c10::NoGradGuard ng;
  const Tensor &lg0 = tensor(a[0]), &rb0 = tensor(a[1]), &x0 = tensor(a[2]), &xs0 = tensor(a[3]), &w13 = tensor(a[4]),
               &s13_0 = tensor(a[5]), &w2 = tensor(a[6]), &s2_0 = tensor(a[7]);
  const int64_t offset = integer(a[8]);
  const float factor = (float)number(a[9]);
  const bool want_ws = PyObject_IsTrue(a[10]) == 1;
  need(x0.dim() >= 1 && w13.dim() >= 1, "moe: hidden_states must be e4m3 [tokens, 7168]");
  const int64_t tokens = x0.size(0), n_local = w13.size(0);
  need(shape_is(lg0, {tokens, E}) && lg0.scalar_type() == at::kFloat, "moe: routing_logits must be fp32 [tokens, 256]");
  const bool bias_bf16 = rb0.scalar_type() == at::kBFloat16;
  need(rb0.numel() == E && (bias_bf16 || rb0.scalar_type() == at::kFloat), "moe: routing_bias must be fp32 or bf16 [256]");
  need(shape_is(x0, {tokens, H}) && x0.element_size() == 1, "moe: hidden_states must be e4m3 [tokens, 7168]");
  need(shape_is(xs0, {H / 128, tokens}) && xs0.scalar_type() == at::kFloat, "moe: hidden_states_scale must be fp32 [56, tokens]");
  need(shape_is(w13, {n_local, 2 * I, H}) && w13.element_size() == 1, "moe: gemm1_weights must be e4m3 [E, 4096, 7168]");
  need(shape_is(s13_0, {n_local, 2 * I / 128, H / 128}) && s13_0.scalar_type() == at::kFloat,
       "moe: gemm1_weights_scale must be fp32 [E, 32, 56]");
  need(shape_is(w2, {n_local, H, I}) && w2.element_size() == 1, "moe: gemm2_weights must be e4m3 [E, 7168, 2048]");
  need(shape_is(s2_0, {n_local, H / 128, I / 128}) && s2_0.scalar_type() == at::kFloat,
       "moe: gemm2_weights_scale must be fp32 [E, 56, 16]");
  const Tensor lg = dense(lg0), rb = dense(rb0), x = dense(x0), xs = dense(xs0), s13 = dense(s13_0), s2 = dense(s2_0);
  Tensor out = empty({tokens, H}, at::kBFloat16, x);
  Workspace ws(ako4x_moe_fp8_block_scale_workspace_bytes(tokens, n_local), x);
  void *p0 = ptr(lg), *p1 = ptr(rb), *p2 = ptr(x), *p3 = ptr(xs), *p4 = ptr(w13), *p5 = ptr(s13), *p6 = ptr(w2), *p7 = ptr(s2),
       *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_moe_fp8_block_scale((const float*)p0, p1, bias_bf16 ? 1 : 0, p2, (const float*)p3, p4,
                                                  (const float*)p5, p6, (const float*)p7, (int32_t)offset, factor,
                                                  out.data_ptr(), tokens, n_local, ws.p, ws.bytes, st);
               }),
               "ako4x_moe_fp8_block_scale");
  if (want_ws) return pack_tuple(std::move(out), std::move(ws.t));
  return pack(std::move(out));
  END_HANDLE_TH_ERRORS
}

// ---- Gated Delta Net and GEMM ------------------------------------------------------------------

float gdn_scale(PyObject* o) {
  if (o == Py_None) return (float)(1.0 / std::sqrt(128.0));
  const double v = number(o);
  return (float)(v == 0.0 ? 1.0 / std::sqrt(128.0) : v);
}

PyObject* gdn_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 9, "gdn_decode");
  c10::NoGradGuard ng;
  const Tensor &q0 = tensor(a[0]), &k0 = tensor(a[1]), &v0 = tensor(a[2]), &A0 = tensor(a[4]), &a0 = tensor(a[5]),
               &d0 = tensor(a[6]), &b0 = tensor(a[7]);
  const bool has_state = a[3] != Py_None;
  need(q0.dim() == 4 && q0.size(1) == 1 && q0.size(2) == 4 && q0.size(3) == 128 && k0.sizes() == q0.sizes(),
       "gdn_decode: q and k must be [batch, 1, 4, 128]");
  const int64_t B = q0.size(0);
  need(shape_is(v0, {B, 1, 8, 128}), "gdn_decode: v must be [batch, 1, 8, 128]");
  for (const Tensor* t : {&q0, &k0, &v0, &a0, &b0})
    need(t->scalar_type() == at::kBFloat16, "gdn_decode: q, k, v, a, b must be bf16");
  need(A0.numel() == 8 && d0.numel() == 8 && a0.numel() == B * 8 && b0.numel() == B * 8,
       "gdn_decode: A_log, dt_bias must have 8 elements, a and b batch * 8");
  Tensor sc;
  if (has_state) {
    const Tensor& s0 = tensor(a[3]);
    need(shape_is(s0, {B, 8, 128, 128}) && s0.scalar_type() == at::kFloat, "gdn_decode: state must be fp32 [batch, 8, 128, 128]");
    sc = dense(s0);
  }
  const float scale = gdn_scale(a[8]);
  const Tensor q = dense(q0), k = dense(k0), v = dense(v0), av = dense(a0), bv = dense(b0), A = dense(A0, at::kFloat),
               d = dense(d0, at::kFloat);
  Tensor out = empty({B, 1, 8, 128}, at::kBFloat16, q), ns = empty({B, 8, 128, 128}, at::kFloat, q);
  void *p0 = ptr(q), *p1 = ptr(k), *p2 = ptr(v), *p3 = has_state ? ptr(sc) : nullptr, *p4 = ptr(A), *p5 = ptr(av), *p6 = ptr(d),
       *p7 = ptr(bv), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_gdn_decode(p0, p1, p2, (const float*)p3, (const float*)p4, p5, (const float*)p6, p7, scale,
                                         out.data_ptr(), (float*)ns.data_ptr(), B, st);
               }),
               "ako4x_gdn_decode");
  return pack_tuple(std::move(out), std::move(ns));
  END_HANDLE_TH_ERRORS
}

// The ten arguments of gdn_prefill.run, then a flag: whether a workspace (the chunked form) is used.
PyObject* gdn_prefill(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  count(nargs, 11, "gdn_prefill");
  c10::NoGradGuard ng;
  const Tensor &q0 = tensor(a[0]), &k0 = tensor(a[1]), &v0 = tensor(a[2]), &A0 = tensor(a[4]), &a0 = tensor(a[5]),
               &d0 = tensor(a[6]), &b0 = tensor(a[7]), &cu0 = tensor(a[8]);
  const bool has_state = a[3] != Py_None;
  need(q0.dim() == 3 && q0.size(1) == 4 && q0.size(2) == 128 && k0.sizes() == q0.sizes(),
       "gdn_prefill: q and k must be [tokens, 4, 128]");
  const int64_t T = q0.size(0);
  need(shape_is(v0, {T, 8, 128}), "gdn_prefill: v must be [tokens, 8, 128]");
  for (const Tensor* t : {&q0, &k0, &v0, &a0, &b0})
    need(t->scalar_type() == at::kBFloat16, "gdn_prefill: q, k, v, a, b must be bf16");
  need(A0.numel() == 8 && d0.numel() == 8 && a0.numel() == T * 8 && b0.numel() == T * 8,
       "gdn_prefill: A_log, dt_bias must have 8 elements, a and b tokens * 8");
  const int64_t n = cu0.numel() - 1;
  need(n >= 0, "gdn_prefill: cu_seqlens must have num_seqs + 1 entries");
  Tensor sc;
  if (has_state) {
    const Tensor& s0 = tensor(a[3]);
    need(shape_is(s0, {n, 8, 128, 128}) && s0.scalar_type() == at::kFloat,
         "gdn_prefill: state must be fp32 [num_seqs, 8, 128, 128]");
    sc = dense(s0);
  }
  const float scale = gdn_scale(a[9]);
  const bool use_ws = PyObject_IsTrue(a[10]) == 1;
  const Tensor q = dense(q0), k = dense(k0), v = dense(v0), av = dense(a0), bv = dense(b0), A = dense(A0, at::kFloat),
               d = dense(d0, at::kFloat), cu = dense(cu0, at::kLong);
  Tensor out = empty({T, 8, 128}, at::kBFloat16, q), ns = empty({n, 8, 128, 128}, at::kFloat, q);
  Workspace ws(use_ws ? ako4x_gdn_prefill_workspace_bytes(T, n) : 0, q);
  if (!ws.p) out.zero_();   // tokens outside every sequence are zero (the chunked form writes them itself)
  void *p0 = ptr(q), *p1 = ptr(k), *p2 = ptr(v), *p3 = has_state ? ptr(sc) : nullptr, *p4 = ptr(A), *p5 = ptr(av), *p6 = ptr(d),
       *p7 = ptr(bv), *p8 = ptr(cu), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_gdn_prefill(p0, p1, p2, (const float*)p3, (const float*)p4, p5, (const float*)p6, p7,
                                          (const int64_t*)p8, scale, out.data_ptr(), (float*)ns.data_ptr(), T, n, ws.p, ws.bytes,
                                          st);
               }),
               "ako4x_gdn_prefill");
  return pack_tuple(std::move(out), std::move(ns));
  END_HANDLE_TH_ERRORS
}

PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  count(n, 2, "gemm");
  c10::NoGradGuard ng;
  const Tensor &A0 = tensor(a[0]), &B0 = tensor(a[1]);
  need(A0.dim() == 2 && B0.dim() == 2 && A0.size(1) == B0.size(1), "gemm: A must be [M, K] and B [N, K]");
  const ScalarType dt = A0.scalar_type();
  need(B0.scalar_type() == dt && (dt == at::kHalf || dt == at::kBFloat16), "gemm: fp16 or bf16 operands of one type expected");
  const int64_t m = A0.size(0), k = A0.size(1), nn = B0.size(0);
  const Tensor A = dense(A0), B = dense(B0);
  Tensor c = empty({m, nn}, dt, A);
  // small and medium M split K over CTAs; the fp32 partial products live in this workspace
  Workspace ws(ako4x_gemm_workspace_bytes(m, nn, k), A);
  void *p0 = ptr(A), *p1 = ptr(B), *st = current_stream();
  check_status(without_gil([&] {
                 return ako4x_gemm_f16_nt_ws(p0, p1, c.data_ptr(), m, nn, k, dt == at::kBFloat16 ? 1 : 0, ws.p, ws.bytes, st);
               }),
               "ako4x_gemm_f16_nt_ws");
  return pack(std::move(c));
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
#define AKO_METHOD(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
    AKO_METHOD(rmsnorm),       AKO_METHOD(gqa_decode),  AKO_METHOD(mla_decode),
    AKO_METHOD(mla_prefill),   AKO_METHOD(dsa_indexer), AKO_METHOD(dsa_attention),
    AKO_METHOD(dsa_indexer_attention), AKO_METHOD(quantize_1x128), AKO_METHOD(index_k_cache_write),
    AKO_METHOD(moe),           AKO_METHOD(gdn_decode),  AKO_METHOD(gdn_prefill),
    AKO_METHOD(gemm),          {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Native operator entry points.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  PyObject* cabi = PyImport_ImportModule("ako4x_b200._cabi");
  if (!cabi) return nullptr;
  g_error = PyObject_GetAttrString(cabi, "Ako4xError");
  Py_DECREF(cabi);
  if (!g_error) return nullptr;
  return PyModule_Create(&kModule);
}
