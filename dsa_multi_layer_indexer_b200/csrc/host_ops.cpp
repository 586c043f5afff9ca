// Native half of ops.py: argument checks, allocation of results and the C-ABI calls of the entry
// points that a decode step or a full-sequence layer makes eagerly, in one step from Python objects
// to the launch. A ctypes call with its checks in Python cost 10-20 us per operation, more than the
// kernels of a small step take; here an operation costs one to three microseconds plus its launches.
// The library's functions arrive as addresses (bind), so the build that _lib.py loaded is the one that
// runs. Nothing here computes: it checks, allocates with torch's allocator and launches on torch's
// current stream.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <exception>
#include <initializer_list>
#include <optional>
#include <stdexcept>
#include <string>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/dsa_b200.h"

namespace {

using at::Tensor;

// ---------------------------------------------------------------- the library's functions
#define DSA_HOST_API(X)                                                                                        \
  X(dsa_indexer_scan_fp8) X(dsa_indexer_scan_fp8_paged) X(dsa_indexer_scan_f32) X(dsa_topk_workspace_bytes)    \
  X(dsa_topk_select) X(dsa_topk_select_paged) X(dsa_sparse_mla_partials) X(dsa_sparse_mla_combine)             \
  X(dsa_sparse_mla_decode) X(dsa_sparse_mla_decode_beside) X(dsa_sparse_mla_prompt) X(dsa_sparse_mla_f32) X(dsa_rmsnorm)                \
  X(dsa_add_rmsnorm_bf16) X(dsa_silu_mul_bf16) X(dsa_add_rmsnorm_f32) X(dsa_silu_mul_f32) X(dsa_linear_f32)                \
  X(dsa_indexer_stage_fp8) X(dsa_latent_append) X(dsa_prefill_latents) X(dsa_prefill_queries)
struct Api {
#define X(name) decltype(&::name) name = nullptr;
  DSA_HOST_API(X)
#undef X
} api;
PyObject* status_check = nullptr;  // _lib.check: raises for a negative status

// ---------------------------------------------------------------- errors
// Thrown without touching the interpreter (its lock may be released) and translated in entry().
struct PyErrorSet {};  // a Python exception is already set
struct ValueError {
  std::string msg;
};
struct StatusError {
  int status;
};
[[noreturn]] void bad(const std::string& msg) { throw ValueError{msg}; }
inline void need(bool cond, const char* msg) {
  if (__builtin_expect(!cond, 0)) bad(msg);
}
inline void ok(int status) {
  if (__builtin_expect(status != 0, 0)) throw StatusError{status};
}
struct NoGil {  // the interpreter's lock is released while this lives
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// The call itself runs without the interpreter's lock (a full launch queue blocks it): its arguments
// must not touch Python objects.
#define LAUNCH(expr)                         \
  do {                                       \
    int status_;                             \
    Py_BEGIN_ALLOW_THREADS status_ = (expr); \
    Py_END_ALLOW_THREADS ok(status_);        \
  } while (0)

// ---------------------------------------------------------------- arguments
inline const Tensor* opt(PyObject* o, const char* name) {
  if (o == Py_None) return nullptr;
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor, got %s", name, Py_TYPE(o)->tp_name);
    throw PyErrorSet();
  }
  return &THPVariable_Unpack(o);
}
inline const Tensor& ten(PyObject* o, const char* name) {
  const Tensor* t = opt(o, name);
  if (!t) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor, got None", name);
    throw PyErrorSet();
  }
  return *t;
}
inline int64_t integer(PyObject* o) {
  int64_t v = PyLong_Check(o) ? PyLong_AsLongLong(o) : -1;
  if (!PyLong_Check(o)) {  // numpy integers and the like
    PyObject* i = PyNumber_Index(o);
    if (!i) throw PyErrorSet();
    v = PyLong_AsLongLong(i);
    Py_DECREF(i);
  }
  if (v == -1 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
// int(o): for the arguments that Python code converted so, where a float or a one-element tensor was taken.
inline int64_t whole(PyObject* o) {
  if (PyLong_Check(o)) return integer(o);
  PyObject* i = PyNumber_Long(o);
  if (!i) throw PyErrorSet();
  const int64_t v = PyLong_AsLongLong(i);
  Py_DECREF(i);
  if (v == -1 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
inline double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyErrorSet();
  return v;
}
inline bool truth(PyObject* o) { return PyObject_IsTrue(o) == 1; }
void contig(const Tensor& t, const char* name, std::initializer_list<at::ScalarType> types, bool pinned_too = false) {
  if (!t.is_cuda() && !(pinned_too && t.is_pinned()))
    bad(std::string(name) + (pinned_too ? " must be a CUDA tensor or pinned host memory" : " must be a CUDA tensor"));
  if (!t.is_contiguous()) bad(std::string(name) + " must be contiguous");
  const at::ScalarType st = t.scalar_type();
  for (at::ScalarType x : types)
    if (x == st) return;
  std::string msg = std::string(name) + " has dtype " + c10::toString(st) + ", expected one of";
  for (at::ScalarType x : types) msg += std::string(" ") + c10::toString(x);
  bad(msg);
}
inline void* ptr(const Tensor& t) { return t.data_ptr(); }
inline void* ptr(const Tensor* t) { return t ? t->data_ptr() : nullptr; }
template <class T>
inline T* as(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <class T>
inline T* as(const Tensor* t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }
inline void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
inline Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
}
const Tensor* lens_of(PyObject* o, int64_t rows) {
  const Tensor* t = opt(o, "seq_lens");
  if (t) {
    contig(*t, "seq_lens", {at::kInt});
    if (t->numel() != rows)
      bad("seq_lens has " + std::to_string(t->numel()) + " entries, expected " + std::to_string(rows));
  }
  return t;
}
const Tensor* hist_of(PyObject* o, int64_t rows) {
  const Tensor* t = opt(o, "hist");
  if (t) {
    contig(*t, "hist", {at::kInt, at::kUInt32});
    need(t->numel() == rows * DSA_TOPK_HIST_BINS, "hist must be [R, 4096]");
  }
  return t;
}
inline PyObject* same(PyObject* o) {
  Py_INCREF(o);
  return o;
}
// `given` when the caller passed the buffer, else a wrapper of the new tensor.
inline PyObject* result(PyObject* given, const Tensor& t) { return given != Py_None ? same(given) : THPVariable_Wrap(t); }
PyObject* columns(PyObject* given, const Tensor& t, int64_t n) {
  if (t.size(1) == n) return result(given, t);
  return THPVariable_Wrap(t.narrow(1, 0, n));
}

constexpr auto kFp8 = at::kFloat8_e4m3fn;

// ---------------------------------------------------------------- indexer scan
// (index_q, index_w, index_k, k_scale, seq_lens, rows_per_seq, ctx, out, hist, impl)
PyObject* scan_fp8(PyObject* const* a) {
  const Tensor &q = ten(a[0], "index_q"), &w = ten(a[1], "index_w"), &k = ten(a[2], "index_k"), &ks = ten(a[3], "k_scale");
  contig(q, "index_q", {kFp8, at::kByte});
  contig(w, "index_w", {at::kFloat});
  contig(k, "index_k", {kFp8, at::kByte});
  contig(ks, "k_scale", {at::kFloat});
  need(q.dim() == 3 && q.size(2) == DSA_INDEX_DIM, "index_q must be [R, Hidx, 128]");
  const int64_t R = q.size(0), heads = q.size(1), rps = integer(a[5]);
  need(w.dim() == 2 && w.size(0) == R && w.size(1) == heads, "index_w must be [R, Hidx]");
  int64_t n_seq = 1, cap;
  if (k.dim() == 2) {
    need(k.size(1) == DSA_INDEX_DIM, "index_k must be [n_seq, cap, 128]");
    cap = k.size(0);
    need(ks.numel() == cap, "k_scale must be [n_seq, cap]");
  } else {
    need(k.dim() == 3 && k.size(2) == DSA_INDEX_DIM, "index_k must be [n_seq, cap, 128]");
    n_seq = k.size(0), cap = k.size(1);
    need(ks.dim() == 2 && ks.size(0) == n_seq && ks.size(1) == cap, "k_scale must be [n_seq, cap]");
  }
  if (R != n_seq * rps)
    bad("R=" + std::to_string(R) + " must equal n_seq=" + std::to_string(n_seq) + " * rows_per_seq=" + std::to_string(rps));
  const int64_t ctx = a[6] == Py_None ? cap : whole(a[6]);
  need(ctx > 0 && ctx <= cap, "ctx must be in (0, cap]");
  const Tensor* lens = lens_of(a[4], R);
  const Tensor* given = opt(a[7], "out");
  const Tensor out = given ? *given : fresh({R, (ctx + 3) / 4 * 4}, at::kFloat, q);
  contig(out, "out", {at::kFloat});
  need(out.dim() == 2 && out.size(0) == R && out.size(1) >= ctx, "out must be [R, >= ctx]");
  const Tensor* hist = hist_of(a[8], R);
  const int impl = int(integer(a[9]));
  void* st = stream();
  LAUNCH(api.dsa_indexer_scan_fp8(as<uint8_t>(q), as<float>(w), as<uint8_t>(k), as<float>(ks), as<int32_t>(lens), as<float>(out),
                              as<uint32_t>(hist), int(R), int(rps), int(heads), ctx, n_seq, cap, cap, out.size(1),
                              impl, st));
  return columns(a[7], out, ctx);
}

// (index_q, index_w, pages, page_table, seq_lens, ctx, out, hist)
PyObject* scan_paged(PyObject* const* a) {
  const Tensor &q = ten(a[0], "index_q"), &w = ten(a[1], "index_w"), &pages = ten(a[2], "index_k_pages"),
               &table = ten(a[3], "page_table");
  contig(q, "index_q", {kFp8, at::kByte});
  contig(w, "index_w", {at::kFloat});
  contig(pages, "index_k_pages", {at::kByte});
  contig(table, "page_table", {at::kInt});
  need(q.dim() == 3 && q.size(2) == DSA_INDEX_DIM, "index_q must be [R, Hidx, 128]");
  const int64_t R = q.size(0), heads = q.size(1), ctx = integer(a[5]);
  need(pages.dim() == 2 && pages.size(1) == DSA_INDEX_PAGE_BYTES, "index_k_pages must be [num_pages, 8448]");
  need(table.dim() == 2 && table.size(0) == R, "page_table must be [R, pt_stride]");
  const Tensor* lens = lens_of(a[4], R);
  need(lens != nullptr, "paged scan needs seq_lens");
  const Tensor* given = opt(a[6], "out");
  const Tensor out = given ? *given : fresh({R, (ctx + 3) / 4 * 4}, at::kFloat, q);
  contig(out, "out", {at::kFloat});
  need(out.dim() == 2 && out.size(0) == R && out.size(1) >= ctx, "out must be [R, >= ctx]");
  need(w.dim() == 2 && w.size(0) == R && w.size(1) == heads, "index_w must be [R, Hidx]");
  need(table.size(1) * DSA_PAGE_TOKENS >= ctx, "page_table rows cannot cover ctx positions");
  const Tensor* hist = hist_of(a[7], R);
  void* st = stream();
  LAUNCH(api.dsa_indexer_scan_fp8_paged(as<uint8_t>(q), as<float>(w), as<uint8_t>(pages), pages.size(0), as<int32_t>(table),
                                    table.size(1), as<int32_t>(lens), as<float>(out), as<uint32_t>(hist), int(R), int(heads), ctx,
                                    out.size(1), st));
  return columns(a[6], out, ctx);
}

// (index_q, index_w, index_k, seq_lens, rows_per_seq, ctx, out)
PyObject* scan_f32(PyObject* const* a) {
  const Tensor &q = ten(a[0], "index_q"), &w = ten(a[1], "index_w"), &k = ten(a[2], "index_k");
  contig(q, "index_q", {at::kFloat});
  contig(w, "index_w", {at::kFloat});
  contig(k, "index_k", {at::kFloat});
  need(q.dim() == 3, "index_q must be [R, H, D]");
  const int64_t R = q.size(0), heads = q.size(1), d = q.size(2), rps = integer(a[4]);
  need(k.dim() == 2 || k.dim() == 3, "index_k must be [n_seq, cap, D]");
  const int64_t n_seq = k.dim() == 2 ? 1 : k.size(0), cap = k.size(-2);
  const int64_t ctx = a[5] == Py_None ? cap : integer(a[5]);
  need(ctx > 0 && ctx <= cap, "ctx must be in (0, cap]");
  need(k.size(-1) == d, "index_k width differs from index_q");
  need(w.numel() >= R * heads, "index_w must be [R, H]");
  need(R == n_seq * rps, "R must equal n_seq * rows_per_seq");
  const Tensor* lens = lens_of(a[3], R);
  const Tensor* given = opt(a[6], "out");
  const Tensor out = given ? *given : fresh({R, (ctx + 3) / 4 * 4}, at::kFloat, q);
  contig(out, "out", {at::kFloat});
  need(out.dim() == 2 && out.size(0) >= R && out.size(1) >= ctx, "out must be [>= R, >= ctx]");
  void* st = stream();
  LAUNCH(api.dsa_indexer_scan_f32(as<float>(q), as<float>(w), as<float>(k), as<int32_t>(lens), as<float>(out), int(R), int(rps),
                              int(heads), int(d), ctx, cap, out.size(1), st));
  return columns(a[6], out, ctx);
}

// ---------------------------------------------------------------- top-k
// Scratch of a call: the caller's, or a fresh zeroed one where rows of n logits need any.
struct Workspace {
  Tensor own;
  void* data = nullptr;
  int64_t bytes = 0;
};
Workspace workspace_for(PyObject* given, int64_t R, int64_t n, const Tensor& like) {
  Workspace ws;
  if (const Tensor* t = opt(given, "workspace")) {
    contig(*t, "workspace", {at::kByte});
    ws.data = ptr(*t), ws.bytes = t->numel();
    return ws;
  }
  ws.bytes = api.dsa_topk_workspace_bytes(int(R), n);
  if (ws.bytes > 16) {
    ws.own = fresh({ws.bytes}, at::kByte, like).zero_();
    ws.data = ptr(ws.own);
  }
  return ws;
}

// (logits, topk, seq_lens, hist, index_map, pad, offset, out_idx, out_val, return_values, workspace)
PyObject* topk(PyObject* const* a) {
  const Tensor& x = ten(a[0], "logits");
  need(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 2, "logits must be CUDA fp32 [R, n]");
  need(x.stride(1) == 1, "logits rows must be dense");
  const int64_t R = x.size(0), n = x.size(1), k = a[7] == Py_None ? integer(a[1]) : whole(a[1]);
  const int64_t slab = R > 1 ? x.stride(0) : std::max(x.stride(0), n);
  const Tensor* lens = lens_of(a[2], R);
  const Tensor* map = opt(a[4], "index_map");
  if (map) {
    contig(*map, "index_map", {at::kInt});
    need(map->dim() == 2 && map->size(0) == R && map->size(1) == n, "index_map must be [R, n]");
  }
  need(k > 0 && k <= 65536, "topk must be in [1, 65536]");
  const std::string shape = "[" + std::to_string(R) + ", " + std::to_string(k) + "]";
  const Tensor* gi = opt(a[7], "out_idx");
  const Tensor idx = gi ? *gi : fresh({R, k}, at::kInt, x);
  contig(idx, "out_idx", {at::kInt});
  if (!(idx.dim() == 2 && idx.size(0) == R && idx.size(1) == k)) bad("out_idx must be [R, topk] = " + shape);
  const Tensor* gv = opt(a[8], "out_val");
  Tensor val;
  if (gv) val = *gv;
  else if (truth(a[9])) val = fresh({R, k}, at::kFloat, x);
  if (val.defined()) {
    contig(val, "out_val", {at::kFloat});
    if (!(val.dim() == 2 && val.size(0) == R && val.size(1) == k)) bad("out_val must be [R, topk] = " + shape);
  }
  const Tensor* hist = hist_of(a[3], R);
  const Workspace ws = workspace_for(a[10], R, n, x);
  const int32_t pad = int32_t(whole(a[5])), offset = int32_t(whole(a[6]));
  void* st = stream();
  LAUNCH(api.dsa_topk_select(as<float>(x), as<int32_t>(lens), as<uint32_t>(hist), as<int32_t>(map), as<int32_t>(idx),
                         val.defined() ? as<float>(val) : nullptr, ws.data, ws.bytes, int(R), n, slab, int(k),
                         pad, offset, st));
  PyObject* pi = result(a[7], idx);
  if (!val.defined()) return pi;
  PyObject* pv = result(a[8], val);
  PyObject* both = PyTuple_Pack(2, pi, pv);
  Py_DECREF(pi);
  Py_DECREF(pv);
  return both;
}

// (logits, topk, seq_lens, hist, page_table, pad, out_idx): the selection as slots of the 64-token pages
PyObject* topk_paged(PyObject* const* a) {
  const Tensor &x = ten(a[0], "logits"), &table = ten(a[4], "page_table"), &idx = ten(a[6], "out_idx");
  need(x.is_cuda() && x.scalar_type() == at::kFloat && x.dim() == 2 && x.stride(1) == 1, "logits must be CUDA fp32 [R, n] with dense rows");
  const int64_t R = x.size(0), n = x.size(1), k = integer(a[1]);
  const Tensor* lens = lens_of(a[2], R);
  const Tensor* hist = hist_of(a[3], R);
  contig(table, "page_table", {at::kInt});
  need(table.dim() == 2 && table.size(0) == R && table.size(1) * DSA_PAGE_TOKENS >= n, "page_table rows cannot cover the logits");
  contig(idx, "out_idx", {at::kInt});
  need(idx.dim() == 2 && idx.size(0) == R && idx.size(1) == k, "out_idx must be [R, topk]");
  const int32_t pad = int32_t(integer(a[5]));
  void* st = stream();
  LAUNCH(api.dsa_topk_select_paged(as<float>(x), as<int32_t>(lens), as<uint32_t>(hist), as<int32_t>(table), table.size(1),
                               as<int32_t>(idx), int(R), n, R > 1 ? x.stride(0) : std::max(x.stride(0), n), int(k),
                               pad, st));
  return same(a[6]);
}

// ---------------------------------------------------------------- sparse MLA
// The split count where a caller gives none. Head counts that are a multiple of 64 run on the tcgen05 kernels once the launch
// has 128 tiles of 64 heads x 64 keys: about one CTA per SM in total with 64 heads per CTA, and a split count that divides
// the tiles so no split is empty. (128 heads over bf16 rows may run on persistent pairs of CTAs, for which other counts have not
// been measured: 10-14, 19-28 and 38-56 rows of 2048 keys occupy half to three quarters of the pairs.) Smaller launches and other head counts run on the mma.sync
// kernel: two CTAs of 16 heads per SM, or one of 32 where a split has several tiles or fp8 rows. With more (row, head) pairs than SMs at most 16 splits: the merge reads
// every split's partials, and more of them cost more than the shorter splits save (2 rows x 128 heads: 12.8 us with 16
// splits, 14.9 with 32).
constexpr int64_t kSms = 148;  // the default of ops.default_nsplit, which plans are made with on any machine
int64_t default_split_count(int64_t rows, int64_t heads, int64_t k, int64_t sms) {
  const int64_t tiles = std::max<int64_t>(1, (k + 63) / 64);
  if (heads % 64 == 0 && rows * (heads / 64) * tiles >= 128) {
    const int64_t blocks = std::max<int64_t>(1, rows * (heads / 64));
    int64_t want = std::max<int64_t>(1, std::min(std::min<int64_t>(sms / blocks, 16), tiles));
    while (tiles % want) --want;
    return want;
  }
  const int64_t blocks = std::max<int64_t>(1, rows * (heads / 16));
  int64_t want = std::max<int64_t>(1, 2 * sms / blocks);
  if (rows * heads > sms) want = std::min<int64_t>(want, 16);
  return std::max<int64_t>(1, std::min(want, tiles));
}

// (rows, heads, topk, sm_count)
PyObject* default_nsplit(PyObject* const* a) {
  return PyLong_FromLongLong(default_split_count(whole(a[0]), whole(a[1]), whole(a[2]), whole(a[3])));
}

// (q, kv, indices, sm_scale, seq_lens, rows_per_seq, nsplit, acc, m, l, out, dense_keys, stage 0 both / 1 partials /
//  2 combine, beside, prompt)
PyObject* mla(PyObject* const* a) {
  const Tensor &q = ten(a[0], "q"), &kv = ten(a[1], "kv");
  contig(q, "q", {at::kBFloat16});
  need(q.dim() == 3 && q.size(2) == DSA_LATENT_DIM, "q must be [R, H, 576]");
  const int64_t R = q.size(0), H = q.size(1), rps = integer(a[5]);
  if (H % DSA_HEAD_BLOCK) bad("H=" + std::to_string(H) + " must be a multiple of 16 (pad heads with zero queries)");
  need(kv.is_cuda() && kv.is_contiguous() && (kv.dim() == 3 || kv.dim() == 2), "kv must be a contiguous CUDA [n_seq, cap, w] tensor");
  const bool fp8 = kv.scalar_type() != at::kBFloat16;
  if (!fp8) need(kv.size(-1) == DSA_LATENT_DIM, "bf16 kv rows must be 576 wide");
  else need(kv.scalar_type() == at::kByte && kv.size(-1) == DSA_FP8_LATENT_ROW, "fp8 kv rows must be 656 bytes of uint8");
  const int64_t n_seq = kv.dim() == 2 ? 1 : kv.size(0), cap = kv.size(-2);
  need(R == n_seq * rps, "R must equal n_seq * rows_per_seq");
  const Tensor* idx = opt(a[2], "indices");
  int64_t k;
  if (idx) {
    contig(*idx, "indices", {at::kInt});
    need(idx->dim() == 2 && idx->size(0) == R, "indices must be [R, topk]");
    k = idx->size(1);
  } else {
    k = a[11] == Py_None ? cap : whole(a[11]);
  }
  const Tensor* lens = lens_of(a[4], R);
  const Tensor* ga = opt(a[7], "scratch.acc");
  const int64_t nsplit = a[6] != Py_None ? integer(a[6]) : ga ? ga->size(1) : default_split_count(R, H, k, kSms);
  const int64_t stage = integer(a[12]);
  Tensor acc, m, l;
  if (ga) {
    need(ga->dim() == 4 && ga->size(0) >= R && ga->size(1) == nsplit && ga->size(2) == H, "scratch does not match the launch");
    acc = *ga, m = ten(a[8], "scratch.m"), l = ten(a[9], "scratch.l");
  } else if (nsplit > 1 || stage != 0) {  // (one split: the result is written at once)
    acc = fresh({R, nsplit, H, DSA_VALUE_DIM}, at::kFloat, q);
    m = fresh({R, nsplit, H}, at::kFloat, q);
    l = fresh({R, nsplit, H}, at::kFloat, q);
  }
  const Tensor* go = opt(a[10], "out");
  const Tensor out = go ? *go : fresh({R, H, DSA_VALUE_DIM}, at::kBFloat16, q);
  contig(out, "out", {at::kBFloat16}, true);
  need(out.numel() >= R * H * DSA_VALUE_DIM, "out must be [R, H, 512]");
  float *pa = acc.defined() ? as<float>(acc) : nullptr, *pm = m.defined() ? as<float>(m) : nullptr,
        *pl = l.defined() ? as<float>(l) : nullptr;
  const float scale = float(real(a[3]));
  const bool beside = truth(a[13]);
  need(!beside || stage == 0, "beside_previous goes with stage='both'");
  void* st = stream();
  if (stage == 0)
    LAUNCH((beside ? api.dsa_sparse_mla_decode_beside : truth(a[14]) ? api.dsa_sparse_mla_prompt : api.dsa_sparse_mla_decode)(
        ptr(q), ptr(kv), as<int32_t>(idx), as<int32_t>(lens), pa, pm, pl, ptr(out), int(R), int(rps), int(H), int(k), int(nsplit),
        scale, cap, fp8 ? 1 : 0, st));
  else if (stage == 1)
    LAUNCH(api.dsa_sparse_mla_partials(ptr(q), ptr(kv), as<int32_t>(idx), as<int32_t>(lens), pa, pm, pl, int(R), int(rps), int(H),
                                       int(k), int(nsplit), scale, cap, fp8 ? 1 : 0, st));
  else
    LAUNCH(api.dsa_sparse_mla_combine(pa, pm, pl, ptr(out), int(R), int(H), int(nsplit), st));
  return result(a[10], out);
}

// (q, kv, slots, sm_scale, next_idx, out_index_pool, skv_cap): whether the serving entry may enqueue the attention behind
// scan and top-k. Not where it will refuse its operands (a refused call leaves the last selection alone), where it
// reads the list that the top-k writes, or where the pool cannot be the top-k's index map (the selection then takes
// further launches). One call: in Python these checks took 2 us of a pass whose enqueueing takes 25.
PyObject* attention_last(PyObject* const* a) {
  const Tensor &q = ten(a[0], "q"), &kv = ten(a[1], "kv"), &slots = ten(a[2], "slots"), &next = ten(a[4], "next_idx");
  const Tensor* map = opt(a[5], "out_index_pool");
  const auto begin = [](const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()); };
  const PyNumberMethods* number = Py_TYPE(a[3])->tp_as_number;
  const bool taken = q.is_cuda() && q.scalar_type() == at::kBFloat16 && begin(q) % 16 == 0 && kv.is_cuda() && kv.is_contiguous() &&
                     kv.numel() > 0 && begin(kv) % 16 == 0 && slots.is_cuda() && number && number->nb_float;
  const bool mapped = !map || (map->scalar_type() == at::kInt && map->size(1) == integer(a[6]) && map->is_contiguous());
  const bool apart = begin(slots) + slots.nbytes() <= begin(next) || begin(next) + next.nbytes() <= begin(slots);
  return PyBool_FromLong(taken && mapped && apart);
}

// (q, kv, indices, value_dim, sm_scale, seq_lens, rows_per_seq)
PyObject* mla_f32(PyObject* const* a) {
  const Tensor &q = ten(a[0], "q"), &kv = ten(a[1], "kv");
  contig(q, "q", {at::kFloat});
  contig(kv, "kv", {at::kFloat});
  need(q.dim() == 3 && (kv.dim() == 2 || kv.dim() == 3), "q must be [R, H, Dqk], kv [n_seq, ctx, Dqk]");
  const int64_t R = q.size(0), H = q.size(1), d = q.size(2), rps = integer(a[6]), vd = integer(a[3]);
  const int64_t n_seq = kv.dim() == 2 ? 1 : kv.size(0), ctx = kv.size(-2);
  need(kv.size(-1) == d && R == n_seq * rps, "q / kv shapes disagree");
  const Tensor* idx = opt(a[2], "indices");
  if (idx) {
    contig(*idx, "indices", {at::kInt});
    need(idx->dim() == 2 && idx->size(0) >= R, "indices must be [>= R, topk]");
  }
  const Tensor* lens = lens_of(a[5], R);
  const Tensor out = fresh({R, H, vd}, at::kFloat, q);
  const float scale = float(real(a[4]));
  void* st = stream();
  LAUNCH(api.dsa_sparse_mla_f32(as<float>(q), as<float>(kv), as<int32_t>(idx), as<int32_t>(lens), as<float>(out), int(R), int(rps), int(H),
                            int(d), int(vd), idx ? int(idx->size(1)) : 0, scale, ctx, st));
  return THPVariable_Wrap(out);
}

// ---------------------------------------------------------------- norms and the MLP's product
// (x, weight, eps)
PyObject* rmsnorm(PyObject* const* a) {
  const Tensor& x0 = ten(a[0], "x");
  need(x0.is_cuda() && (x0.scalar_type() == at::kFloat || x0.scalar_type() == at::kBFloat16), "x must be CUDA fp32 / bf16");
  const Tensor x = x0.contiguous();
  const Tensor w = ten(a[1], "weight").to(x.scalar_type()).contiguous();
  const Tensor out = at::empty_like(x);
  const int64_t dim = x.size(-1);
  need(dim > 0, "rows of no elements have no norm");
  const float eps = float(real(a[2]));
  void* st = stream();
  LAUNCH(api.dsa_rmsnorm(ptr(x), ptr(w), ptr(out), x.numel() / dim, int(dim), eps, x.scalar_type() == at::kFloat ? 0 : 1, st));
  return THPVariable_Wrap(out);
}

// (x, delta, weight, eps)
PyObject* add_rmsnorm(PyObject* const* a) {
  const Tensor &x0 = ten(a[0], "x"), &d0 = ten(a[1], "delta");
  const at::ScalarType type = x0.scalar_type();
  need(x0.is_cuda() && (type == at::kBFloat16 || type == at::kFloat) && d0.scalar_type() == type && x0.sizes() == d0.sizes(),
       "x and delta must be CUDA bf16 or fp32 tensors of one shape");
  const int64_t dim = x0.size(-1);
  need(dim > 0, "rows of no elements have no norm");
  need(type == at::kFloat || (dim % 8 == 0 && dim <= 8192), "the row length must be a multiple of 8 and at most 8192");
  const Tensor x = x0.contiguous(), d = d0.contiguous();
  const Tensor w = ten(a[2], "weight").to(type).contiguous();
  const Tensor s = at::empty_like(x), out = at::empty_like(x);
  const float eps = float(real(a[3]));
  void* st = stream();
  if (type == at::kFloat)
    LAUNCH(api.dsa_add_rmsnorm_f32(as<float>(x), as<float>(d), as<float>(w), as<float>(s), as<float>(out), x.numel() / dim, int(dim), eps, st));
  else
    LAUNCH(api.dsa_add_rmsnorm_bf16(ptr(x), ptr(d), ptr(w), ptr(s), ptr(out), x.numel() / dim, int(dim), eps, st));
  PyObject *ps = THPVariable_Wrap(s), *po = THPVariable_Wrap(out);
  PyObject* both = PyTuple_Pack(2, ps, po);
  Py_DECREF(ps);
  Py_DECREF(po);
  return both;
}

// (gate, up)
PyObject* silu_mul(PyObject* const* a) {
  const Tensor &g0 = ten(a[0], "gate"), &u0 = ten(a[1], "up");
  const at::ScalarType type = g0.scalar_type();
  need(g0.is_cuda() && (type == at::kBFloat16 || type == at::kFloat) && u0.scalar_type() == type && g0.sizes() == u0.sizes(),
       "gate and up must be CUDA bf16 or fp32 tensors of one shape");
  const Tensor g = g0.contiguous(), u = u0.contiguous(), out = at::empty_like(g);
  void* st = stream();
  if (type == at::kFloat) LAUNCH(api.dsa_silu_mul_f32(as<float>(g), as<float>(u), as<float>(out), g.numel(), st));
  else LAUNCH(api.dsa_silu_mul_bf16(ptr(g), ptr(u), ptr(out), g.numel(), st));
  return THPVariable_Wrap(out);
}

// ---------------------------------------------------------------- staging of a new token
// (q_raw, k_raw, w_raw, norm_w, norm_b, eps, cos, sin, positions, index_q, index_w, cache_k, cache_scale, pages, page_table,
//  interleave, round_scale, softmax_scale)
PyObject* indexer_stage(PyObject* const* a) {
  const Tensor &q = ten(a[0], "q_raw"), &k = ten(a[1], "k_raw"), &w = ten(a[2], "w_raw"), &nw = ten(a[3], "k_norm_weight"),
               &nb = ten(a[4], "k_norm_bias"), &cs = ten(a[6], "rope_cos"), &sn = ten(a[7], "rope_sin"), &pos = ten(a[8], "positions"),
               &iq = ten(a[9], "index_q"), &iw = ten(a[10], "index_w");
  contig(q, "q_raw", {at::kBFloat16});
  contig(k, "k_raw", {at::kBFloat16});
  contig(w, "w_raw", {at::kFloat});
  contig(nw, "k_norm_weight", {at::kFloat});
  contig(nb, "k_norm_bias", {at::kFloat});
  contig(cs, "rope_cos", {at::kFloat});
  contig(sn, "rope_sin", {at::kFloat});
  contig(iw, "index_w", {at::kFloat});
  contig(pos, "positions", {at::kLong});
  contig(iq, "index_q", {at::kByte, kFp8});
  need(q.dim() == 3 && q.size(2) == DSA_INDEX_DIM, "q_raw must be [B, heads, 128]");
  const int64_t B = q.size(0), heads = q.size(1);
  need(k.dim() == 2 && k.size(0) == B && k.size(1) == DSA_INDEX_DIM && w.dim() == 2 && w.size(0) == B && w.size(1) == heads &&
           iw.sizes() == w.sizes() && iq.sizes() == q.sizes() && pos.dim() == 1 && pos.size(0) == B,
       "operand shapes disagree");
  need(nw.numel() == DSA_INDEX_DIM && nb.numel() == DSA_INDEX_DIM, "LayerNorm parameters must be [128]");
  int64_t cap = cs.size(0);
  need(cs.dim() == 2 && cs.size(1) == 32 && sn.sizes() == cs.sizes(), "rotary tables must be [cap, 32]");
  const Tensor *pages = opt(a[13], "pages"), *table = nullptr, *ck = nullptr, *csc = nullptr;
  if (pages) {
    table = &ten(a[14], "page_table");
    contig(*pages, "pages", {at::kByte});
    contig(*table, "page_table", {at::kInt});
    need(table->dim() == 2 && table->size(0) == B, "page_table must be [B, pages per sequence]");
    need(pages->numel() % DSA_INDEX_PAGE_BYTES == 0, "page pool must be whole pages");
    cap = std::min(cap, table->size(1) * DSA_PAGE_TOKENS);
  } else {
    ck = &ten(a[11], "cache_index_k"), csc = &ten(a[12], "cache_k_scale");
    contig(*ck, "cache_index_k", {at::kByte, kFp8});
    contig(*csc, "cache_k_scale", {at::kFloat});
    need(ck->dim() == 3 && ck->size(0) == B && ck->size(2) == DSA_INDEX_DIM && csc->dim() == 2 && csc->size(0) == B &&
             csc->size(1) == ck->size(1),
         "caches must be [B, cap, 128] and [B, cap]");
    cap = std::min(cap, ck->size(1));
  }
  const float eps = float(real(a[5])), head_scale = float(std::pow(double(heads), -0.5));
  const float softmax_scale = float(a[17] == Py_None ? std::pow(double(DSA_INDEX_DIM), -0.5) : real(a[17]));
  const int interleave = truth(a[15]), round_scale = truth(a[16]);
  void* st = stream();
  LAUNCH(api.dsa_indexer_stage_fp8(
      ptr(q), ptr(k), as<float>(w), as<float>(nw), as<float>(nb), eps, as<float>(cs), as<float>(sn), as<int64_t>(pos), as<uint8_t>(iq),
      as<float>(iw), as<uint8_t>(ck), as<float>(csc), as<uint8_t>(pages), pages ? pages->numel() / DSA_INDEX_PAGE_BYTES : 0,
      as<int32_t>(table), table ? table->size(1) : 0, int(B), int(heads), cap, interleave, round_scale, head_scale, softmax_scale, st));
  Py_RETURN_NONE;
}

// (kv_a, norm_w, eps, cos, sin, positions, slots, pool, interleave, format, round_scale)
PyObject* latent_append(PyObject* const* a) {
  const Tensor &kv = ten(a[0], "kv_a"), &nw = ten(a[1], "kv_norm_weight"), &cs = ten(a[3], "rope_cos"), &sn = ten(a[4], "rope_sin"),
               &pos = ten(a[5], "positions"), &slots = ten(a[6], "slots"), &pool = ten(a[7], "pool");
  contig(kv, "kv_a", {at::kBFloat16});
  contig(nw, "kv_norm_weight", {at::kFloat});
  contig(cs, "rope_cos", {at::kFloat});
  contig(sn, "rope_sin", {at::kFloat});
  contig(pos, "positions", {at::kLong});
  contig(slots, "slots", {at::kLong});
  need(kv.dim() == 2 && kv.size(1) == DSA_LATENT_DIM, "kv_a must be [B, 576]");
  const int64_t B = kv.size(0);
  need(pos.dim() == 1 && pos.size(0) == B && slots.dim() == 1 && slots.size(0) == B, "positions and slots must be [B]");
  need(nw.numel() == DSA_VALUE_DIM, "kv_norm_weight must be [512]");
  need(cs.dim() == 2 && cs.size(1) == 32 && sn.sizes() == cs.sizes(), "rotary tables must be [cap, 32]");
  const int format = int(integer(a[9])), interleave = truth(a[8]), round_scale = truth(a[10]);
  if (format == 2) {
    contig(pool, "pool", {at::kByte});
    need(pool.dim() == 2 && pool.size(1) == DSA_FP8_LATENT_ROW, "an fp8 pool is [n_slots, 656] uint8");
  } else {
    contig(pool, "pool", {at::kBFloat16});
    need(pool.dim() == 2 && pool.size(1) == DSA_LATENT_DIM, "a bf16 pool is [n_slots, 576]");
  }
  const float eps = float(real(a[2]));
  void* st = stream();
  LAUNCH(api.dsa_latent_append(ptr(kv), as<float>(nw), eps, as<float>(cs), as<float>(sn), as<int64_t>(pos), as<int64_t>(slots), ptr(pool),
                               int(B), cs.size(0), pool.size(0), interleave, format, round_scale, st));
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------- full-sequence preparation
int64_t rows_of(const Tensor* t, const char* name, at::ScalarType type) {
  if (!t) return 0;
  if (!(t->is_cuda() && t->scalar_type() == type && t->dim() == 2 && t->stride(1) == 1))
    bad(std::string(name) + " must be CUDA [rows, n] of the operands' type with dense rows");
  return t->stride(0);
}
struct Rope {
  const Tensor &mc, &ms, &ic, &is;
};
Rope rope_of(PyObject* const* a, at::ScalarType type, int64_t seq) {
  Rope r{ten(a[0], "mla_cos"), ten(a[1], "mla_sin"), ten(a[2], "idx_cos"), ten(a[3], "idx_sin")};
  for (const Tensor* t : {&r.mc, &r.ms, &r.ic, &r.is}) {
    contig(*t, "rotary table", {type});
    need(t->dim() == 2 && t->size(0) >= seq, "a rotary table is shorter than the sequence");
  }
  need(r.mc.size(1) == r.ms.size(1) && r.ic.size(1) == r.is.size(1), "the rotary tables' widths disagree");
  return r;
}
int dtype_of(at::ScalarType t) {
  need(t == at::kFloat || t == at::kBFloat16, "operands must be fp32 or bf16");
  return t == at::kFloat ? 0 : 1;
}

// (qa, kv_a, ik, q_norm_w, kv_norm_w, mla_cos, mla_sin, idx_cos, idx_sin, c_q, kv_out, ik_out, ik_scale, seq, interleave, eps)
PyObject* prefill_latents(PyObject* const* a) {
  const Tensor *qa = opt(a[0], "qa"), *kv = opt(a[1], "kv_a"), *ik = opt(a[2], "ik"), *qw = opt(a[3], "q_norm_w"),
               *kw = opt(a[4], "kv_norm_w"), *cq = opt(a[9], "c_q"), *kvo = opt(a[10], "kv_out"), *iko = opt(a[11], "ik_out"),
               *iks = opt(a[12], "ik_scale");
  const Tensor* ref = qa ? qa : kv ? kv : ik;
  need(ref != nullptr, "nothing to do");
  const at::ScalarType type = ref->scalar_type();
  const int dt = dtype_of(type);
  const int64_t qs = rows_of(qa, "qa", type), kvs = rows_of(kv, "kv_a", type), iks_ = rows_of(ik, "ik", type);
  const int64_t rows = ref->size(0), seq = integer(a[13]);
  for (const Tensor* t : {qa, kv, ik}) need(!t || t->size(0) == rows, "operand rows disagree");
  const Rope rope = rope_of(a + 5, type, seq);
  int64_t q_rank = 0, kv_rank = 0, rope_dim = 0, idx_dim = 0, kv_cap = 0, ik_cap = 0;
  if (qa) {
    q_rank = qa->size(1);
    need(cq && qw, "c_q and q_norm_w go with qa");
    contig(*cq, "c_q", {type});
    need(cq->numel() == rows * q_rank && qw->numel() == q_rank && qw->scalar_type() == type, "c_q / q_norm_w shapes");
  }
  if (kv) {
    rope_dim = rope.mc.size(1), kv_rank = kv->size(1) - rope_dim;
    need(kvo && kw, "kv_out and kv_norm_w go with kv_a");
    contig(*kvo, "kv_out", {type});
    need(kvo->dim() == 3 && kvo->size(2) == kv->size(1) && kvo->size(0) * seq == rows && kvo->size(1) >= seq && kw->numel() == kv_rank &&
             kw->scalar_type() == type,
         "kv_out must be [n_seq, cap, w]");
    kv_cap = kvo->size(1);
  }
  if (ik) {
    idx_dim = ik->size(1);
    need(iko != nullptr, "ik_out goes with ik");
    if (iks) contig(*iko, "ik_out", {at::kByte, kFp8});
    else contig(*iko, "ik_out", {type});
    need(iko->dim() == 3 && iko->size(2) == idx_dim && iko->size(0) * seq == rows && iko->size(1) >= seq && rope.ic.size(1) == idx_dim,
         "ik_out must be [n_seq, cap, D]");
    ik_cap = iko->size(1);
    if (iks) {
      contig(*iks, "ik_scale", {at::kFloat});
      need(iks->dim() == 2 && iks->size(0) == iko->size(0) && iks->size(1) == ik_cap, "ik_scale must be [n_seq, cap]");
    }
  }
  const int interleave = truth(a[14]);
  const float eps = float(real(a[15]));
  void* st = stream();
  LAUNCH(api.dsa_prefill_latents(ptr(qa), qs, ptr(kv), kvs, ptr(ik), iks_, ptr(qw), ptr(kw), ptr(rope.mc), ptr(rope.ms), ptr(rope.ic),
                                 ptr(rope.is), ptr(cq), ptr(kvo), kv_cap, ptr(iko), as<float>(iks), ik_cap, rows, int(seq), int(q_rank),
                                 int(kv_rank), int(rope_dim), int(idx_dim), interleave, eps, dt, st));
  Py_RETURN_NONE;
}

// (q, nope, iq, w, mla_cos, mla_sin, idx_cos, idx_sin, q_full, index_q, index_w, seq, interleave)
PyObject* prefill_queries(PyObject* const* a) {
  const Tensor *q = opt(a[0], "q"), *iq = opt(a[2], "iq"), *w = opt(a[3], "w"), *qf = opt(a[8], "q_full"), *iqo = opt(a[9], "index_q"),
               *iwo = opt(a[10], "index_w");
  const Tensor* ref = q ? q : iq;
  need(ref != nullptr, "nothing to do");
  const at::ScalarType type = ref->scalar_type();
  const int dt = dtype_of(type);
  const int64_t rows = ref->size(0), seq = integer(a[11]), nope = integer(a[1]);
  const Rope rope = rope_of(a + 4, type, seq);
  int64_t H = 0, Hidx = 0, kv_rank = 0, rope_dim = 0, idx_dim = 0, qs = 0, qh = 0;
  const int64_t iqs = rows_of(iq, "iq", type), ws = rows_of(w, "w", type);
  if (q) {
    rope_dim = rope.mc.size(1);
    need(q->is_cuda() && q->scalar_type() == type && q->dim() == 3 && q->stride(2) == 1 && q->size(2) == nope + rope_dim,
         "q must be [rows, H, nope + rope]");
    H = q->size(1), qs = q->stride(0), qh = q->stride(1);
    need(qf != nullptr, "q_full goes with q");
    contig(*qf, "q_full", {type});
    need(qf->dim() == 3 && qf->size(0) == rows && qf->size(1) == H, "q_full must be [rows, H, kv_rank + rope]");
    kv_rank = qf->size(2) - rope_dim;
  }
  if (iq) {
    need(iqo != nullptr, "index_q goes with iq");
    if (iwo) contig(*iqo, "index_q", {at::kByte, kFp8});
    else contig(*iqo, "index_q", {type});
    need(iqo->dim() == 3 && iqo->size(0) == rows, "index_q must be [rows, Hidx, D]");
    Hidx = iqo->size(1), idx_dim = iqo->size(2);
    need(iq->size(0) == rows && iq->size(1) == Hidx * idx_dim && rope.ic.size(1) == idx_dim, "iq must be [rows, Hidx * D]");
    if (iwo) {
      contig(*iwo, "index_w", {at::kFloat});
      need(w && w->size(0) == rows && w->size(1) == Hidx && iwo->numel() == rows * Hidx, "w must be [rows, Hidx]");
    }
  }
  const int interleave = truth(a[12]);
  void* st = stream();
  LAUNCH(api.dsa_prefill_queries(ptr(q), qs, qh, int(nope), ptr(iq), iqs, ptr(w), ws, ptr(rope.mc), ptr(rope.ms), ptr(rope.ic), ptr(rope.is),
                                 ptr(qf), ptr(iqo), as<float>(iwo), rows, int(seq), int(H), int(Hidx), int(kv_rank), int(rope_dim),
                                 int(idx_dim), interleave, dt, st));
  Py_RETURN_NONE;
}

// ---------------------------------------------------------------- a full-sequence layer
// The chain DSALayer runs per layer of a prompt, without the interpreter between its launches: at a few
// hundred tokens of the small preset a layer is some twenty launches of 3-8 us, and calling each from
// Python took twice that.

// Up to this many multiply-adds a product of fp32 matrices goes to the library's own small-tile kernel,
// beyond it to the GEMM library (1024 x 1024 x 256,
// two weights: 23 us against the library's 19; three weights of 2^25.6 in all: 6 us against 20).
constexpr double kSmallLinear = double(1 << 28);

// (What the GEMM library would refuse - a weight of another device, type or inner dimension - goes to it.)
bool small_f32(const Tensor& x, std::initializer_list<const Tensor*> ws) {
  if (!x.is_cuda() || x.dim() != 2 || x.scalar_type() != at::kFloat || !x.is_contiguous() || (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15u))
    return false;
  double n = 0;
  for (const Tensor* w : ws) {
    if (w->device() != x.device() || w->scalar_type() != at::kFloat || w->dim() != 2 || w->size(1) != x.size(1) || !w->is_contiguous() ||
        (reinterpret_cast<uintptr_t>(w->data_ptr()) & 15u))
      return false;
    n += double(w->size(0));
  }
  return x.size(1) % 4 == 0 && double(x.size(0)) * n * double(x.size(1)) <= kSmallLinear;
}
// y_i = x w_i^T for weights that read the same rows x.
void linears(const Tensor& x, std::initializer_list<std::pair<const Tensor*, Tensor*>> jobs) {
  const Tensor* w[3] = {};
  Tensor* y[3] = {};
  int n = 0;
  bool small = x.scalar_type() == at::kFloat;
  for (const auto& j : jobs)
    if (j.first) w[n] = j.first, y[n++] = j.second;
  if (n == 0) return;
  small = small && (n == 1 ? small_f32(x, {w[0]}) : n == 2 ? small_f32(x, {w[0], w[1]}) : small_f32(x, {w[0], w[1], w[2]}));
  if (!small) {
    for (int i = 0; i < n; ++i) *y[i] = at::mm(x, w[i]->t());
    return;
  }
  for (int i = 0; i < n; ++i) *y[i] = fresh({x.size(0), w[i]->size(0)}, at::kFloat, x);
  void* st = stream();
  ok(api.dsa_linear_f32(as<float>(x), x.size(0), int(x.size(1)), as<float>(w[0]), int(w[0]->size(0)), as<float>(*y[0]), as<float>(w[1]),
                            w[1] ? int(w[1]->size(0)) : 0, y[1] ? as<float>(*y[1]) : nullptr, as<float>(w[2]),
                            w[2] ? int(w[2]->size(0)) : 0, y[2] ? as<float>(*y[2]) : nullptr, 0, st));
}
Tensor linear_of(const Tensor& x, const Tensor& w) {
  Tensor y;
  linears(x, {{&w, &y}});
  return y;
}

// (modules, names, nn.Linear, nn.Parameter, torch.Tensor, bf16) -> the weights of the named modules of a layer, or None
// unless every one of them is a bias-free nn.Linear of fp32 or bf16 that only multiplies by its weight: nothing hooked,
// replaced, patched (a `forward` of the instance) or quantised (a tensor subclass has its own product).
PyObject* plain_weights(PyObject* const* a) {
  static PyObject *s_hooks = PyUnicode_InternFromString("_forward_hooks"), *s_pre = PyUnicode_InternFromString("_forward_pre_hooks"),
                  *s_forward = PyUnicode_InternFromString("forward"), *s_params = PyUnicode_InternFromString("_parameters"),
                  *s_weight = PyUnicode_InternFromString("weight"), *s_bias = PyUnicode_InternFromString("bias");
  if (!PyDict_Check(a[0]) || !PyTuple_Check(a[1])) bad("plain_weights(modules, names, ...)");
  const at::ScalarType type = truth(a[5]) ? at::kBFloat16 : at::kFloat;
  const Py_ssize_t n = PyTuple_GET_SIZE(a[1]);
  PyObject* out = PyList_New(n);
  if (!out) throw PyErrorSet();
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* m = PyDict_GetItem(a[0], PyTuple_GET_ITEM(a[1], i));
    PyObject* w = nullptr;
    if (m && reinterpret_cast<PyObject*>(Py_TYPE(m)) == a[2]) {
      PyObject* d = PyObject_GenericGetDict(m, nullptr);  // a new reference; what is looked up in it lives as long
      if (!d) PyErr_Clear();
      const auto none = [&](PyObject* key) {  // no hooks
        PyObject* h = PyDict_GetItem(d, key);
        return h && PyDict_Check(h) && PyDict_Size(h) == 0;
      };
      PyObject* params = d ? PyDict_GetItem(d, s_params) : nullptr;
      if (params && PyDict_Check(params) && none(s_hooks) && none(s_pre) && PyDict_Contains(d, s_forward) == 0) {
        PyObject *weight = PyDict_GetItem(params, s_weight), *bias = PyDict_GetItem(params, s_bias);
        PyObject* kind = weight ? reinterpret_cast<PyObject*>(Py_TYPE(weight)) : nullptr;
        if ((!bias || bias == Py_None) && (kind == a[3] || kind == a[4]) && THPVariable_Unpack(weight).scalar_type() == type)
          w = same(weight);
      }
      Py_XDECREF(d);
    }
    if (!w) {
      Py_DECREF(out);
      Py_RETURN_NONE;
    }
    PyList_SET_ITEM(out, i, w);
  }
  return out;
}

// (x_norm, seq, c_q | None, wx | None, wc | None, q_a, kv_a, ik, q_b, iq, w, q_norm, kv_norm, kv_b,
//  mla_cos, mla_sin, idx_cos, idx_sin, kv | None, ik_out | None, ik_scale | None, attention, indexer, fp8,
//  heads, nope, index_heads, interleave, eps) -> (q_full, kv, iq, iw, ik, ik_scale)
PyObject* full_operands(PyObject* const* a) {
  const Tensor& xn = ten(a[0], "x_norm");
  const at::ScalarType type = xn.scalar_type();
  const int dt = dtype_of(type);
  const int64_t seq = integer(a[1]), hidden = xn.size(-1);
  need(seq > 0 && hidden > 0, "x_norm must be [B, S, hidden] with S, hidden > 0");
  const int64_t rows = xn.numel() / hidden;
  const Tensor *cq_in = opt(a[2], "c_q"), *wx = opt(a[3], "wx"), *wc = opt(a[4], "wc");
  const Tensor &q_a = ten(a[5], "q_a"), &kv_a = ten(a[6], "kv_a"), &ik_w = ten(a[7], "ik"), &q_b = ten(a[8], "q_b"), &iq_w = ten(a[9], "iq"),
               &w_w = ten(a[10], "w"), &q_norm = ten(a[11], "q_norm"), &kv_norm = ten(a[12], "kv_norm"), &kv_b = ten(a[13], "kv_b");
  const Rope rope = rope_of(a + 14, type, seq);
  const Tensor *kv_given = opt(a[18], "kv"), *ik_given = opt(a[19], "ik"), *iks_given = opt(a[20], "ik_scale");
  const bool attention = truth(a[21]), indexer = truth(a[22]), fp8 = truth(a[23]);
  const int64_t H = integer(a[24]), nope = integer(a[25]), Hidx = integer(a[26]);
  need(H > 0, "no heads");
  const int interleave = truth(a[27]);
  const float eps = float(real(a[28]));
  Tensor q_full, kv, iq, iw, ik, iks;
  {
    NoGil unlocked;
    const int64_t q_rank = q_a.size(0), width = kv_a.size(0), rope_dim = rope.mc.size(1), rank = width - rope_dim, D = ik_w.size(0);
    const bool keep_kv = attention || kv_given, keep_ik = indexer || ik_given;
    for (const Tensor* t : {&q_norm, &kv_norm}) contig(*t, "norm weight", {type});
    for (const Tensor* t : {&q_norm, &kv_norm, &rope.mc, &rope.ms, &rope.ic, &rope.is})
      need(t->device() == xn.device(), "norm weights and rotary tables must be on the activations' device");
    need(rope_dim > 0 && rank > 0 && rope.ic.size(1) == D, "the rotary tables' widths must be those of the projections");
    need(q_norm.numel() == q_rank && kv_norm.numel() == rank, "the norms' weights must have q_rank and kv_rank elements");
    void* st = stream();

    const Tensor x = xn.reshape({rows, hidden});
    // what reads x_norm
    Tensor qa, kva, ikr, c_q;
    if (wx && !cq_in && keep_kv && keep_ik) {
      const Tensor y = linear_of(x, *wx);
      qa = y.narrow(1, 0, q_rank), kva = y.narrow(1, q_rank, width), ikr = y.narrow(1, q_rank + width, D);
    } else {
      linears(x, {{cq_in ? nullptr : &q_a, &qa}, {keep_kv ? &kv_a : nullptr, &kva}, {keep_ik ? &ik_w : nullptr, &ikr}});
    }
    c_q = cq_in ? cq_in->reshape({rows, q_rank}).contiguous() : fresh({rows, q_rank}, type, x);
    if (kv_given) kv = *kv_given;
    else if (keep_kv) kv = fresh({rows / seq, seq, width}, type, x);
    if (ik_given) {
      ik = *ik_given;
      if (iks_given) iks = *iks_given;
    } else if (keep_ik) {
      ik = fresh({rows / seq, seq, D}, fp8 ? at::kByte : type, x);
      if (fp8) iks = fresh({rows / seq, seq}, at::kFloat, x);
    }
    if (keep_kv)
      need(kv.is_contiguous() && kv.scalar_type() == type && kv.dim() == 3 && kv.size(0) * seq == rows && kv.size(1) >= seq &&
               kv.size(2) == width,
           "latent cache: [n_seq, cap, w] of the operands' type");
    if (keep_ik)
      need(ik.is_contiguous() && ik.dim() == 3 && ik.size(0) * seq == rows && ik.size(1) >= seq && ik.size(2) == D &&
               (fp8 ? iks.defined() && iks.is_contiguous() : ik.scalar_type() == type),
           "index-key cache: [n_seq, cap, D]");
    if (qa.defined() || keep_kv || keep_ik)
      ok(api.dsa_prefill_latents(
          qa.defined() ? ptr(qa) : nullptr, qa.defined() ? qa.stride(0) : 0, keep_kv ? ptr(kva) : nullptr, keep_kv ? kva.stride(0) : 0,
          keep_ik ? ptr(ikr) : nullptr, keep_ik ? ikr.stride(0) : 0, ptr(q_norm), ptr(kv_norm), ptr(rope.mc), ptr(rope.ms), ptr(rope.ic),
          ptr(rope.is), ptr(c_q), keep_kv ? ptr(kv) : nullptr, keep_kv ? kv.size(1) : 0, keep_ik ? ptr(ik) : nullptr,
          iks.defined() ? as<float>(iks) : nullptr, keep_ik ? ik.size(1) : 0, rows, int(seq), int(q_rank), int(rank), int(rope_dim), int(D),
          interleave, eps, dt, st));

    // what reads c_q
    Tensor q, iqr, w;
    if (wc && attention && indexer) {
      const Tensor y = linear_of(c_q, *wc);
      q = y.narrow(1, 0, q_b.size(0)), iqr = y.narrow(1, q_b.size(0), iq_w.size(0)), w = y.narrow(1, q_b.size(0) + iq_w.size(0), Hidx);
    } else {
      linears(c_q, {{attention ? &q_b : nullptr, &q}, {indexer ? &iq_w : nullptr, &iqr}, {indexer ? &w_w : nullptr, &w}});
    }
    if (attention) {
      q = q.unflatten(1, {H, nope + rope_dim});
      q_full = fresh({rows, H, width}, type, x);
      const Tensor w_uk = kv_b.view({H, kv_b.size(0) / H, rank}).narrow(1, 0, nope);
      Tensor dst = q_full.narrow(2, 0, rank).transpose(0, 1);  // absorb W_UK: the GEMM writes its columns in place
      at::bmm_out(dst, q.narrow(2, 0, nope).transpose(0, 1), w_uk);
    }
    if (indexer) {
      need(iqr.size(1) == Hidx * D && w.size(1) == Hidx, "index_q_proj / index_weights_proj: wrong number of outputs");
      iq = fresh({rows, Hidx, D}, fp8 ? at::kByte : type, x);
      iw = fp8 ? fresh({rows, Hidx}, at::kFloat, x) : w.contiguous();
    }
    if (attention || indexer)
      ok(api.dsa_prefill_queries(attention ? ptr(q) : nullptr, attention ? q.stride(0) : 0, attention ? q.stride(1) : 0, int(nope),
                                     indexer ? ptr(iqr) : nullptr, indexer ? iqr.stride(0) : 0, indexer ? ptr(w) : nullptr,
                                     indexer ? w.stride(0) : 0, ptr(rope.mc), ptr(rope.ms), ptr(rope.ic), ptr(rope.is),
                                     attention ? ptr(q_full) : nullptr, indexer ? ptr(iq) : nullptr, indexer && fp8 ? as<float>(iw) : nullptr,
                                     rows, int(seq), int(H), int(Hidx), int(rank), int(rope_dim), int(D), interleave, dt, st));
  }
  PyObject* t = PyTuple_New(6);
  const Tensor* parts[6] = {&q_full, &kv, &iq, &iw, &ik, &iks};
  for (int i = 0; i < 6; ++i) PyTuple_SET_ITEM(t, i, parts[i]->defined() ? THPVariable_Wrap(*parts[i]) : same(Py_None));
  return t;
}

// (o [rows, H', rank], kv_b, o_proj, heads, v_dim) -> [rows, hidden]: W_UV per head, then o_proj
PyObject* project_output(PyObject* const* a) {
  const Tensor &o = ten(a[0], "o"), &kv_b = ten(a[1], "kv_b"), &o_proj = ten(a[2], "o_proj");
  const int64_t H = integer(a[3]), v = integer(a[4]), rows = o.size(0);
  need(H > 0, "no heads");
  Tensor y;
  {
    NoGil unlocked;
    const Tensor ov = fresh({rows, H, v}, o.scalar_type(), o);
    const int64_t per = kv_b.size(0) / H;
    const Tensor w_uv = kv_b.view({H, per, kv_b.size(1)}).narrow(1, per - v, v);
    Tensor dst = ov.transpose(0, 1);
    at::bmm_out(dst, o.narrow(1, 0, H).transpose(0, 1), w_uv.transpose(1, 2));
    y = linear_of(ov.view({rows, H * v}), o_proj);
  }
  return THPVariable_Wrap(y);
}

// (h_norm [rows, hidden], gate, up, down) -> [rows, hidden]: the SwiGLU MLP
PyObject* mlp(PyObject* const* a) {
  const Tensor &x = ten(a[0], "h_norm"), &gate = ten(a[1], "gate"), &up = ten(a[2], "up"), &down = ten(a[3], "down");
  const at::ScalarType type = x.scalar_type();
  dtype_of(type);
  Tensor y;
  {
    NoGil unlocked;
    Tensor act;
    void* st = stream();
    if (small_f32(x, {&gate, &up}) && gate.size(0) == up.size(0)) {
      act = fresh({x.size(0), gate.size(0)}, type, x);
      ok(api.dsa_linear_f32(as<float>(x), x.size(0), int(x.size(1)), as<float>(gate), int(gate.size(0)), as<float>(act), as<float>(up),
                                int(up.size(0)), nullptr, nullptr, 0, nullptr, 1, st));
    } else {
      const Tensor g = at::mm(x, gate.t()), u = at::mm(x, up.t());
      need(g.is_cuda() && g.sizes() == u.sizes(), "gate and up must have one shape");
      act = at::empty_like(g);
      if (type == at::kFloat) ok(api.dsa_silu_mul_f32(as<float>(g), as<float>(u), as<float>(act), g.numel(), st));
      else ok(api.dsa_silu_mul_bf16(ptr(g), ptr(u), ptr(act), g.numel(), st));
    }
    y = linear_of(act, down);
  }
  return THPVariable_Wrap(y);
}

// ---------------------------------------------------------------- the ABI's functions as they are
// abi_<name>(args without the stream): a pointer argument is a tensor, None or an address. For callers that
// mirror another extension's argument lists and hand over what they were given (kernels_ext.py).
template <class T>
T from_py(PyObject* o) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) return nullptr;
    if (THPVariable_Check(o)) return static_cast<T>(THPVariable_Unpack(o).data_ptr());
    return reinterpret_cast<T>(static_cast<uintptr_t>(integer(o)));
  } else if constexpr (std::is_floating_point_v<T>) {
    return T(real(o));
  } else {
    return T(integer(o));
  }
}
template <class... A, size_t... I>
void call_abi(int (*fn)(A...), PyObject* const* a, std::index_sequence<I...>) {
  using Types = std::tuple<A...>;
  std::tuple<std::tuple_element_t<I, Types>...> v{from_py<std::tuple_element_t<I, Types>>(a[I])...};
  void* st = stream();
  LAUNCH(fn(std::get<I>(v)..., st));
}
template <class... A>
PyObject* abi(int (*fn)(A...), PyObject* const* a) {
  call_abi(fn, a, std::make_index_sequence<sizeof...(A) - 1>());
  Py_RETURN_NONE;
}
template <class F>
struct AbiArgs;
template <class... A>
struct AbiArgs<int(A...)> { static constexpr int value = int(sizeof...(A)) - 1; };
PyObject* abi_scan(PyObject* const* a) { return abi(api.dsa_indexer_scan_fp8, a); }
PyObject* abi_scan_paged(PyObject* const* a) { return abi(api.dsa_indexer_scan_fp8_paged, a); }
PyObject* abi_topk(PyObject* const* a) { return abi(api.dsa_topk_select, a); }
PyObject* abi_mla(PyObject* const* a) { return abi(api.dsa_sparse_mla_decode, a); }

// ---------------------------------------------------------------- module
template <PyObject* (*fn)(PyObject* const*), int n_args>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != n_args) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", n_args, n);
    return nullptr;
  }
  try {
    // Without gradients the torch calls inside (allocations, views, library GEMMs) go straight to their
    // kernels instead of through the autograd and view-tracking keys, about a microsecond each.
    std::optional<at::AutoDispatchBelowADInplaceOrView> direct;
    if (!c10::GradMode::is_enabled()) direct.emplace();
    return fn(args);
  } catch (const PyErrorSet&) {
  } catch (const ValueError& e) {
    PyErr_SetString(PyExc_ValueError, e.msg.c_str());
  } catch (const StatusError& e) {
    PyObject* r = PyObject_CallFunction(status_check, "i", e.status);  // raises with the library's message
    if (r) PyErr_SetString(PyExc_RuntimeError, "dsa_b200: call failed");
    Py_XDECREF(r);
  } catch (...) {  // torch's own errors, as its Python functions raise them (an allocation's OutOfMemoryError among them)
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}

// bind({name: address}, check): the functions of the loaded library and the status check that raises
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2 || !PyDict_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "bind(addresses, check)");
    return nullptr;
  }
#define X(name)                                                                       \
  {                                                                                   \
    PyObject* v = PyDict_GetItemString(args[0], #name);                               \
    if (!v) {                                                                         \
      PyErr_SetString(PyExc_ImportError, "the library does not provide " #name);      \
      return nullptr;                                                                 \
    }                                                                                 \
    void* p = PyLong_AsVoidPtr(v);                                                    \
    if (!p && PyErr_Occurred()) return nullptr;                                       \
    api.name = reinterpret_cast<decltype(&::name)>(p);                                \
  }
  DSA_HOST_API(X)
#undef X
  Py_INCREF(args[1]);
  Py_XSETREF(status_check, args[1]);
  Py_RETURN_NONE;
}

#define M(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&bind)), METH_FASTCALL, nullptr},
    M(scan_fp8, 10), M(scan_paged, 8), M(scan_f32, 7), M(topk, 11), M(topk_paged, 7), M(default_nsplit, 4), M(mla, 15), M(attention_last, 7), M(mla_f32, 7), M(rmsnorm, 3),
    M(add_rmsnorm, 4), M(silu_mul, 2), M(indexer_stage, 18), M(latent_append, 11), M(prefill_latents, 16), M(prefill_queries, 13),
    M(plain_weights, 6), M(full_operands, 29), M(project_output, 5), M(mlp, 4),
    M(abi_scan, AbiArgs<decltype(::dsa_indexer_scan_fp8)>::value), M(abi_scan_paged, AbiArgs<decltype(::dsa_indexer_scan_fp8_paged)>::value),
    M(abi_topk, AbiArgs<decltype(::dsa_topk_select)>::value), M(abi_mla, AbiArgs<decltype(::dsa_sparse_mla_decode)>::value),
    {nullptr, nullptr, 0, nullptr}};
#undef M
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "native half of the tensor entry points", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }
