// Call path from Python to kernels that last a few microseconds: one call per operator that checks its tensors, allocates the
// results and launches, instead of a dozen Python and ctypes steps. A decoder layer's four small kernels (64 sequences) took
// 50 us of host time for 11 us of GPU time through ctypes, a dispatch and combine of 100 tokens about 85 us,
// a low-latency dispatch and combine 22.5 (18.7 through here).
// The checks are those of the Python functions that call in here (umdk_b200/ops), and raise as they did.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include "ep_params.h"

extern "C" {
int umdk_add_rmsnorm(const void*, const void*, const void*, const void*, void*, void*, int, int, int, float, void*);
int umdk_qkv_post(const void*, int, int, const void*, const void*, const float*, const float*, void*, void*, const long long*,
                  long long, float, int*, void*);
int umdk_q_rope(const void*, int, int, int, const float*, const float*, void*, void*);
int umdk_router_topk(const void*, int, int, int, int, int, long long*, float*, void*);
int umdk_sparse_mla_decode(const void*, const void*, const int*, const int*, const int*, void*, float*, float*, float*, int, int,
                           int, int, int, float, int*, void*, long long*);
int umdk_ep_layout(const int64_t*, int, int, int, int, int*, int*, uint8_t*, int*, int*, int*, uint32_t*, int*, void*);
int umdk_ep_dispatch(const UmdkEpDispatchParams*, void*);
int umdk_ep_combine(const UmdkEpCombineParams*, void*);
int umdk_ep_ll_dispatch(const UmdkEpLLDispatchParams*, void*);
int umdk_ep_ll_combine(const UmdkEpLLCombineParams*, void*);
}

namespace {

using at::Tensor;
using NoGil = pybind11::gil_scoped_release;

struct Assertion {};   // a failed check, reported as Python's assert statement does
void check(bool ok) {
  if (!ok) throw Assertion();
}

// Arguments of one call, in order.
struct Args {
  PyObject* const* a;
  Py_ssize_t n, i = 0;
  PyObject* next() {
    if (i >= n) throw python_error_of("too few arguments");
    return a[i++];
  }
  static python_error python_error_of(const char* msg) {
    PyErr_SetString(PyExc_TypeError, msg);
    return python_error();
  }
  const Tensor& tensor() {
    PyObject* o = next();
    if (!THPVariable_Check(o)) throw python_error_of("expected a tensor");
    return THPVariable_Unpack(o);
  }
  Tensor maybe() {   // undefined for None
    PyObject* o = next();
    if (o == Py_None) return Tensor();
    if (!THPVariable_Check(o)) throw python_error_of("expected a tensor or None");
    return THPVariable_Unpack(o);
  }
  long long integer() {
    const long long v = PyLong_AsLongLong(next());
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
  }
  bool truth() {
    const int v = PyObject_IsTrue(next());
    if (v < 0) throw python_error();
    return v != 0;
  }
  double real() {
    const double v = PyFloat_AsDouble(next());
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return v;
  }
};

const void* cptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
template <class T = void>
T* ptr(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
Tensor empty(at::IntArrayRef sizes, at::ScalarType t, const Tensor& like) {
  return at::empty(sizes, at::TensorOptions().dtype(t).device(like.device()));
}
void ok_or_throw(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + " failed: " + std::to_string(rc));
}

PyObject* wrap(const Tensor& t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(t);
}
template <class... T>
PyObject* tuple(const T&... ts) {
  PyObject* items[] = {wrap(ts)...};
  PyObject* r = PyTuple_New(sizeof...(ts));
  for (size_t i = 0; i < sizeof...(ts); ++i) PyTuple_SET_ITEM(r, i, items[i]);
  return r;
}

// ---- decoder glue ------------------------------------------------------------------------------------------------------
PyObject* add_rmsnorm(Args v) {   // x, w, a, b, x_out, h, eps
  const Tensor x = v.tensor(), w = v.maybe(), a = v.maybe(), b = v.maybe();
  Tensor x_out = v.maybe(), h = v.maybe();
  const float eps = (float)v.real();
  check(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1);
  const int64_t T = x.size(0), H = x.size(1);
  {
    NoGil nogil;
    if (!h.defined()) h = empty({T, H}, at::kBFloat16, x);
    if (!a.defined() && !b.defined()) x_out = Tensor();
    else if (!x_out.defined()) x_out = empty({T, H}, at::kBFloat16, x);
    for (const Tensor* t : {&a, &b})
      check(!t->defined() ||
            (t->is_contiguous() && t->dim() == 2 && t->size(0) == T && t->size(1) == H && t->scalar_type() == at::kBFloat16));
    ok_or_throw(umdk_add_rmsnorm(cptr(x), cptr(a), cptr(b), cptr(w), ptr(x_out), ptr(h), (int)T, (int)H, (int)x.stride(0), eps,
                                 stream()),
                "umdk_add_rmsnorm");
  }
  return x_out.defined() ? tuple(x_out, h) : tuple(x, h);
}

PyObject* qkv_post(Args v) {   // qkv, q_lora, q_norm, kv_norm, cos, sin, kv_pool, new_row, status, qa, eps
  const Tensor qkv = v.tensor();
  const int64_t q_lora = v.integer();
  const Tensor q_norm = v.maybe(), kv_norm = v.maybe(), cos = v.tensor(), sin = v.maybe(), pool = v.tensor(), row = v.tensor(),
               status = v.maybe();
  Tensor qa = v.maybe();
  const float eps = (float)v.real();
  check(qkv.is_contiguous() && qkv.dim() >= 2 && qkv.size(1) == q_lora + 576 && row.scalar_type() == at::kLong);
  check(cos.scalar_type() == at::kFloat && cos.numel() == 32 && pool.is_contiguous());
  const int64_t T = qkv.size(0);
  {
    NoGil nogil;
    if (!qa.defined()) qa = empty({T, q_lora}, at::kBFloat16, qkv);
    ok_or_throw(umdk_qkv_post(cptr(qkv), (int)T, (int)q_lora, cptr(q_norm), cptr(kv_norm), ptr<float>(cos), ptr<float>(sin), ptr(qa),
                              ptr(pool), ptr<long long>(row), (long long)(pool.numel() / 576), eps, ptr<int>(status), stream()),
                "umdk_qkv_post");
  }
  return wrap(qa);
}

PyObject* q_rope(Args v) {   // q, nope, cos, sin, q_full
  const Tensor q = v.tensor();
  const int64_t nope = v.integer();
  const Tensor cos = v.maybe(), sin = v.maybe(), q_full = v.tensor();
  check(q.is_contiguous() && q_full.is_contiguous() && q.dim() >= 3 && q_full.dim() >= 1 && q_full.size(-1) == 576);
  {
    NoGil nogil;
    ok_or_throw(umdk_q_rope(cptr(q), (int)(q.size(0) * q.size(1)), (int)q.size(2), (int)nope, ptr<float>(cos), ptr<float>(sin),
                            ptr(q_full), stream()),
                "umdk_q_rope");
  }
  Py_RETURN_NONE;
}

PyObject* router_topk(Args v) {   // logits, k, fold_el, rank
  const Tensor lg = v.tensor();
  const int64_t k = v.integer(), fold = v.integer(), rank = v.integer();
  check(lg.is_cuda() && lg.scalar_type() == at::kBFloat16 && lg.is_contiguous() && lg.dim() == 2);
  const int64_t T = lg.size(0), E = lg.size(1), ko = k + (fold > 0 ? 1 : 0);
  Tensor idx, w;
  {
    NoGil nogil;
    idx = empty({T, ko}, at::kLong, lg);
    w = empty({T, ko}, at::kFloat, lg);
    ok_or_throw(umdk_router_topk(cptr(lg), (int)T, (int)E, (int)k, (int)fold, (int)rank, ptr<long long>(idx), ptr<float>(w),
                                 stream()),
                "umdk_router_topk");
  }
  return tuple(idx, w);
}

// ---- attention ---------------------------------------------------------------------------------------------------------
// q, kv_pages, block_table, indices, sm_scale, seq_lens, num_splits (resolved), out, status, part_o, part_lse, diag: the caller has
// checked them
PyObject* sparse_mla_decode(Args v) {
  const Tensor q = v.tensor(), kv = v.tensor(), table = v.tensor(), indices = v.tensor();
  const float scale = (float)v.real();
  const Tensor lens = v.maybe();
  const int64_t splits = v.integer();
  Tensor out = v.maybe(), status = v.maybe(), po = v.maybe(), pl = v.maybe();
  const Tensor diag = v.maybe();
  const int64_t B = q.size(0), topk = indices.size(1), heads = q.size(1);
  Tensor lse;
  {
    NoGil nogil;
    if (!out.defined()) out = empty({B, heads, 512}, at::kBFloat16, q);
    lse = empty({B, heads}, at::kFloat, q);
    if (!status.defined()) status = at::zeros({4}, at::TensorOptions().dtype(at::kInt).device(q.device()));
    if (splits > 1 && !po.defined()) {
      po = empty({B, splits, heads, 512}, at::kFloat, q);
      pl = empty({B, splits, heads}, at::kFloat, q);
    }
    ok_or_throw(umdk_sparse_mla_decode(cptr(q), cptr(kv), ptr<int>(table), ptr<int>(indices), ptr<int>(lens), ptr(out),
                                       ptr<float>(lse), splits > 1 ? ptr<float>(po) : nullptr, splits > 1 ? ptr<float>(pl) : nullptr,
                                       (int)B, (int)topk, (int)table.size(1), (int)kv.size(0), (int)splits, scale, ptr<int>(status),
                                       stream(), ptr<long long>(diag)),
                "umdk_sparse_mla_decode");
  }
  return tuple(out, lse);
}

// ---- normal-mode expert parallelism --------------------------------------------------------------------------------------
PyObject* ep_layout(Args v) {   // topk_idx [T, K] (checked), E, R, scratch (large enough), bar, status
  const Tensor idx = v.tensor();
  const int64_t E = v.integer(), R = v.integer();
  const Tensor scratch = v.tensor(), bar = v.tensor(), status = v.tensor();
  const int64_t T = idx.size(0), K = idx.size(1);
  Tensor npe, npr, inr, sidx, slot;
  {
    NoGil nogil;
    npe = empty({E}, at::kInt, idx);
    npr = empty({R}, at::kInt, idx);
    inr = empty({T, R}, at::kBool, idx);
    sidx = empty({T, K}, at::kInt, idx);
    slot = empty({T, R}, at::kInt, idx);
    ok_or_throw(umdk_ep_layout(ptr<int64_t>(idx), (int)T, (int)K, (int)E, (int)R, ptr<int>(npe), ptr<int>(npr), ptr<uint8_t>(inr),
                               ptr<int>(sidx), ptr<int>(slot), ptr<int>(scratch), ptr<uint32_t>(bar), ptr<int>(status), stream()),
                "umdk_ep_layout");
  }
  return tuple(npe, npr, inr, sidx, slot);
}

// base (address of the block with what never changes), x (checked), topk_idx, topk_weights, send_idx, rank_slot, num_per_expert,
// num_per_rank, quant, n_cap, a_cap, row_info, num_ctas, phase_mask, host_tag, diag
// -> recv_x, recv_scales, expand_idx, recv_count, recv_per_expert, recv_meta, counts, row_expert, row_weight
PyObject* ep_dispatch(Args v) {
  UmdkEpDispatchParams p = *reinterpret_cast<const UmdkEpDispatchParams*>(v.integer());
  const Tensor x = v.tensor(), idx = v.tensor(), w = v.maybe(), sidx = v.tensor(), slot = v.tensor(), npe = v.tensor(),
               npr = v.tensor();
  p.quant = v.truth();
  const int64_t n_cap = v.integer(), a_cap = v.integer();
  const bool row_info = v.truth();
  p.num_ctas = (int)v.integer();
  p.phase_mask = (int)v.integer();
  p.host_tag = (int)v.integer();
  const Tensor diag = v.maybe();
  Tensor rx, rs, expand, count, per_expert, meta, counts, row_expert, row_weight;
  {
    NoGil nogil;
    const int64_t H = p.H;
    rx = empty({n_cap, H}, p.quant ? at::kFloat8_e4m3fn : at::kBFloat16, x);
    if (p.quant) rs = empty({n_cap, H / 128}, at::kFloat, x);
    expand = empty({n_cap, 3}, at::kInt, x);
    count = empty({p.E}, at::kInt, x);
    per_expert = empty({p.E / p.R}, at::kLong, x);
    meta = empty({a_cap, 2 * p.K + 2}, at::kInt, x);
    counts = empty({4 + kUmdkMaxRanks}, at::kInt, x);
    if (row_info) {
      row_expert = empty({n_cap}, at::kLong, x);
      row_weight = empty({n_cap}, at::kFloat, x);
    }
    p.T = (int)x.size(0);
    p.n_cap = (int)n_cap;
    p.a_cap = (int)a_cap;
    p.x = cptr(x);
    p.topk_idx = ptr<int64_t>(idx);
    p.topk_w = ptr<float>(w);
    p.send_idx = ptr<int>(sidx);
    p.rank_slot = ptr<int>(slot);
    p.num_per_expert = ptr<int>(npe);
    p.num_per_rank = ptr<int>(npr);
    p.recv_x = ptr(rx);
    p.recv_scales = ptr<float>(rs);
    p.expand_idx = ptr<int>(expand);
    p.recv_count = ptr<int>(count);
    p.recv_per_expert = ptr<int64_t>(per_expert);
    p.recv_meta = ptr<int>(meta);
    p.counts_dev = ptr<int>(counts);
    p.diag = ptr<long long>(diag);
    p.row_expert = ptr<int64_t>(row_expert);
    p.row_weight = ptr<float>(row_weight);
    ok_or_throw(umdk_ep_dispatch(&p, stream()), "umdk_ep_dispatch");
  }
  return tuple(rx, rs, expand, count, per_expert, meta, counts, row_expert, row_weight);
}

PyObject* ep_combine(Args v) {   // base, y (checked), recv_meta, counts, in_rank, T, apply_weights, num_ctas, phase_mask, out, diag
  UmdkEpCombineParams p = *reinterpret_cast<const UmdkEpCombineParams*>(v.integer());
  const Tensor y = v.tensor(), meta = v.tensor(), counts = v.tensor(), in_rank = v.tensor();
  p.T = (int)v.integer();
  p.apply_weights = v.truth();
  p.num_ctas = (int)v.integer();
  p.phase_mask = (int)v.integer();
  Tensor out = v.maybe();
  const Tensor diag = v.maybe();
  {
    NoGil nogil;
    if (!out.defined()) out = empty({p.T, p.H}, at::kBFloat16, y);
    p.mode = 0;
    p.n_rows = (int)y.size(0);
    p.a_cap = (int)meta.size(0);
    p.y = cptr(y);
    p.recv_meta = ptr<int>(meta);
    p.counts_dev = ptr<int>(counts);
    p.in_rank = ptr<uint8_t>(in_rank);
    p.out = ptr(out);
    p.diag = ptr<long long>(diag);
    ok_or_throw(umdk_ep_combine(&p, stream()), "umdk_ep_combine");
  }
  return wrap(out);
}

// ---- low-latency expert parallelism --------------------------------------------------------------------------------------
PyObject* ll_dispatch(Args v) {   // base, x, topk_idx (both checked), send_idx, num_per_expert, num_ctas, phase_mask
  UmdkEpLLDispatchParams p = *reinterpret_cast<const UmdkEpLLDispatchParams*>(v.integer());
  const Tensor x = v.tensor(), idx = v.tensor(), sidx = v.maybe(), npe = v.maybe();
  p.num_ctas = (int)v.integer();
  p.phase_mask = (int)v.integer();
  p.T = (int)x.size(0);
  p.x = cptr(x);
  p.topk_idx = ptr<int64_t>(idx);
  p.send_idx = ptr<int>(sidx);
  p.num_per_expert = ptr<int>(npe);
  {
    NoGil nogil;
    ok_or_throw(umdk_ep_ll_dispatch(&p, stream()), "umdk_ep_ll_dispatch");
  }
  Py_RETURN_NONE;
}

PyObject* ll_combine(Args v) {   // base, y, topk_idx (both checked), topk_w, out, num_ctas, phase_mask
  UmdkEpLLCombineParams p = *reinterpret_cast<const UmdkEpLLCombineParams*>(v.integer());
  const Tensor y = v.tensor(), idx = v.tensor(), w = v.tensor();
  Tensor out = v.maybe();
  p.num_ctas = (int)v.integer();
  p.phase_mask = (int)v.integer();
  {
    NoGil nogil;
    p.T = (int)idx.size(0);
    if (!out.defined()) out = empty({p.T, p.H}, at::kBFloat16, y);
    p.y = cptr(y);
    p.topk_idx = ptr<int64_t>(idx);
    p.topk_w = ptr<float>(w);
    p.out = ptr(out);
    ok_or_throw(umdk_ep_ll_combine(&p, stream()), "umdk_ep_ll_combine");
  }
  return wrap(out);
}

template <PyObject* (*F)(Args)>
PyObject* entry(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    return F(Args{a, n});
  } catch (const Assertion&) {
    PyErr_SetNone(PyExc_AssertionError);
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define ENTRY(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<f>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ENTRY(add_rmsnorm), ENTRY(qkv_post),   ENTRY(q_rope),      ENTRY(router_topk), ENTRY(sparse_mla_decode),
                         ENTRY(ep_layout),   ENTRY(ep_dispatch), ENTRY(ep_combine),  ENTRY(ll_dispatch), ENTRY(ll_combine),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "umdk_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_umdk_calls(void) { return PyModule_Create(&module); }
