// Native form of the tensor-level wrappers in ops.py: checks the tensors, fills the C structs and calls the library,
// without a Python operation per field.  A wrapper tries its function here first and goes through Python when this
// one answers None: on anything but the plain case (an argument of another kind, a failed check), so that checks,
// messages and every less common form live in ops.py alone.  Once the library has been called there is no second try:
// an error code is raised as ops.py raises it (the first attempt may have enqueued launches, and has consumed the error).
//
// Measured host time per pass, through Python -> here: a decode step 24 -> 10 us, an append 26 -> 8 us, a gate step
// (prepare, scores and selection, attention) 98 -> 46 us; the decode and append kernels take 8 and 12 us.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <limits>

#include "../../include/compactattn_b200.h"

namespace {

// Entry points of the loaded library, set by bind().
struct Library {
  decltype(&ca_attn_compact) attn_compact;
  decltype(&ca_rope_append) rope_append;
  decltype(&ca_gate_prepare) gate_prepare;
  decltype(&ca_select_union_table) select_union_table;
  decltype(&ca_gate_score_select) gate_score_select;
  decltype(&ca_select_union_scratch_bytes) scratch_bytes;
  decltype(&ca_last_error) last_error;
};
Library lib = {};

struct NotPlain {};  // thrown for everything that ops.py should look at
struct Failed {};    // thrown with a Python error set

void require(bool ok) {
  if (!ok) throw NotPlain();
}

// Reads a METH_FASTCALL argument vector front to back.
class Args {
 public:
  Args(PyObject* const* v, Py_ssize_t n) : v_(v), n_(n) {}
  PyObject* next() {
    require(i_ < n_);
    return v_[i_++];
  }
  long long integer() {
    PyObject* o = next();
    require(PyLong_Check(o));
    const long long x = PyLong_AsLongLong(o);
    if (x == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      throw NotPlain();
    }
    return x;
  }
  int32_t i32() {
    const long long x = integer();
    require(x >= std::numeric_limits<int32_t>::min() && x <= std::numeric_limits<int32_t>::max());
    return static_cast<int32_t>(x);
  }
  double number() {
    PyObject* o = next();
    require(PyFloat_CheckExact(o) || PyLong_Check(o));
    const double x = PyFloat_AsDouble(o);
    if (x == -1.0 && PyErr_Occurred()) {
      PyErr_Clear();
      throw NotPlain();
    }
    return x;
  }
  // nullptr for None; only plain CUDA tensors
  const at::Tensor* optional() {
    PyObject* o = next();
    if (o == Py_None) return nullptr;
    require(THPVariable_CheckExact(o));
    const at::Tensor& t = THPVariable_Unpack(o);
    require(t.is_cuda());
    return &t;
  }
  const at::Tensor& tensor() {
    const at::Tensor* t = optional();
    require(t != nullptr);
    return *t;
  }
  void done() { require(i_ == n_); }

 private:
  PyObject* const* v_;
  Py_ssize_t n_, i_ = 0;
};

int dtype_of(const at::Tensor& t) {
  const auto d = t.scalar_type();
  if (d == at::kBFloat16) return CA_DTYPE_BF16;
  if (d == at::kHalf) return CA_DTYPE_F16;
  require(d == at::kFloat);
  return CA_DTYPE_F32;
}
void* ptr(const at::Tensor& t) { return t.data_ptr(); }
void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
bool is_int32(const at::Tensor& t) { return t.scalar_type() == at::kInt && t.is_contiguous(); }
void* stream_of(Args& a) { return reinterpret_cast<void*>(a.integer()); }

// k, v, page_stride, token_stride, head_stride, page_size, num_pages, pages_per_seq, head_div, page_table
ca_kv_layout layout(Args& a, const at::Tensor** k_out, const at::Tensor** v_out) {
  const at::Tensor &k = a.tensor(), &v = a.tensor();
  ca_kv_layout l;
  l.k = ptr(k), l.v = ptr(v);
  l.page_stride = a.integer(), l.token_stride = a.integer(), l.head_stride = a.integer();
  l.page_size = a.i32(), l.num_pages = a.i32(), l.pages_per_seq = a.i32(), l.head_div = a.i32();
  l.page_table = static_cast<const int32_t*>(ptr(a.optional()));
  *k_out = &k, *v_out = &v;
  return l;
}

// Calls the library, without the GIL: a launch waits while the stream's queue is full, and what it waits for may need
// the GIL itself (a host callback).  An error code becomes the RuntimeError of _lib.check().
template <typename F>
void enqueue(const char* what, F&& f) {
  PyThreadState* const state = PyEval_SaveThread();
  const int rc = f();
  PyEval_RestoreThread(state);
  if (rc == CA_OK) return;
  PyErr_Format(PyExc_RuntimeError, "%s failed (code %d): %s", what, rc, lib.last_error());
  throw Failed();
}

template <typename F>
PyObject* guarded(F&& body) {
  try {
    return body();
  } catch (const Failed&) {
    return nullptr;
  } catch (const NotPlain&) {
  } catch (const std::exception&) {
    // whatever it was, the same call through Python reports it
  }
  PyErr_Clear();
  Py_RETURN_NONE;
}

PyObject* bind(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a(v, n);
    lib.attn_compact = reinterpret_cast<decltype(lib.attn_compact)>(a.integer());
    lib.rope_append = reinterpret_cast<decltype(lib.rope_append)>(a.integer());
    lib.gate_prepare = reinterpret_cast<decltype(lib.gate_prepare)>(a.integer());
    lib.select_union_table = reinterpret_cast<decltype(lib.select_union_table)>(a.integer());
    lib.gate_score_select = reinterpret_cast<decltype(lib.gate_score_select)>(a.integer());
    lib.scratch_bytes = reinterpret_cast<decltype(lib.scratch_bytes)>(a.integer());
    lib.last_error = reinterpret_cast<decltype(lib.last_error)>(a.integer());
    a.done();
    Py_RETURN_TRUE;
  });
}

// (stream, workspace, q, <layout>, kv_len, num_kv_heads, block_idx, counts, block_size, softmax_scale, out, lse, status) -> out
PyObject* attn_compact(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a(v, n);
    void* stream = stream_of(a);
    const at::Tensor& ws = a.tensor();
    const at::Tensor& q = a.tensor();
    const at::Tensor *k, *val;
    ca_attn_params p = {};
    p.kv = layout(a, &k, &val);
    p.kv_len = a.i32();
    p.Hkv = a.i32();
    const at::Tensor *idx = a.optional(), *counts = a.optional();
    p.block_size = a.i32();
    PyObject* scale = a.next();
    require(q.dim() == 4 && q.stride(3) == 1);
    p.dtype = dtype_of(q);
    require(p.dtype != CA_DTYPE_F32 && k->scalar_type() == q.scalar_type() && val->scalar_type() == q.scalar_type());
    p.B = q.size(0), p.Q = q.size(1), p.Hq = q.size(2), p.D = q.size(3);
    require(scale == Py_None || PyFloat_CheckExact(scale));
    p.softmax_scale = static_cast<float>(scale == Py_None ? 1.0 / std::sqrt(static_cast<double>(p.D)) : PyFloat_AS_DOUBLE(scale));
    const at::Tensor* given = a.optional();
    const at::Tensor* lse = a.optional();
    const at::Tensor* status = a.optional();
    a.done();
    if (idx) {
      require(counts != nullptr && idx->dim() > 0 && is_int32(*idx) && is_int32(*counts));
      const int64_t cap = idx->size(-1), rows = static_cast<int64_t>(p.B) * p.Hkv;
      require(idx->numel() / (cap > 0 ? cap : 1) == rows && counts->numel() == rows);
      p.block_idx = static_cast<const int32_t*>(ptr(idx)), p.block_idx_stride = cap;
    }
    p.counts = static_cast<const int32_t*>(ptr(counts));
    if (lse) {
      require(lse->scalar_type() == at::kFloat && lse->dim() == 3 && lse->size(0) == p.B && lse->size(1) == p.Hq && lse->size(2) == p.Q &&
              lse->is_contiguous());
    }
    at::Tensor out = given ? *given : at::empty({p.B, p.Q, p.Hq, p.D}, q.options());
    require(out.dim() == 4 && out.stride(3) == 1 && out.scalar_type() == q.scalar_type());
    p.q = ptr(q), p.q_stride_b = q.stride(0), p.q_stride_t = q.stride(1), p.q_stride_h = q.stride(2);
    p.out = ptr(out), p.o_stride_b = out.stride(0), p.o_stride_t = out.stride(1), p.o_stride_h = out.stride(2);
    p.lse = static_cast<float*>(ptr(lse));
    p.status = static_cast<int32_t*>(ptr(status));
    p.workspace = ptr(ws), p.workspace_bytes = ws.nbytes();
    enqueue("ca_attn_compact", [&] { return lib.attn_compact(&p, stream); });
    return THPVariable_Wrap(out);
  });
}

// (stream, q, k, v, cos, sin, <layout>, position, mean_k, block_size, q_out, status) -> q_out
PyObject* rope_append(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a(v, n);
    void* stream = stream_of(a);
    const at::Tensor &q = a.tensor(), &k = a.tensor(), &val = a.tensor(), &cos = a.tensor(), &sin = a.tensor();
    const at::Tensor *ck, *cv;
    ca_rope_append_params p = {};
    p.cache = layout(a, &ck, &cv);
    p.position = a.i32();
    const at::Tensor* mean_k = a.optional();
    p.block_size = a.i32();
    const at::Tensor* given = a.optional();
    p.status = static_cast<int32_t*>(ptr(a.optional()));
    a.done();
    p.dtype = dtype_of(k);
    const auto type = k.scalar_type();
    require(p.dtype != CA_DTYPE_F32 && k.dim() == 4 && val.sizes() == k.sizes() && val.scalar_type() == type);
    p.B = k.size(0), p.Q = k.size(1), p.Hkv = k.size(2), p.D = k.size(3);
    require(ck->scalar_type() == type && ck->dim() > 0 && ck->size(-1) == p.D);
    require(cos.dim() == 3 && cos.sizes() == sin.sizes() && cos.strides() == sin.strides() && cos.size(1) == p.Q && cos.size(2) == p.D &&
            (cos.size(0) == 1 || cos.size(0) == p.B));
    p.rope_dtype = dtype_of(cos);
    require(sin.scalar_type() == cos.scalar_type() && (cos.scalar_type() == type || p.rope_dtype == CA_DTYPE_F32));
    require(q.dim() == 4 && q.size(0) == p.B && q.size(1) == p.Q && q.size(3) == p.D && q.scalar_type() == type);
    require(q.stride(3) == 1 && k.stride(3) == 1 && val.stride(3) == 1 && cos.stride(2) == 1);
    p.Hq = q.size(2);
    at::Tensor out = given ? *given : at::empty(q.sizes(), q.options());
    require(out.sizes() == q.sizes() && out.scalar_type() == type && out.stride(3) == 1);
    if (mean_k) {
      require(mean_k->dim() == 4 && mean_k->size(0) == p.B && mean_k->size(2) == p.Hkv && mean_k->size(3) == p.D &&
              mean_k->scalar_type() == type && mean_k->stride(3) == 1 && p.block_size > 0 && p.position >= 0 && p.position % p.block_size == 0 &&
              p.position / p.block_size + (p.Q + p.block_size - 1) / p.block_size <= mean_k->size(1));
      p.mean_k = ptr(mean_k), p.mk_stride_b = mean_k->stride(0), p.mk_stride_blk = mean_k->stride(1), p.mk_stride_h = mean_k->stride(2);
    }
    p.q = ptr(q), p.q_stride_b = q.stride(0), p.q_stride_t = q.stride(1), p.q_stride_h = q.stride(2);
    p.q_out = ptr(out), p.qo_stride_b = out.stride(0), p.qo_stride_t = out.stride(1), p.qo_stride_h = out.stride(2);
    p.k = ptr(k), p.k_stride_b = k.stride(0), p.k_stride_t = k.stride(1), p.k_stride_h = k.stride(2);
    p.v = ptr(val), p.v_stride_b = val.stride(0), p.v_stride_t = val.stride(1), p.v_stride_h = val.stride(2);
    p.cos = ptr(cos), p.sin = ptr(sin);
    p.cs_stride_b = cos.size(0) == 1 ? 0 : cos.stride(0), p.cs_stride_t = cos.stride(1);
    enqueue("ca_rope_append", [&] { return lib.rope_append(&p, stream); });
    return THPVariable_Wrap(out);
  });
}

// x, kinds (bits), weight, cos, sin, out, out_block_offset; D and C of the shapes go to the caller
ca_gate_side gate_side(Args& a, const at::Tensor** x_out, const at::Tensor** out_out) {
  const at::Tensor& x = a.tensor();
  ca_gate_side s = {};
  s.kinds = a.i32();
  const at::Tensor *w = a.optional(), *cos = a.optional(), *sin = a.optional();
  const at::Tensor& out = a.tensor();
  s.out_block_offset = a.i32();
  require(x.dim() == 4 && x.stride(3) == 1 && out.dim() == 4 && out.stride(3) == 1);
  s.x = ptr(x), s.x_stride_b = x.stride(0), s.x_stride_t = x.stride(1), s.x_stride_h = x.stride(2);
  s.x_dtype = dtype_of(x), s.H = x.size(2), s.Hw = s.H, s.rope_batch = 1;
  if (w) {
    require(w->dim() > 0 && w->is_contiguous());
    s.w = ptr(w), s.w_dtype = dtype_of(*w), s.Hw = w->size(0);
  }
  if (cos) {
    require(sin != nullptr && cos->scalar_type() == at::kFloat && sin->scalar_type() == at::kFloat && cos->is_contiguous() &&
            sin->is_contiguous() && cos->dim() > 0);
    s.cos = static_cast<const float*>(ptr(cos)), s.sin = static_cast<const float*>(ptr(sin)), s.rope_batch = cos->size(0);
  }
  require(out.size(2) == s.Hw);
  s.out = ptr(out), s.out_stride_b = out.stride(0), s.out_stride_blk = out.stride(1), s.out_stride_h = out.stride(2);
  s.out_dtype = dtype_of(out);
  *x_out = &x, *out_out = &out;
  return s;
}

// (stream, block_size, <q side>, <k side>) -> True
PyObject* gate_prepare(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a(v, n);
    void* stream = stream_of(a);
    ca_gate_prepare_params p = {};
    p.block_size = a.i32();
    const at::Tensor *q, *k, *q_out, *k_out;
    p.q = gate_side(a, &q, &q_out);
    p.k = gate_side(a, &k, &k_out);
    a.done();
    require(q->size(0) == k->size(0) && q->size(1) == k->size(1) && q->size(3) == k->size(3) && q_out->size(3) == k_out->size(3));
    p.B = q->size(0), p.L = q->size(1), p.D = q->size(3), p.C = q_out->size(3);
    enqueue("ca_gate_prepare", [&] { return lib.gate_prepare(&p, stream); });
    Py_RETURN_TRUE;
  });
}

// (stream, scratch, score, past_blocks, rule, num_kv_heads, block_size, page_size, keep_recent, valid, softmax, threshold, alpha,
//  topk_k, topk_num, topk_den, min_budget, sink, local, rows_voting, score_max, block_idx, counts, cache_seqlens, pages_per_row[,
//  q_blocks, k_blocks, scale, masked_value, write_scores]) -> (block_idx, counts, cache_seqlens, pages_per_row)
PyObject* select_union_table(PyObject*, PyObject* const* v, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    Args a(v, n);
    void* stream = stream_of(a);
    const at::Tensor &scratch = a.tensor(), &score = a.tensor();
    ca_select_params p = {};
    ca_union_params u = {};
    require(score.dim() == 4);
    p.B = score.size(0), p.H = score.size(1), p.Qb = score.size(2), p.Kb = score.size(3);
    p.Pb = a.i32();
    p.rule = a.i32();
    require(p.rule != CA_RULE_MASK);
    u.Hkv = a.i32();
    u.block_size = a.i32(), u.page_size = a.i32(), u.keep_recent = a.i32();
    if (const at::Tensor* valid = a.optional()) {
      require(valid->dim() == 4 && (valid->scalar_type() == at::kBool || valid->scalar_type() == at::kByte));
      const int64_t want[4] = {p.B, valid->size(1), p.Qb, p.Kb};
      int64_t st[4];
      for (int i = 0; i < 4; ++i) {
        require(valid->size(i) == want[i] || valid->size(i) == 1);
        st[i] = valid->size(i) == 1 && want[i] != 1 ? 0 : valid->stride(i);
      }
      p.valid = ptr(valid);
      p.valid_stride_b = st[0], p.valid_stride_h = valid->size(1) > 1 ? st[1] : 0, p.valid_stride_q = st[2], p.valid_stride_k = st[3];
    }
    p.softmax = a.i32();
    p.threshold = static_cast<float>(a.number()), p.alpha = static_cast<float>(a.number());
    p.topk_k = a.i32(), p.topk_num = a.i32(), p.topk_den = a.i32();
    p.min_budget = a.i32(), p.sink = a.i32(), p.local = a.i32(), p.rows_voting = a.i32();
    p.score = ptr(score), p.score_dtype = dtype_of(score);
    p.score_stride_b = score.stride(0), p.score_stride_h = score.stride(1), p.score_stride_q = score.stride(2), p.score_stride_k = score.stride(3);
    if (const at::Tensor* mx = a.optional()) {
      require(mx->scalar_type() == at::kFloat && p.score_dtype == CA_DTYPE_F32 && mx->sizes() == score.sizes() && mx->strides() == score.strides());
      p.score_max = static_cast<const float*>(ptr(mx));
    }
    require(u.Hkv > 0 && p.H % u.Hkv == 0 && p.Kb - p.Pb == p.Qb);
    u.B = p.B, u.G = p.H / u.Hkv, u.Qin = p.Qb, u.Kb = p.Kb, u.Pb = p.Pb;
    const at::Tensor* given[4];
    for (const at::Tensor*& t : given) t = a.optional();
    at::Tensor out[4];
    for (int i = 0; i < 4; ++i) {
      if (given[0]) {
        require(given[i] != nullptr && given[i]->dim() > 0 && given[i]->scalar_type() == at::kInt);
        out[i] = *given[i];
      } else if (i == 0) {
        out[i] = at::empty({p.B, u.Hkv, p.Pb > 0 ? p.Pb : 1}, score.options().dtype(at::kInt));
      } else {
        out[i] = at::empty({p.B, u.Hkv}, score.options().dtype(at::kInt));
      }
    }
    u.block_idx = static_cast<int32_t*>(ptr(out[0])), u.idx_stride = out[0].size(-1);
    u.counts = static_cast<int32_t*>(ptr(out[1]));
    u.cache_seqlens = static_cast<int32_t*>(ptr(out[2]));
    u.pages_per_row = static_cast<int32_t*>(ptr(out[3]));
    size_t need = 0;
    require(is_int32(scratch) && lib.scratch_bytes(p.B, p.H, u.Hkv, p.Qb, p.Kb, &need) == CA_OK && scratch.nbytes() >= need);
    PyObject* first_gate = nullptr;
    ca_gate_score_params g = {};
    int write_scores = 0;
    try {
      first_gate = a.next();
    } catch (const NotPlain&) {
    }
    if (first_gate) {
      require(THPVariable_CheckExact(first_gate));
      const at::Tensor& q = THPVariable_Unpack(first_gate);
      const at::Tensor& k = a.tensor();
      require(q.is_cuda() && q.dim() == 4 && k.dim() == 4 && q.stride(3) == 1 && k.stride(3) == 1);
      g.B = q.size(0), g.Qb = q.size(1), g.Hq = q.size(2), g.C = q.size(3);
      g.Kb = k.size(1), g.Hk = k.size(2), g.Pb = p.Pb;
      require(g.B == p.B && g.Hq == p.H && g.Qb == p.Qb && g.Kb == p.Kb && p.score_dtype == CA_DTYPE_F32 && score.is_contiguous());
      g.q = ptr(q), g.q_stride_b = q.stride(0), g.q_stride_blk = q.stride(1), g.q_stride_h = q.stride(2), g.q_dtype = dtype_of(q);
      g.k = ptr(k), g.k_stride_b = k.stride(0), g.k_stride_blk = k.stride(1), g.k_stride_h = k.stride(2), g.k_dtype = dtype_of(k);
      g.out = static_cast<float*>(ptr(score));
      g.scale = static_cast<float>(a.number()), g.masked_value = static_cast<float>(a.number());
      write_scores = a.i32();
    }
    a.done();
    if (first_gate) {
      enqueue("ca_gate_score_select",
              [&] { return lib.gate_score_select(&g, &p, &u, ptr(scratch), scratch.nbytes(), write_scores, stream); });
    } else {
      enqueue("ca_select_union_table", [&] { return lib.select_union_table(&p, &u, ptr(scratch), scratch.nbytes(), stream); });
    }
    PyObject* res = PyTuple_New(4);
    if (res) {
      for (int i = 0; i < 4; ++i) PyTuple_SET_ITEM(res, i, THPVariable_Wrap(out[i]));
    }
    return res;
  });
}

#define CA_TEXT_OF(x) #x
#define CA_TEXT(x) CA_TEXT_OF(x)
PyObject* header_hash(PyObject*, PyObject* const*, Py_ssize_t) { return PyBytes_FromString(CA_TEXT(CA_HEADER_HASH)); }

#define CALL(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {CALL(header_hash), CALL(bind), CALL(attn_compact), CALL(rope_append), CALL(gate_prepare), CALL(select_union_table),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&module); }
