// Host path of the tensor-level entry points: torch tensors in, one C-ABI call out.
//
// A small attention call takes the GPU a few microseconds, so what bounds it is the work on the
// host: reading shapes and strides, checking them, filling the argument record, allocating the
// output, finding the current stream. In Python (ctypes records, one attribute at a time) that
// took 13-20 us per launch; here it takes about 1 us plus the allocation and the launch itself.
// The checks and their messages are those of the Python functions in functional.py that call in
// here; errors are raised as the same Python exception types.
//
// `Call` is a call of a compiled graph bound to one set of sizes; `Dispatcher` is the callable a
// compiled graph becomes: it compares the sizes and scalar arguments with those it has seen (the
// plan cache of CompiledAttention, looked up without building a key) and launches.
//
// The kernels' entry points come in as addresses (bind()), so that the module serves the normal
// and the range-checking build of the library alike.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cstring>
#include <string>
#include <vector>

#include "../../include/lf_sm100.h"

namespace {

using at::Tensor;

// ---------------------------------------------------------------------------------------
// Errors
// ---------------------------------------------------------------------------------------
struct Raise {  // a Python exception to set
  PyObject* type;
  std::string text;
};
struct PyErrorSet {};  // a Python exception is already set

[[noreturn]] void value_error(const std::string& s) { throw Raise{PyExc_ValueError, s}; }
[[noreturn]] void type_error(const std::string& s) { throw Raise{PyExc_TypeError, s}; }

std::string shape_text(at::IntArrayRef s) {
  std::string r = "(";
  for (size_t i = 0; i < s.size(); ++i) r += (i ? ", " : "") + std::to_string(s[i]);
  return r + (s.size() == 1 ? ",)" : ")");
}

template <class F>
PyObject* guarded(F f) {
  try {
    return f();
  } catch (const Raise& e) {
    PyErr_SetString(e.type, e.text.c_str());
  } catch (const PyErrorSet&) {
  } catch (...) {  // (out of memory, an index out of range, ... as the types that torch raises)
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}

// ---------------------------------------------------------------------------------------
// The bound library
// ---------------------------------------------------------------------------------------
struct Lib {
  int (*prefill)(const LfPrefillArgs*, void*) = nullptr;
  int (*prefill_row_bias)(const LfPrefillArgs*, const LfRowBias*, void*) = nullptr;
  int (*q_tile)(const LfPrefillArgs*) = nullptr;
  int (*decode)(const LfDecodeArgs*, void*) = nullptr;
  int (*decode_paged)(const LfDecodeArgs*, void*) = nullptr;
  int (*auto_splits)(int32_t, int32_t, int32_t, int32_t, int32_t, int32_t) = nullptr;
  size_t (*workspace_bytes)(int32_t, int32_t, int32_t, int32_t, int32_t) = nullptr;
  int (*launches)(const LfDecodeArgs*, int32_t) = nullptr;
  int (*kv_append)(const LfKvAppendArgs*, void*) = nullptr;
  int (*add)(const void*, const void*, void*, int32_t, int32_t, int32_t, int32_t, const int64_t*,
             const int64_t*, const int64_t*, void*) = nullptr;
  PyObject* check = nullptr;  // _native.check(rc, what): raises LfError
} lib;

void check_rc(int rc, const char* what) {
  if (rc == LF_OK) return;
  PyObject* r = PyObject_CallFunction(lib.check, "is", rc, what);
  Py_XDECREF(r);
  if (r) PyErr_Format(PyExc_RuntimeError, "%s failed: %d", what, rc);
  throw PyErrorSet{};
}

struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// Runs `f(stream)` with the tensors' device current, without the GIL (a launch may block when the
// queue of the stream is full).
template <class F>
int launch(const c10::Device& dev, F f) {
  const c10::cuda::CUDAGuard guard(dev);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const NoGil no_gil;
  return f(stream);
}

// ---------------------------------------------------------------------------------------
// Arguments
// ---------------------------------------------------------------------------------------
const Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) type_error(std::string(name) + " must be a tensor");
  return THPVariable_Unpack(o);
}
const Tensor* optional_tensor(PyObject* o, const char* name) {
  return o == Py_None ? nullptr : &tensor_arg(o, name);
}
long long int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    PyObject* n = PyNumber_Long(o);  // (accepts what int() accepts, as the Python code did)
    if (!n) throw PyErrorSet{};
    const long long w = PyLong_AsLongLong(n);
    Py_DECREF(n);
    if (w == -1 && PyErr_Occurred()) throw PyErrorSet{};
    return w;
  }
  return v;
}
int splits_arg(PyObject* o) {  // (None: the library chooses, like 0)
  return o == Py_None ? 0 : static_cast<int>(int_arg(o));
}
double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyErrorSet{};
  return v;
}

struct Mods {
  int n = 0;
  int op[LF_MAX_MODS];
  float arg[LF_MAX_MODS];
};

Mods mods_arg(PyObject* o) {
  static PyObject* s_op = PyUnicode_InternFromString("op");
  static PyObject* s_arg = PyUnicode_InternFromString("arg");
  Mods m;
  PyObject* seq = PySequence_Fast(o, "mods must be a sequence of score mods");
  if (!seq) throw PyErrorSet{};
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  try {
    if (n > LF_MAX_MODS)
      value_error("at most " + std::to_string(LF_MAX_MODS) + " score-mod ops");
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* it = PySequence_Fast_GET_ITEM(seq, i);
      PyObject* op = PyObject_GetAttr(it, s_op);
      PyObject* arg = op ? PyObject_GetAttr(it, s_arg) : nullptr;
      if (!arg) {
        Py_XDECREF(op);
        throw PyErrorSet{};
      }
      const long v = PyLong_AsLong(op);
      const double a = PyFloat_AsDouble(arg);
      Py_DECREF(op);
      Py_DECREF(arg);
      if (PyErr_Occurred()) throw PyErrorSet{};
      m.op[i] = static_cast<int>(v);
      m.arg[i] = static_cast<float>(a);
    }
  } catch (...) {
    Py_DECREF(seq);
    throw;
  }
  Py_DECREF(seq);
  m.n = static_cast<int>(n);
  return m;
}

template <class Args>
void fill_mods(Args& a, double scale, const Mods& m) {
  a.scale = static_cast<float>(scale);
  a.n_mod = m.n;
  for (int i = 0; i < m.n; ++i) {
    a.mod_op[i] = m.op[i];
    a.mod_arg[i] = m.arg[i];
  }
}

void require_cuda(const Tensor& t, const c10::Device& dev) {
  if (!t.is_cuda())
    throw Raise{PyExc_RuntimeError,
                "loopfuse_b200 kernels need CUDA tensors on an sm_100 GPU; there is no CPU path"};
  if (t.device() != dev) value_error("all tensors must live on the same device");
}

void check_bf16(const Tensor& t, const char* name) {
  if (t.scalar_type() != at::kBFloat16) {
    const at::ScalarType st = t.scalar_type();
    type_error(std::string(name) + " must be bfloat16, got torch." +
               (st == at::kFloat ? "float32" : st == at::kHalf ? "float16" : c10::toString(st)));
  }
  if (t.dim() == 0 || t.stride(-1) != 1)
    value_error(std::string(name) + " must have a contiguous last dim");
}

Tensor new_bf16(at::IntArrayRef sizes, const c10::Device& dev) {
  return at::empty(sizes, at::TensorOptions().dtype(at::kBFloat16).device(dev));
}

void strides3(int64_t* dst, const Tensor& t) {
  for (int i = 0; i < 3; ++i) dst[i] = t.stride(i);
}

int32_t i32(int64_t v) { return static_cast<int32_t>(v); }

// A pool [pages, page_size, Hkv, D]; [pages, Hkv, D] means one token per page.
Tensor pool_view(const Tensor& t, const char* name) {
  check_bf16(t, name);
  if (t.dim() == 3) return t.unsqueeze(1);
  if (t.dim() != 4)
    value_error(std::string(name) + " must be [pages, page_size, Hkv, D] or [pages, Hkv, D]");
  return t;
}

Tensor table_i32(const Tensor& t) {
  if (t.dim() != 2) value_error("block_table must be [batch, blocks]");
  Tensor r = t.scalar_type() == at::kInt ? t : t.to(at::kInt);
  return r.stride(1) == 1 ? r : r.contiguous();
}

int32_t* status_ptr(const Tensor* st) {
  return st ? static_cast<int32_t*>(st->data_ptr()) : nullptr;
}

// ---------------------------------------------------------------------------------------
// Prefill
// ---------------------------------------------------------------------------------------
struct PrefillOptions {
  double scale = 1.0;
  Mods mods;
  int mask_kind = 0, window = 0, causal_offset = 0, kv_tile = 0, sm_margin = 0;
  int64_t seq_len = -1;  // -1: what k / v hold
  int bias_pos = -1;     // -1: after the whole chain
};

struct PrefillTensors {
  const Tensor *q, *k, *v;
  const Tensor *status = nullptr, *dbg = nullptr, *k_table = nullptr, *v_table = nullptr,
               *score_bias = nullptr, *q_pe = nullptr, *k_pe = nullptr;
};

// Argument record of lf_prefill_bf16. `out` is allocated when it is not defined; tensors that had
// to be converted for the call are appended to `keep`.
void fill_prefill(LfPrefillArgs& a, const PrefillTensors& t, const PrefillOptions& o, Tensor& out,
                  std::vector<Tensor>& keep) {
  const Tensor& q = *t.q;
  const c10::Device dev = q.device();
  require_cuda(q, dev);
  require_cuda(*t.k, dev);
  require_cuda(*t.v, dev);
  check_bf16(q, "q");
  if (q.dim() != 4) value_error("q must be 4-D");
  const int64_t B = q.size(0), Hq = q.size(1), Sq = q.size(2), D = q.size(3);

  // A paged operand is a pool plus its block table; a dense one is [B, Hkv, Skv, D].
  struct Operand {
    Tensor t, table;
    int64_t heads, tokens;
  } kv[2];
  for (int i = 0; i < 2; ++i) {
    const std::string name = i ? "v" : "k";
    const Tensor& ten = i ? *t.v : *t.k;
    const Tensor* table = i ? t.v_table : t.k_table;
    Operand& x = kv[i];
    if (!table) {
      check_bf16(ten, name.c_str());
      if (ten.dim() != 4 || ten.size(0) != B || ten.size(3) != D)
        value_error("shape mismatch: q " + shape_text(q.sizes()) + " " + name + " " +
                    shape_text(ten.sizes()));
      x = {ten, Tensor(), ten.size(1), ten.size(2)};
    } else {
      x.t = pool_view(ten, (name + " pool").c_str());
      x.table = table_i32(*table);
      if (!x.table.is_cuda() || x.table.size(0) != B || x.t.size(3) != D)
        value_error(name + ": pool " + shape_text(x.t.sizes()) + " / block table " +
                    shape_text(x.table.sizes()) + " do not fit q " + shape_text(q.sizes()));
      x.heads = x.t.size(2);
      x.tokens = x.table.size(1) * x.t.size(1);
    }
  }
  const Operand &k = kv[0], &v = kv[1];
  const bool kp = k.table.defined(), vp = v.table.defined();
  if (k.heads != v.heads) value_error("k and v must have the same number of kv heads");
  if (!kp && !vp && k.tokens != v.tokens) value_error("k and v must have the same length");
  const int64_t held = std::min(k.tokens, v.tokens);
  const int64_t Skv = o.seq_len >= 0 ? o.seq_len : held;
  if (Skv > held || Skv <= 0) value_error("seq_len exceeds what k / v hold");
  if (k.heads == 0 || Hq % k.heads) value_error("Hq must be a multiple of Hkv");
  if (!out.defined()) {
    out = new_bf16({B, Hq, Sq, D}, dev);
  } else {
    if (!out.is_cuda()) require_cuda(out, dev);
    check_bf16(out, "out");
  }

  std::memset(&a, 0, sizeof(a));
  a.q = q.data_ptr();
  a.k = k.t.data_ptr();
  a.v = v.t.data_ptr();
  a.out = out.data_ptr();
  a.B = i32(B), a.Hq = i32(Hq), a.Hkv = i32(k.heads), a.Sq = i32(Sq), a.Skv = i32(Skv);
  a.D = i32(D);
  strides3(a.q_stride, q);
  strides3(a.k_stride, k.t);
  strides3(a.v_stride, v.t);
  strides3(a.o_stride, out);
  if (kp || vp) {
    if (kp && vp && (k.t.size(0) != v.t.size(0) || k.t.size(1) != v.t.size(1)))
      value_error("paged k and v must share the page geometry");
    Tensor kt = k.table, vt = v.table;
    if (kp && vp && kt.stride(0) != vt.stride(0)) {
      kt = kt.contiguous();
      vt = vt.contiguous();
    }
    if (kp) a.k_block_table = static_cast<const int32_t*>(kt.data_ptr()), keep.push_back(kt);
    if (vp) a.v_block_table = static_cast<const int32_t*>(vt.data_ptr()), keep.push_back(vt);
    a.bt_stride = (kp ? kt : vt).stride(0);
    const Tensor& pool = kp ? k.t : v.t;
    a.page_size = i32(pool.size(1));
    a.n_pages = i32(pool.size(0));
  }
  fill_mods(a, o.scale, o.mods);
  a.mask_kind = o.mask_kind;
  a.window = o.window;
  a.causal_offset = o.causal_offset;
  a.status = status_ptr(t.status);
  a.kv_tile = o.kv_tile;
  a.sm_margin = o.sm_margin;
  if (t.dbg) {
    const int q_tile = lib.q_tile(&a);
    if (q_tile < 0) check_rc(q_tile, "lf_prefill_q_tile");
    const int64_t need = B * Hq * ((Sq + q_tile - 1) / q_tile) * 2;
    if (t.dbg->scalar_type() != at::kInt || t.dbg->numel() < need || !t.dbg->is_cuda())
      value_error("dbg_ranges must be a CUDA int32 tensor with >= " + std::to_string(need) +
                  " elements");
    a.dbg_ranges = static_cast<int32_t*>(t.dbg->data_ptr());
  }
  if (t.score_bias) {
    const Tensor& sb = *t.score_bias;
    require_cuda(sb, sb.device());
    check_bf16(sb, "score_bias");
    if (sb.dim() != 4 || sb.size(0) != B || sb.size(1) != Hq || sb.size(2) != Sq ||
        sb.size(3) != Skv)
      value_error("score_bias must be [B, Hq, Sq, Skv] = " + shape_text({B, Hq, Sq, Skv}) +
                  ", got " + shape_text(sb.sizes()));
    a.score_bias = sb.data_ptr();
    strides3(a.bias_stride, sb);
    a.bias_pos = o.bias_pos < 0 ? a.n_mod : o.bias_pos;
  }
  if (!t.q_pe != !t.k_pe) value_error("q_pe and k_pe go together");
  if (t.q_pe) {
    const Tensor &qp = *t.q_pe, &kpe = *t.k_pe;
    require_cuda(qp, qp.device());
    require_cuda(kpe, qp.device());
    check_bf16(qp, "q_pe");
    check_bf16(kpe, "k_pe");
    if (qp.dim() != 4 || kpe.dim() != 4 || qp.size(0) != B || qp.size(1) != Hq ||
        qp.size(2) != Sq || kpe.size(0) != B || kpe.size(1) != k.heads || kpe.size(2) != Skv ||
        qp.size(3) != kpe.size(3))
      value_error("q_pe " + shape_text(qp.sizes()) + " / k_pe " + shape_text(kpe.sizes()) +
                  " do not fit q " + shape_text(q.sizes()) + " and the keys");
    a.q_pe = qp.data_ptr();
    a.k_pe = kpe.data_ptr();
    a.D_pe = i32(qp.size(3));
    strides3(a.qpe_stride, qp);
    strides3(a.kpe_stride, kpe);
  }
}

Tensor run_prefill(const PrefillTensors& t, const PrefillOptions& o, Tensor out) {
  LfPrefillArgs a;
  std::vector<Tensor> keep;
  fill_prefill(a, t, o, out, keep);
  check_rc(launch(t.q->device(), [&](void* st) { return lib.prefill(&a, st); }),
           "lf_prefill_bf16");
  return out;
}

// ---------------------------------------------------------------------------------------
// Elementwise add, cache append
// ---------------------------------------------------------------------------------------
void check_add(const Tensor& x, at::IntArrayRef x_sizes, const Tensor& y) {
  require_cuda(x, x.device());
  require_cuda(y, x.device());
  check_bf16(x, "a");
  check_bf16(y, "b");
  if (x_sizes.size() != 4 || x_sizes != y.sizes())
    value_error("add_bf16 takes two 4-D tensors of one shape, got " + shape_text(x_sizes) +
                " and " + shape_text(y.sizes()));
}

Tensor run_add(const Tensor& x, const Tensor& y, Tensor out) {
  const c10::Device dev = x.device();
  check_add(x, x.sizes(), y);
  if (!out.defined()) {
    out = new_bf16(x.sizes(), dev);
  } else {
    require_cuda(out, out.device());
    check_bf16(out, "out");
    if (out.sizes() != x.sizes()) value_error("out must have the operands' shape");
  }
  int64_t xs[3], ys[3], os[3];
  strides3(xs, x);
  strides3(ys, y);
  strides3(os, out);
  check_rc(launch(dev,
                  [&](void* st) {
                    return lib.add(x.data_ptr(), y.data_ptr(), out.data_ptr(), i32(x.size(0)),
                                   i32(x.size(1)), i32(x.size(2)), i32(x.size(3)), xs, ys, os, st);
                  }),
           "lf_add_bf16");
  return out;
}

// A prefill with a query and / or output bias. In one launch where the library can (a score bias in front
// of the mask); otherwise the query bias is added first and the output bias in place, by kernels of their
// own. The same bits: each is one bf16 rounding, as in the eager graph.
// (Out of line: its argument records would be part of every call's frame.)
[[gnu::noinline]] Tensor run_row_biased(const PrefillTensors& p, const PrefillOptions& o,
                                        const Tensor* q_bias, const Tensor* out_bias, Tensor out) {
  // (What neither way takes is refused before anything is launched.)
  for (const Tensor* bias : {q_bias, out_bias}) {
    if (!bias) continue;
    check_add(*p.q, p.q->sizes(), *bias);
    bool aligned = reinterpret_cast<uintptr_t>(bias->data_ptr()) % 16 == 0;
    for (int i = 0; i < 3; ++i) aligned = aligned && bias->stride(i) % 8 == 0;
    if (!aligned) check_rc(LF_ERR_ALIGNMENT, "lf_add_bf16");
  }
  LfPrefillArgs a;
  std::vector<Tensor> keep;
  fill_prefill(a, p, o, out, keep);
  const c10::Device dev = p.q->device();
  if (p.score_bias) {
    LfRowBias rows;
    std::memset(&rows, 0, sizeof(rows));
    if (q_bias) rows.q_bias = q_bias->data_ptr(), strides3(rows.q_bias_stride, *q_bias);
    if (out_bias) rows.out_bias = out_bias->data_ptr(), strides3(rows.out_bias_stride, *out_bias);
    const int rc = launch(dev, [&](void* st) { return lib.prefill_row_bias(&a, &rows, st); });
    if (rc != LF_ERR_UNSUPPORTED && rc != LF_ERR_ALIGNMENT) {
      check_rc(rc, "lf_prefill_row_bias_bf16");
      return out;
    }
  }
  Tensor biased;
  if (q_bias) {
    biased = run_add(*p.q, *q_bias, Tensor());
    a.q = biased.data_ptr();
    strides3(a.q_stride, biased);
  }
  check_rc(launch(dev, [&](void* st) { return lib.prefill(&a, st); }), "lf_prefill_bf16");
  if (out_bias) run_add(out, *out_bias, out);
  return out;
}

void run_kv_append(const Tensor& kn, const Tensor& vn, const Tensor& k_pool, const Tensor& v_pool,
                   const Tensor& table, const Tensor* table_v, const Tensor* seq_pos,
                   int64_t start_pos, const Tensor* status) {
  const c10::Device dev = kn.device();
  for (const Tensor* t : {&kn, &vn, &k_pool, &v_pool, &table}) require_cuda(*t, dev);
  check_bf16(kn, "k_new");
  if (kn.dim() != 4) value_error("k_new must be [B, Hkv, T, D]");
  check_bf16(vn, "v_new");
  if (vn.dim() != 4) value_error("v_new must be [B, Hkv, T, D]");
  const Tensor kp = pool_view(k_pool, "k_pool"), vp = pool_view(v_pool, "v_pool");
  const int64_t B = kn.size(0), Hkv = kn.size(1), D = kn.size(3);
  if (vn.sizes() != kn.sizes()) value_error("k_new and v_new must have the same shape");
  if (kp.size(2) != Hkv || kp.size(3) != D || vp.sizes() != kp.sizes())
    value_error("pool shape mismatch: new " + shape_text(kn.sizes()) + " pool " +
                shape_text(kp.sizes()));
  Tensor bt = table_i32(table), btv = table_v ? table_i32(*table_v) : Tensor();
  if (bt.size(0) != B) value_error("block_table batch mismatch");
  if (btv.defined() && (btv.sizes() != bt.sizes() || btv.stride(0) != bt.stride(0))) {
    btv = btv.contiguous();
    bt = bt.contiguous();
  }
  Tensor pos;
  if (seq_pos) {
    if (seq_pos->scalar_type() != at::kInt || seq_pos->dim() != 1 || seq_pos->size(0) != B ||
        !seq_pos->is_cuda())
      value_error("seq_pos must be a CUDA int32 tensor of shape [B]");
    pos = seq_pos->contiguous();
  }
  LfKvAppendArgs a;
  std::memset(&a, 0, sizeof(a));
  a.k_new = kn.data_ptr();
  a.v_new = vn.data_ptr();
  a.k_pool = kp.data_ptr();
  a.v_pool = vp.data_ptr();
  a.block_table = static_cast<const int32_t*>(bt.data_ptr());
  a.block_table_v = btv.defined() ? static_cast<const int32_t*>(btv.data_ptr()) : nullptr;
  a.seq_pos = pos.defined() ? static_cast<const int32_t*>(pos.data_ptr()) : nullptr;
  a.start_pos = i32(start_pos);
  a.B = i32(B), a.Hkv = i32(Hkv), a.T = i32(kn.size(2)), a.D = i32(D);
  strides3(a.kn_stride, kn);
  strides3(a.vn_stride, vn);
  strides3(a.kp_stride, kp);
  strides3(a.vp_stride, vp);
  a.bt_stride = bt.stride(0);
  a.bt_blocks = i32(bt.size(1));
  a.page_size = i32(kp.size(1));
  a.n_pages = i32(kp.size(0));
  a.status = status_ptr(status);
  check_rc(launch(dev, [&](void* st) { return lib.kv_append(&a, st); }), "lf_kv_append_bf16");
}

// ---------------------------------------------------------------------------------------
// Decode
// ---------------------------------------------------------------------------------------
struct DecodeQuery {  // q as [B, Hkv, G, D] with element strides of the first three
  int64_t B, Hkv, G, D;
  int64_t stride[3];
};

DecodeQuery query_of(const Tensor& q) {
  DecodeQuery d{q.size(0), q.size(1), q.size(2), q.size(3), {}};
  strides3(d.stride, q);
  return d;
}

struct Paged {
  const Tensor *table, *table_v;
  int64_t seq_len;  // -1: all the table covers
};

struct DecodeOptions {
  double scale = 1.0;
  Mods mods;
  int splits = 0;
};

// Scratch of `nbytes` from a DecodeWorkspace (its buffer is reused while it is large enough, on the
// stream that it was made on). The caller holds the tensor until the launch is queued: the object may
// let go of it meanwhile.
Tensor workspace_tensor(PyObject* ws, size_t nbytes, const Tensor& like, const void* stream) {
  static PyObject* s_buf = PyUnicode_InternFromString("_buf");
  static PyObject* s_stream = PyUnicode_InternFromString("_stream");
  PyObject* buf = PyObject_GetAttr(ws, s_buf);
  PyObject* on = buf ? PyObject_GetAttr(ws, s_stream) : nullptr;
  Tensor t;
  if (on && THPVariable_Check(buf) && PyLong_Check(on) && PyLong_AsVoidPtr(on) == stream) {
    t = THPVariable_Unpack(buf);
    if (static_cast<size_t>(t.numel()) < nbytes || t.device() != like.device()) t = Tensor();
  }
  Py_XDECREF(buf);
  Py_XDECREF(on);
  PyErr_Clear();  // (an object with a get() of its own need not have these)
  if (t.defined()) return t;
  PyObject* like_obj = THPVariable_Wrap(like);
  PyObject* dev = like_obj ? PyObject_GetAttrString(like_obj, "device") : nullptr;
  Py_XDECREF(like_obj);
  if (!dev) throw PyErrorSet{};
  PyObject* got = PyObject_CallMethod(ws, "get", "nO", static_cast<Py_ssize_t>(nbytes), dev);
  Py_DECREF(dev);
  if (!got) throw PyErrorSet{};
  if (THPVariable_Check(got)) t = THPVariable_Unpack(got);
  Py_DECREF(got);
  if (!t.defined()) type_error("workspace.get() must return a tensor");
  return t;
}

// Dense (`paged` null) or paged decode of query `dq`; `out` has the strides `ostride` in the
// [B, Hkv, G, D] view.
void run_decode(const Tensor& q, const DecodeQuery& dq, const Tensor& k_in, const Tensor& v_in,
                const Paged* paged, const DecodeOptions& o, PyObject* workspace,
                const Tensor* status, const Tensor& out, const int64_t* ostride) {
  const c10::Device dev = q.device();
  LfDecodeArgs a;
  std::memset(&a, 0, sizeof(a));
  Tensor k = k_in, v = v_in, bt, btv;
  int64_t Skv = 0, page = 0;
  if (!paged) {
    if (k.size(0) != dq.B || k.size(1) != dq.Hkv || k.size(3) != dq.D || v.sizes() != k.sizes())
      value_error("shape mismatch: q " + shape_text({dq.B, dq.Hkv, dq.G, dq.D}) + " k " +
                  shape_text(k.sizes()) + " v " + shape_text(v.sizes()));
    Skv = k.size(2);
  } else {
    k = pool_view(k_in, "k_pool");
    v = pool_view(v_in, "v_pool");
    page = k.size(1);
    if (k.size(2) != dq.Hkv || k.size(3) != dq.D || v.sizes() != k.sizes())
      value_error("pool shape mismatch: q " + shape_text({dq.B, dq.Hkv, dq.G, dq.D}) + " pool " +
                  shape_text(k.sizes()));
    bt = table_i32(*paged->table);
    if (paged->table_v) btv = table_i32(*paged->table_v);
    if (bt.size(0) != dq.B) value_error("block_table batch mismatch");
    Skv = paged->seq_len >= 0 ? paged->seq_len : bt.size(1) * page;
    if (Skv > bt.size(1) * page) value_error("seq_len exceeds the block table");
    if (btv.defined() && (btv.sizes() != bt.sizes() || btv.stride(0) != bt.stride(0))) {
      btv = btv.contiguous();
      bt = bt.contiguous();
    }
    a.block_table = static_cast<const int32_t*>(bt.data_ptr());
    a.block_table_v = btv.defined() ? static_cast<const int32_t*>(btv.data_ptr()) : nullptr;
    a.bt_stride = bt.stride(0);
    a.page_size = i32(page);
    a.n_pages = i32(k.size(0));
  }
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.out = out.data_ptr();
  a.B = i32(dq.B), a.Hkv = i32(dq.Hkv), a.G = i32(dq.G), a.Skv = i32(Skv), a.D = i32(dq.D);
  for (int i = 0; i < 3; ++i) {
    a.q_stride[i] = dq.stride[i];
    a.o_stride[i] = ostride[i];
  }
  strides3(a.k_stride, k);
  strides3(a.v_stride, v);
  fill_mods(a, o.scale, o.mods);
  a.status = status_ptr(status);
  const c10::cuda::CUDAGuard guard(dev);
  a.splits = o.splits ? o.splits : lib.auto_splits(a.B, a.Hkv, a.G, a.Skv, a.D, a.page_size);
  a.workspace_bytes = lib.workspace_bytes(a.B, a.Hkv, a.G, a.D, a.splits);
  // Splits that merge in their cluster leave the workspace alone: the library wants one, any address
  // will do. Otherwise, without a workspace of the caller's, the partials are an allocation of this
  // call on its stream. (Into one that calls shared, a call on another stream or thread could write
  // between the two kernels of this one, and a captured graph after it has been replaced.)
  Tensor held;
  c10::DataPtr own;
  if (a.workspace_bytes) {
    a.workspace = out.data_ptr();
    if (lib.launches(&a, paged != nullptr) == 2) {
      if (workspace == Py_None) {
        own = c10::cuda::CUDACachingAllocator::get()->allocate(a.workspace_bytes);
        a.workspace = own.get();
      } else {
        held = workspace_tensor(workspace, a.workspace_bytes, q,
                                c10::cuda::getCurrentCUDAStream(dev.index()).stream());
        a.workspace = held.data_ptr();
      }
    }
  }
  check_rc(launch(dev,
                  [&](void* st) {
                    return paged ? lib.decode_paged(&a, st) : lib.decode(&a, st);
                  }),
           paged ? "lf_decode_paged_bf16" : "lf_decode_bf16");
}

// ---------------------------------------------------------------------------------------
// Python functions (positional arguments only; functional.py has the keyword forms)
// ---------------------------------------------------------------------------------------
void want_args(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) type_error("expected " + std::to_string(want) + " arguments");
}

Tensor out_arg(PyObject* o) { return o == Py_None ? Tensor() : tensor_arg(o, "out"); }

// q, k, v, out, status, dbg_ranges, k_block_table, v_block_table, score_bias, q_pe, k_pe,
// scale, mods, mask_kind, window, causal_offset, kv_tile, sm_margin, seq_len, bias_pos
constexpr Py_ssize_t kPrefillArgCount = 20;

void parse_prefill(PyObject* const* a, PrefillTensors& t, PrefillOptions& o, Tensor& out) {
  t.q = &tensor_arg(a[0], "q");
  t.k = &tensor_arg(a[1], "k");
  t.v = &tensor_arg(a[2], "v");
  out = out_arg(a[3]);
  t.status = optional_tensor(a[4], "status");
  t.dbg = optional_tensor(a[5], "dbg_ranges");
  t.k_table = optional_tensor(a[6], "k_block_table");
  t.v_table = optional_tensor(a[7], "v_block_table");
  t.score_bias = optional_tensor(a[8], "score_bias");
  t.q_pe = optional_tensor(a[9], "q_pe");
  t.k_pe = optional_tensor(a[10], "k_pe");
  o.scale = float_arg(a[11]);
  o.mods = mods_arg(a[12]);
  o.mask_kind = static_cast<int>(int_arg(a[13]));
  o.window = static_cast<int>(int_arg(a[14]));
  o.causal_offset = static_cast<int>(int_arg(a[15]));
  o.kv_tile = static_cast<int>(int_arg(a[16]));
  o.sm_margin = static_cast<int>(int_arg(a[17]));
  if (a[18] != Py_None) {
    o.seq_len = int_arg(a[18]);
    if (o.seq_len <= 0) value_error("seq_len exceeds what k / v hold");
  }
  if (a[19] != Py_None) {
    o.bias_pos = static_cast<int>(int_arg(a[19]));
    if (o.bias_pos < 0) o.bias_pos = 1 << 20;  // out of range: refused by the library
  }
}

PyObject* py_prefill(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, kPrefillArgCount + 2);
    PrefillTensors t;
    PrefillOptions o;
    Tensor out;
    parse_prefill(a, t, o, out);
    const Tensor* q_bias = optional_tensor(a[kPrefillArgCount], "q_bias");
    const Tensor* out_bias = optional_tensor(a[kPrefillArgCount + 1], "out_bias");
    if (q_bias || out_bias)
      return THPVariable_Wrap(run_row_biased(t, o, q_bias, out_bias, std::move(out)));
    return THPVariable_Wrap(run_prefill(t, o, std::move(out)));
  });
}

// The argument record alone, for a call that is launched again and again: (bytes, out, keep).
PyObject* py_prefill_record(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want_args(n, kPrefillArgCount);
    PrefillTensors t;
    PrefillOptions o;
    Tensor out;
    parse_prefill(a, t, o, out);
    LfPrefillArgs rec;
    std::vector<Tensor> keep;
    fill_prefill(rec, t, o, out, keep);
    PyObject* kept = PyList_New(0);
    for (const Tensor& x : keep) {
      PyObject* w = THPVariable_Wrap(x);
      PyList_Append(kept, w);
      Py_XDECREF(w);
    }
    PyObject* bytes = PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&rec), sizeof(rec));
    return Py_BuildValue("(NNN)", bytes, THPVariable_Wrap(out), kept);
  });
}

// q, k, v, out, workspace, status, scale, mods, splits
PyObject* py_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 9);
    const Tensor &q = tensor_arg(a[0], "q"), &k = tensor_arg(a[1], "k"),
                 &v = tensor_arg(a[2], "v");
    const c10::Device dev = q.device();
    const Tensor* ts[3] = {&q, &k, &v};
    const char* names[3] = {"q", "k", "v"};
    for (const Tensor* t : ts) require_cuda(*t, dev);
    for (int i = 0; i < 3; ++i) {
      check_bf16(*ts[i], names[i]);
      if (ts[i]->dim() != 4) value_error(std::string(names[i]) + " must be 4-D");
    }
    Tensor out = out_arg(a[3]);
    const Tensor* status = optional_tensor(a[5], "status");
    DecodeOptions o;
    o.scale = float_arg(a[6]);
    o.mods = mods_arg(a[7]);
    o.splits = splits_arg(a[8]);
    const DecodeQuery dq = query_of(q);
    if (!out.defined()) out = new_bf16(q.sizes(), dev);
    int64_t os[3];
    strides3(os, out);
    run_decode(q, dq, k, v, nullptr, o, a[4], status, out, os);
    return THPVariable_Wrap(out);
  });
}

// q, k_pool, v_pool, block_table, block_table_v, out, workspace, status, seq_len, scale, mods,
// splits
PyObject* py_paged_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 12);
    const Tensor &q = tensor_arg(a[0], "q"), &k = tensor_arg(a[1], "k_pool"),
                 &v = tensor_arg(a[2], "v_pool"), &bt = tensor_arg(a[3], "block_table");
    const c10::Device dev = q.device();
    for (const Tensor* t : {&q, &k, &v, &bt}) require_cuda(*t, dev);
    check_bf16(q, "q");
    if (q.dim() != 4) value_error("q must be 4-D");
    Paged pg{&bt, optional_tensor(a[4], "block_table_v"), -1};
    Tensor out = out_arg(a[5]);
    const Tensor* status = optional_tensor(a[7], "status");
    if (a[8] != Py_None) {
      pg.seq_len = int_arg(a[8]);
      if (pg.seq_len < 0) pg.seq_len = 0;  // refused by the library
    }
    DecodeOptions o;
    o.scale = float_arg(a[9]);
    o.mods = mods_arg(a[10]);
    o.splits = splits_arg(a[11]);
    const DecodeQuery dq = query_of(q);
    if (!out.defined()) out = new_bf16(q.sizes(), dev);
    int64_t os[3];
    strides3(os, out);
    run_decode(q, dq, k, v, &pg, o, a[6], status, out, os);
    return THPVariable_Wrap(out);
  });
}

// k_new, v_new, k_pool, v_pool, block_table, block_table_v, seq_pos, start_pos, status
PyObject* py_kv_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want_args(n, 9);
    run_kv_append(tensor_arg(a[0], "k_new"), tensor_arg(a[1], "v_new"),
                  tensor_arg(a[2], "k_pool"), tensor_arg(a[3], "v_pool"),
                  tensor_arg(a[4], "block_table"), optional_tensor(a[5], "block_table_v"),
                  optional_tensor(a[6], "seq_pos"), int_arg(a[7]),
                  optional_tensor(a[8], "status"));
    Py_RETURN_NONE;
  });
}

PyObject* py_add(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    want_args(n, 3);
    return THPVariable_Wrap(
        run_add(tensor_arg(a[0], "a"), tensor_arg(a[1], "b"), out_arg(a[2])));
  });
}

// ---------------------------------------------------------------------------------------
// Calls of a compiled graph
// ---------------------------------------------------------------------------------------
enum CallKind { kCallPrefill = 0, kCallDecode = 1, kCallPagedDecode = 2 };
// Positions of the operands among the graph's arguments, in this order; -1: none.
enum Operand { kQ, kK, kV, kKTable, kVTable, kQBias, kScoreBias, kOutBias, kQPe, kKPe, kOperands };

struct Call {
  PyObject_HEAD
  int kind;
  int at[kOperands];
  PrefillOptions prefill;
  DecodeOptions decode;
};

void call_dealloc(PyObject* self) { Py_TYPE(self)->tp_free(self); }

// kind, operand positions (a tuple of kOperands ints), scale, mods, mask_kind, window, bias_pos
PyObject* call_new(PyTypeObject* type, PyObject* args, PyObject*) {
  return guarded([&]() -> PyObject* {
    int kind, mask_kind, window, bias_pos;
    double scale;
    PyObject *at, *mods;
    if (!PyArg_ParseTuple(args, "iO!dOiii", &kind, &PyTuple_Type, &at, &scale, &mods, &mask_kind,
                          &window, &bias_pos))
      throw PyErrorSet{};
    if (PyTuple_GET_SIZE(at) != kOperands) type_error("operand positions: wrong count");
    int pos[kOperands];
    for (int i = 0; i < kOperands; ++i)
      pos[i] = static_cast<int>(int_arg(PyTuple_GET_ITEM(at, i)));
    const Mods m = mods_arg(mods);
    Call* c = reinterpret_cast<Call*>(type->tp_alloc(type, 0));
    if (!c) throw PyErrorSet{};
    c->kind = kind;
    std::memcpy(c->at, pos, sizeof(pos));
    c->prefill = PrefillOptions();
    c->prefill.scale = scale;
    c->prefill.mods = m;
    c->prefill.mask_kind = mask_kind;
    c->prefill.window = window;
    c->prefill.bias_pos = bias_pos;
    c->decode = DecodeOptions();
    c->decode.scale = scale;
    c->decode.mods = m;
    return reinterpret_cast<PyObject*>(c);
  });
}

// One pass of the graph on its arguments; returns the output tensor.
Tensor run_call(const Call& c, PyObject* const* args, Py_ssize_t n) {
  const Tensor* t[kOperands];
  for (int i = 0; i < kOperands; ++i) {
    if (c.at[i] >= n) type_error("too few arguments for the compiled graph");
    t[i] = c.at[i] < 0 ? nullptr : &tensor_arg(args[c.at[i]], "operand");
  }
  if (c.kind == kCallPrefill) {
    PrefillTensors p;
    p.q = t[kQ];
    p.k = t[kK];
    p.v = t[kV];
    p.k_table = t[kKTable];
    p.v_table = t[kVTable];
    p.score_bias = t[kScoreBias];
    p.q_pe = t[kQPe];
    p.k_pe = t[kKPe];
    if (t[kQBias] || t[kOutBias])
      return run_row_biased(p, c.prefill, t[kQBias], t[kOutBias], Tensor());
    return run_prefill(p, c.prefill, Tensor());
  }
  const Tensor &q = *t[kQ], &k = *t[kK], &v = *t[kV];
  const bool paged = c.kind == kCallPagedDecode;
  const c10::Device dev = q.device();
  for (const Tensor* x : {&q, &k, &v}) require_cuda(*x, dev);
  check_bf16(q, "q");
  if (q.dim() != 4) value_error("q must be 4-D");
  if (!paged) {
    check_bf16(k, "k");
    check_bf16(v, "v");
    if (k.dim() != 4 || v.dim() != 4) value_error("k and v must be 4-D");
  } else {
    require_cuda(*t[kKTable], dev);
  }
  Tensor out = new_bf16(q.sizes(), dev);
  // G query rows per kv head: either Sq rows of one head (the reference's [B, Hkv, g, D]
  // convention, tests/benchmark.py:438-443) or the g heads that repeat_interleave maps onto one kv
  // head, each with a single row.
  DecodeQuery dq = query_of(q);
  int64_t os[3];
  strides3(os, out);
  const int64_t heads = paged ? k.size(-2) : k.size(1);
  if (dq.G == 1 && dq.Hkv != heads && heads > 0) {
    const int64_t g = dq.Hkv / heads;
    dq.Hkv = heads;
    dq.G = g;
    dq.stride[2] = dq.stride[1];
    dq.stride[1] *= g;
    os[2] = os[1];
    os[1] *= g;
  }
  const bool two = paged && c.at[kVTable] != c.at[kKTable];
  Paged pg{t[kKTable], two ? t[kVTable] : nullptr, -1};
  run_decode(q, dq, k, v, paged ? &pg : nullptr, c.decode, Py_None, nullptr, out, os);
  return out;
}

PyTypeObject call_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// What a call's plan depends on: the sizes of the tensors and the values of everything else, 0-dim
// tensors among them (a float argument or closure variable reaches the graph as one).
struct Seen {
  std::vector<int64_t> key;
  Call* call;
};

struct Dispatcher {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  PyObject* bind;
  std::vector<Seen>* seen;
};

constexpr size_t kMaxSeen = 64;

// Value of a 0-dim tensor. One that lives on the GPU is waited for: the launch takes it as a number.
double scalar_value(const Tensor& t) {
  if (t.is_cpu() && t.scalar_type() == at::kDouble) return *t.const_data_ptr<double>();
  if (t.is_cpu() && t.scalar_type() == at::kFloat) return *t.const_data_ptr<float>();
  const NoGil no_gil;
  return t.item().toDouble();
}

// Key of the arguments into `key` (at most `cap` words); -1: not representable. Each argument is
// preceded by a word that tells tensors from scalars, so keys of different kinds never match.
int make_key(PyObject* const* args, Py_ssize_t n, int64_t* key, int cap) {
  int w = 0;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* o = args[i];
    if (THPVariable_Check(o)) {
      const Tensor& t = THPVariable_Unpack(o);
      const auto s = t.sizes();
      if (w + 2 + static_cast<int>(s.size()) > cap) return -1;
      key[w++] = -1 - static_cast<int64_t>(s.size());
      for (int64_t x : s) key[w++] = x;
      if (s.empty()) {
        const double d = scalar_value(t);
        std::memcpy(&key[w++], &d, 8);
      }
    } else if (PyLong_CheckExact(o)) {
      int over = 0;
      const long long v = PyLong_AsLongLongAndOverflow(o, &over);
      if (over || w + 2 > cap) return -1;
      key[w++] = 1;
      key[w++] = v;
    } else if (PyFloat_CheckExact(o)) {
      const double d = PyFloat_AS_DOUBLE(o);
      if (w + 2 > cap) return -1;
      key[w++] = 2;
      std::memcpy(&key[w++], &d, 8);
    } else {
      return -1;
    }
  }
  return w;
}

PyObject* dispatcher_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Dispatcher* d = reinterpret_cast<Dispatcher*>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  return guarded([&]() -> PyObject* {
    if (kwnames && PyTuple_GET_SIZE(kwnames)) type_error("no keyword arguments");
    int64_t key[128];
    const int words = make_key(args, n, key, 128);
    Call* call = nullptr;
    if (words >= 0)
      for (const Seen& s : *d->seen)
        if (s.key.size() == static_cast<size_t>(words) &&
            std::memcmp(s.key.data(), key, words * sizeof(int64_t)) == 0) {
          call = s.call;
          break;
        }
    PyObject* fresh = nullptr;
    if (!call) {
      fresh = PyObject_Vectorcall(d->bind, args, n, nullptr);
      if (!fresh) throw PyErrorSet{};
      if (Py_TYPE(fresh) != &call_type) return fresh;  // the Python path has run the call itself
      call = reinterpret_cast<Call*>(fresh);
      if (words >= 0) {
        if (d->seen->size() >= kMaxSeen) {
          for (Seen& s : *d->seen) Py_DECREF(reinterpret_cast<PyObject*>(s.call));
          d->seen->clear();
        }
        Py_INCREF(fresh);
        d->seen->push_back({std::vector<int64_t>(key, key + words), call});
      }
    } else {
      Py_INCREF(reinterpret_cast<PyObject*>(call));  // (another thread may clear the list)
    }
    struct Release {
      PyObject* o;
      ~Release() { Py_DECREF(o); }
    } release{reinterpret_cast<PyObject*>(call)};
    PyObject* out = THPVariable_Wrap(run_call(*call, args, n));
    if (!out) throw PyErrorSet{};
    PyObject* tuple = PyTuple_New(1);
    PyTuple_SET_ITEM(tuple, 0, out);
    return tuple;
  });
}

PyObject* dispatcher_new(PyTypeObject* type, PyObject* args, PyObject*) {
  PyObject* bind;
  if (!PyArg_ParseTuple(args, "O", &bind)) return nullptr;
  Dispatcher* d = reinterpret_cast<Dispatcher*>(type->tp_alloc(type, 0));
  if (!d) return nullptr;
  d->vectorcall = dispatcher_call;
  Py_INCREF(bind);
  d->bind = bind;
  d->seen = new std::vector<Seen>();
  return reinterpret_cast<PyObject*>(d);
}

void dispatcher_dealloc(PyObject* self) {
  Dispatcher* d = reinterpret_cast<Dispatcher*>(self);
  for (Seen& s : *d->seen) Py_DECREF(reinterpret_cast<PyObject*>(s.call));
  delete d->seen;
  Py_XDECREF(d->bind);
  Py_TYPE(self)->tp_free(self);
}

PyTypeObject dispatcher_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// ---------------------------------------------------------------------------------------
// Module
// ---------------------------------------------------------------------------------------
// bind(addresses: dict name -> int, check): entry points of the loaded kernel library.
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    want_args(n, 2);
    auto get = [&](const char* name, auto& fn) {
      PyObject* v = PyDict_GetItemString(a[0], name);
      if (!v) value_error(std::string("bind: no address of ") + name);
      void* p = PyLong_AsVoidPtr(v);
      if (!p) throw PyErrorSet{};
      std::memcpy(&fn, &p, sizeof(p));
    };
    get("lf_prefill_bf16", lib.prefill);
    get("lf_prefill_row_bias_bf16", lib.prefill_row_bias);
    get("lf_prefill_q_tile", lib.q_tile);
    get("lf_decode_bf16", lib.decode);
    get("lf_decode_paged_bf16", lib.decode_paged);
    get("lf_decode_auto_splits", lib.auto_splits);
    get("lf_decode_workspace_bytes", lib.workspace_bytes);
    get("lf_decode_launches", lib.launches);
    get("lf_kv_append_bf16", lib.kv_append);
    get("lf_add_bf16", lib.add);
    Py_INCREF(a[1]);
    Py_XSETREF(lib.check, a[1]);
    Py_RETURN_NONE;
  });
}

#define LF_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef methods[] = {
    {"bind", LF_FAST(py_bind), "entry points of the kernel library"},
    {"prefill", LF_FAST(py_prefill), "launch lf_prefill_bf16"},
    {"prefill_record", LF_FAST(py_prefill_record), "argument record of lf_prefill_bf16"},
    {"decode", LF_FAST(py_decode), "launch lf_decode_bf16"},
    {"paged_decode", LF_FAST(py_paged_decode), "launch lf_decode_paged_bf16"},
    {"kv_append", LF_FAST(py_kv_append), "launch lf_kv_append_bf16"},
    {"add", LF_FAST(py_add), "launch lf_add_bf16"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host",
                          "native host path of loopfuse_b200.functional", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  call_type.tp_name = "loopfuse_b200._host.Call";
  call_type.tp_basicsize = sizeof(Call);
  call_type.tp_flags = Py_TPFLAGS_DEFAULT;
  call_type.tp_new = call_new;
  call_type.tp_dealloc = call_dealloc;
  dispatcher_type.tp_name = "loopfuse_b200._host.Dispatcher";
  dispatcher_type.tp_basicsize = sizeof(Dispatcher);
  dispatcher_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  dispatcher_type.tp_vectorcall_offset = offsetof(Dispatcher, vectorcall);
  dispatcher_type.tp_call = PyVectorcall_Call;
  dispatcher_type.tp_new = dispatcher_new;
  dispatcher_type.tp_dealloc = dispatcher_dealloc;
  if (PyType_Ready(&call_type) < 0 || PyType_Ready(&dispatcher_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  Py_INCREF(&call_type);
  Py_INCREF(&dispatcher_type);
  if (PyModule_AddObject(m, "Call", reinterpret_cast<PyObject*>(&call_type)) < 0 ||
      PyModule_AddObject(m, "Dispatcher", reinterpret_cast<PyObject*>(&dispatcher_type)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
