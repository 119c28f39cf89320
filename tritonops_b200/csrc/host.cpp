// The host side of the tensor-level entry points in native code: checks, output and scratch
// allocation, argument structs and the library call of one eager call, without the interpreter.
// (Measured on the 128-row attention call: 25 us of Python around a 6 us kernel.)
//
// Every function takes its arguments by position and answers None for anything but plain strided
// CUDA tensors of one device in the layout the kernels take: subclasses, functorch wrappers,
// active dispatch modes, tracing, other dtypes, odd strides and wrong shapes all go to the Python
// path in ops.py, which copies or raises as it always did.  A non-zero library status is returned
// as an int for that module to raise.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <exception>

#include "../../include/b200attn.h"

namespace {

// entry points of libb200attn.so, resolved by init()
struct Lib {
  decltype(&b200attn_last_launch_count) last_launch_count;
  decltype(&b200attn_prefill_fwd) prefill_fwd, sparse_prefill_fwd;
  decltype(&b200attn_prefill_bwd_workspace_bytes) prefill_bwd_workspace_bytes;
  decltype(&b200attn_prefill_bwd) prefill_bwd;
  decltype(&b200attn_decode_workspace_bytes) decode_workspace_bytes;
  decltype(&b200attn_decode_fwd) decode_fwd, sparse_decode_fwd;
  decltype(&b200attn_paged_decode_workspace_bytes) paged_decode_workspace_bytes;
  decltype(&b200attn_paged_decode_fwd) paged_decode_fwd;
  decltype(&b200attn_kv_append) kv_append;
  decltype(&b200attn_topk_blocks) topk_blocks;
  decltype(&b200attn_rmsnorm_fwd) rmsnorm_fwd;
  decltype(&b200attn_rmsnorm_bwd_workspace_bytes) rmsnorm_bwd_workspace_bytes;
  decltype(&b200attn_rmsnorm_bwd) rmsnorm_bwd;
} L;
bool ready = false;

// Something the Python path should see: thrown by the argument readers, answered with None.
struct Unusual {};

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) throw Unusual();
  const at::Tensor& t = THPVariable_Unpack(o);
  static const c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                        c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                        c10::DispatchKey::Conjugate, c10::DispatchKey::Negative,
                                        c10::DispatchKey::ZeroTensor, c10::DispatchKey::Quantized});
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.key_set().has_any(odd)) throw Unusual();
  return t;
}
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); throw Unusual(); }
  return v;
}
int int32(PyObject* o) {
  const long long v = integer(o);
  if (v < INT32_MIN || v > INT32_MAX) throw Unusual();
  return (int)v;
}
float real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); throw Unusual(); }
  return (float)v;
}
void need(bool ok) { if (!ok) throw Unusual(); }

int dtype16(const at::Tensor& t) {
  if (t.scalar_type() == at::kHalf) return B200ATTN_F16;
  if (t.scalar_type() == at::kBFloat16) return B200ATTN_BF16;
  throw Unusual();
}
int dtype_any(const at::Tensor& t) { return t.scalar_type() == at::kFloat ? (int)B200ATTN_F32 : dtype16(t); }

// rows of 16-byte addressable 16-bit elements (what ops._rowmajor16 would leave alone)
void row_major(const at::Tensor& t, const at::Tensor& like, int64_t dim) {
  need(t.dim() == dim && t.device() == like.device() && t.scalar_type() == like.scalar_type());
  need(t.stride(dim - 1) == 1 && ((uintptr_t)t.data_ptr() & 15) == 0);
  for (int64_t i = 0; i + 1 < dim; ++i) need(t.stride(i) % 8 == 0);
}
// a contiguous int32 tensor of the call's device, or none
const int32_t* int_list(PyObject* o, const at::Tensor& like, at::Tensor* keep = nullptr) {
  if (o == Py_None) return nullptr;
  const at::Tensor& t = tensor(o);
  need(t.scalar_type() == at::kInt && t.is_contiguous() && t.device() == like.device());
  if (keep) *keep = t;
  return t.const_data_ptr<int32_t>();
}

at::Tensor scratch(size_t bytes, const at::Tensor& like) {
  return at::empty({(int64_t)std::max<size_t>(bytes, 16)}, like.options().dtype(at::kByte).requires_grad(false));
}
at::Tensor fresh(at::IntArrayRef sizes, const at::Tensor& like) {
  return at::empty(sizes, like.options().requires_grad(false));
}

// One library call on the current stream of the tensors' device, without the interpreter lock.
template <typename F, typename A>
int call(F fn, const A& args, const at::Tensor& like, long long& launches) {
  b200attn_stream_t stream = c10::cuda::getCurrentCUDAStream(like.device().index()).stream();
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = fn(&args, stream);
  launches = L.last_launch_count();
  Py_END_ALLOW_THREADS
  return status;
}

PyObject* none() { Py_RETURN_NONE; }

// (launches, tensor, ...) of a successful call, the status of a failed one
PyObject* answer(int status, long long launches, std::initializer_list<at::Tensor> out) {
  if (status != B200ATTN_OK) return PyLong_FromLong(status);
  PyObject* r = PyTuple_New(1 + (Py_ssize_t)out.size());
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, PyLong_FromLongLong(launches));
  Py_ssize_t i = 1;
  for (const at::Tensor& t : out) {
    PyObject* o = THPVariable_Wrap(t);
    if (!o) { Py_DECREF(r); return nullptr; }
    PyTuple_SET_ITEM(r, i++, o);
  }
  return r;
}

// Runs an entry point's body; what the body will not take, and every C++ exception, is None
// (ops.py then meets the same condition itself, an allocation that fails for instance).
template <typename Body>
PyObject* guarded(Py_ssize_t n, Py_ssize_t want, Body body) {
  if (!ready || n != want || c10::impl::TorchDispatchModeTLS::stack_len() > 0 || at::tracer::impl::is_dispatch_enabled())
    return none();
  try {
    return body();
  } catch (const Unusual&) {
    return none();
  } catch (const std::exception&) {
    PyErr_Clear();
    return none();
  }
}

template <typename A>
void strides4(A& a, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o,
              const at::Tensor& lse) {
  a.q_stride_b = q.stride(0); a.q_stride_t = q.stride(1); a.q_stride_h = q.stride(2);
  a.k_stride_b = k.stride(0); a.k_stride_t = k.stride(1); a.k_stride_h = k.stride(2);
  a.v_stride_b = v.stride(0); a.v_stride_t = v.stride(1); a.v_stride_h = v.stride(2);
  a.o_stride_b = o.stride(0); a.o_stride_t = o.stride(1); a.o_stride_h = o.stride(2);
  a.lse_stride_b = lse.stride(0); a.lse_stride_t = lse.stride(1); a.lse_stride_h = lse.stride(2);
}
template <typename A>
void extents(A& a, const at::Tensor& q, const at::Tensor& k, const at::Tensor& cu, const int32_t* cu_ptr,
             int max_seqlen) {
  const int64_t rows = q.size(0), tokens = q.size(1);
  need(tokens <= INT32_MAX);
  a.dtype = dtype16(q);
  a.heads_q = (int)q.size(2); a.heads_kv = (int)k.size(2); a.head_dim = (int)q.size(3);
  if (cu_ptr) {
    need(rows == 1);
    a.batch = (int)cu.numel() - 1; a.cu_seqlens = cu_ptr;
    a.max_seqlen = max_seqlen; a.total_tokens = tokens; a.seqlen = 0;
  } else {
    a.batch = (int)rows; a.seqlen = (int)tokens; a.max_seqlen = (int)tokens; a.total_tokens = tokens;
  }
}

// q, k, v, cu | None, max_seqlen, scale, scale_has_log2e, causal, lse_base2, sparsity, window_local,
// window_global, block_idx | None, block_cnt | None, block_size
PyObject* prefill(PyObject*, PyObject* const* x, Py_ssize_t n) {
  return guarded(n, 15, [&]() -> PyObject* {
    const at::Tensor &q = tensor(x[0]), &k = tensor(x[1]), &v = tensor(x[2]);
    row_major(q, q, 4); row_major(k, q, 4); row_major(v, q, 4);
    need(k.size(3) == q.size(3) && v.size(3) == q.size(3));
    at::Tensor cu;
    const int32_t* cu_ptr = int_list(x[3], q, &cu);
    b200attn_prefill_args a = {};
    extents(a, q, k, cu, cu_ptr, int32(x[4]));
    a.softmax_scale = real(x[5]); a.scale_has_log2e = int32(x[6]);
    a.causal = int32(x[7]); a.lse_base2 = int32(x[8]); a.sparsity = int32(x[9]);
    a.window_local = int32(x[10]); a.window_global = int32(x[11]);
    if (x[12] != Py_None) {
      at::Tensor idx;
      a.block_idx = int_list(x[12], q, &idx); a.block_cnt = int_list(x[13], q);
      need(idx.dim() == 4);
      a.block_size = int32(x[14]); a.n_qblocks = (int)idx.size(2); a.max_nnz = (int)idx.size(3);
    }
    const c10::cuda::CUDAGuard device(q.device());
    at::Tensor o = fresh(q.sizes(), q);
    at::Tensor lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat).requires_grad(false));
    a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = o.data_ptr(); a.lse = lse.data_ptr<float>();
    strides4(a, q, k, v, o, lse);
    long long launches;
    const int st = call(a.sparsity == B200ATTN_DENSE ? L.prefill_fwd : L.sparse_prefill_fwd, a, q, launches);
    return answer(st, launches, {o, lse});
  });
}

// q, k, v, o, do, lse, cu | None, max_seqlen, scale, scale_has_log2e, causal, lse_base2
PyObject* prefill_bwd(PyObject*, PyObject* const* x, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const at::Tensor &q = tensor(x[0]), &k = tensor(x[1]), &v = tensor(x[2]), &o = tensor(x[3]), &g = tensor(x[4]),
                     &lse = tensor(x[5]);
    for (const at::Tensor* t : {&q, &k, &v, &o, &g}) {
      row_major(*t, q, 4);
      need(t->size(3) == q.size(3));
    }
    need(lse.scalar_type() == at::kFloat && lse.dim() == 3 && lse.is_contiguous() && lse.device() == q.device());
    at::Tensor cu;
    const int32_t* cu_ptr = int_list(x[6], q, &cu);
    b200attn_prefill_bwd_args a = {};
    extents(a, q, k, cu, cu_ptr, int32(x[7]));
    a.softmax_scale = real(x[8]); a.scale_has_log2e = int32(x[9]); a.causal = int32(x[10]); a.lse_base2 = int32(x[11]);
    const c10::cuda::CUDAGuard device(q.device());
    at::Tensor dq = fresh(q.sizes(), q), dk = fresh(k.sizes(), k), dv = fresh(v.sizes(), v);
    a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = o.data_ptr(); a.d_o = g.data_ptr();
    a.lse = lse.data_ptr<float>();
    a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
    strides4(a, q, k, v, o, lse);
    a.do_stride_b = g.stride(0); a.do_stride_t = g.stride(1); a.do_stride_h = g.stride(2);
    a.dq_stride_b = dq.stride(0); a.dq_stride_t = dq.stride(1); a.dq_stride_h = dq.stride(2);
    a.dk_stride_b = dk.stride(0); a.dk_stride_t = dk.stride(1); a.dk_stride_h = dk.stride(2);
    a.dv_stride_b = dv.stride(0); a.dv_stride_t = dv.stride(1); a.dv_stride_h = dv.stride(2);
    at::Tensor ws = scratch(L.prefill_bwd_workspace_bytes(&a), q);
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
    long long launches;
    const int st = call(L.prefill_bwd, a, q, launches);
    return answer(st, launches, {dq, dk, dv});
  });
}

// q, k, v, lens, lens_are_cu, max_seqlen, scale, chunk, sparsity, window_global, window_local,
// block_idx | None, block_cnt | None, block_size
PyObject* decode(PyObject*, PyObject* const* x, Py_ssize_t n) {
  return guarded(n, 14, [&]() -> PyObject* {
    const at::Tensor &q = tensor(x[0]), &k = tensor(x[1]), &v = tensor(x[2]);
    row_major(q, q, 3); row_major(k, q, 4); row_major(v, q, 4);
    need(k.size(3) == q.size(2) && v.size(3) == q.size(2) && x[3] != Py_None && q.size(0) <= INT32_MAX);
    const int32_t* lens = int_list(x[3], q);
    b200attn_decode_args a = {};
    a.dtype = dtype16(q);
    a.batch = (int)q.size(0); a.heads_q = (int)q.size(1); a.heads_kv = (int)k.size(2); a.head_dim = (int)q.size(2);
    a.max_seqlen = (int)std::min<long long>(int32(x[5]), k.size(1));
    if (PyObject_IsTrue(x[4])) a.cu_seqlens = lens; else a.seqlens = lens;
    a.softmax_scale = real(x[6]); a.chunk_tokens = int32(x[7]); a.sparsity = int32(x[8]);
    a.window_global = int32(x[9]); a.window_local = int32(x[10]);
    if (x[11] != Py_None) {
      at::Tensor idx;
      a.block_idx = int_list(x[11], q, &idx); a.block_cnt = int_list(x[12], q);
      need(idx.dim() >= 1 && idx.numel() > 0);
      a.block_size = int32(x[13]); a.max_sel = (int)idx.size(idx.dim() - 1);
    }
    const c10::cuda::CUDAGuard device(q.device());
    at::Tensor o = fresh(q.sizes(), q);
    a.q = q.data_ptr(); a.k_cache = k.data_ptr(); a.v_cache = v.data_ptr(); a.o = o.data_ptr();
    a.q_stride_b = q.stride(0); a.q_stride_h = q.stride(1);
    a.k_stride_b = k.stride(0); a.k_stride_t = k.stride(1); a.k_stride_h = k.stride(2);
    a.v_stride_b = v.stride(0); a.v_stride_t = v.stride(1); a.v_stride_h = v.stride(2);
    a.o_stride_b = o.stride(0); a.o_stride_h = o.stride(1);
    at::Tensor ws = scratch(L.decode_workspace_bytes(&a), q);
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
    long long launches;
    const int st = call(a.sparsity == B200ATTN_DENSE ? L.decode_fwd : L.sparse_decode_fwd, a, q, launches);
    return answer(st, launches, {o});
  });
}

// q, k_pages, v_pages, page_table, seqlens, max_seqlen | None, scale | None, chunk
PyObject* paged_decode(PyObject*, PyObject* const* x, Py_ssize_t n) {
  return guarded(n, 8, [&]() -> PyObject* {
    const at::Tensor &q = tensor(x[0]), &k = tensor(x[1]), &v = tensor(x[2]);
    row_major(q, q, 3); row_major(k, q, 4); row_major(v, q, 4);
    need(k.size(3) == q.size(2) && v.size(3) == q.size(2) && x[3] != Py_None && x[4] != Py_None);
    at::Tensor table;
    b200attn_paged_decode_args a = {};
    a.page_table = int_list(x[3], q, &table); a.seqlens = int_list(x[4], q);
    need(table.dim() == 2 && k.size(0) <= INT32_MAX);
    a.dtype = dtype16(q);
    a.batch = (int)q.size(0); a.heads_q = (int)q.size(1); a.heads_kv = (int)k.size(2); a.head_dim = (int)q.size(2);
    a.page_size = (int)k.size(1); a.num_pages = (int)k.size(0); a.max_pages_per_seq = (int)table.size(1);
    const long long cap = table.size(1) * k.size(1);
    need(cap <= INT32_MAX);
    a.max_seqlen = x[5] == Py_None ? (int)cap : int32(x[5]);
    a.softmax_scale = x[6] == Py_None ? (float)std::pow((double)q.size(2), -0.5) : real(x[6]);
    a.chunk_tokens = int32(x[7]);
    const c10::cuda::CUDAGuard device(q.device());
    at::Tensor o = fresh(q.sizes(), q);
    a.q = q.data_ptr(); a.k_pages = k.data_ptr(); a.v_pages = v.data_ptr(); a.o = o.data_ptr();
    a.q_stride_b = q.stride(0); a.q_stride_h = q.stride(1);
    a.k_stride_page = k.stride(0); a.k_stride_t = k.stride(1); a.k_stride_h = k.stride(2);
    a.v_stride_page = v.stride(0); a.v_stride_t = v.stride(1); a.v_stride_h = v.stride(2);
    a.o_stride_b = o.stride(0); a.o_stride_h = o.stride(1);
    at::Tensor ws = scratch(L.paged_decode_workspace_bytes(&a), q);
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
    long long launches;
    const int st = call(L.paged_decode_fwd, a, q, launches);
    return answer(st, launches, {o});
  });
}

// k_cache, v_cache, new_k, new_v, seqlens
PyObject* append_kv(PyObject*, PyObject* const* x, Py_ssize_t n) {
  return guarded(n, 5, [&]() -> PyObject* {
    const at::Tensor &k = tensor(x[0]), &v = tensor(x[1]), &nk = tensor(x[2]), &nv = tensor(x[3]);
    need(k.dim() == 4 && v.dim() == 4 && nk.dim() == 3 && nv.dim() == 3);
    need(k.strides() == v.strides() && nk.strides() == nv.strides());
    for (const at::Tensor* t : {&v, &nk, &nv}) need(t->device() == k.device());
    need(x[4] != Py_None);
    b200attn_kv_append_args a = {};
    a.seqlens = int_list(x[4], k);
    a.new_k = nk.data_ptr(); a.new_v = nv.data_ptr(); a.k_cache = k.data_ptr(); a.v_cache = v.data_ptr();
    a.batch = (int)k.size(0); a.heads = (int)k.size(2); a.head_dim = (int)k.size(3); a.capacity = (int)k.size(1);
    a.new_stride_b = nk.stride(0); a.new_stride_h = nk.stride(1);
    a.cache_stride_b = k.stride(0); a.cache_stride_t = k.stride(1); a.cache_stride_h = k.stride(2);
    const c10::cuda::CUDAGuard device(k.device());
    long long launches;
    const int st = call(L.kv_append, a, k, launches);
    return answer(st, launches, {});
  });
}

// scores, top_k, n_valid | None, force_first, force_last
PyObject* topk_blocks(PyObject*, PyObject* const* x, Py_ssize_t n) {
  return guarded(n, 5, [&]() -> PyObject* {
    const at::Tensor& s = tensor(x[0]);
    need(s.scalar_type() == at::kFloat && s.dim() >= 1 && s.numel() > 0 && s.is_contiguous());
    const int64_t blocks = s.size(s.dim() - 1), rows = s.numel() / blocks;
    need(blocks <= INT32_MAX && rows <= INT32_MAX);
    const int top_k = int32(x[1]);
    need(top_k >= 0);
    b200attn_topk_blocks_args a = {};
    at::Tensor valid;
    a.n_valid = int_list(x[2], s, &valid);
    need(!valid.defined() || valid.numel() == rows);
    a.scores = s.data_ptr<float>(); a.score_stride_row = blocks;
    a.rows = (int)rows; a.n_blocks = (int)blocks; a.top_k = top_k;
    a.force_first = int32(x[3]); a.force_last = int32(x[4]);
    const c10::cuda::CUDAGuard device(s.device());
    std::vector<int64_t> sizes(s.sizes().begin(), s.sizes().end() - 1);
    const auto ints = s.options().dtype(at::kInt).requires_grad(false);
    at::Tensor cnt = at::empty(sizes, ints);
    sizes.push_back(top_k);
    at::Tensor idx = at::empty(sizes, ints);
    a.block_idx = idx.data_ptr<int32_t>(); a.block_cnt = cnt.data_ptr<int32_t>();
    long long launches;
    const int st = call(L.topk_blocks, a, s, launches);
    return answer(st, launches, {idx, cnt});
  });
}

// [..., dim] as rows that can be walked with one stride
int64_t rows_of(const at::Tensor& t, int64_t& stride) {
  need(t.dim() >= 1 && t.numel() > 0 && t.stride(t.dim() - 1) == 1);
  const int64_t dim = t.size(t.dim() - 1);
  if (t.dim() == 2) { stride = t.stride(0); return t.size(0); }
  need(t.is_contiguous());
  stride = dim;
  return t.numel() / dim;
}
void rms_types(const at::Tensor& x, const at::Tensor& w, int& xd, int& wd) {
  xd = dtype_any(x); wd = dtype_any(w);
  need(wd == xd || wd == B200ATTN_F32);
  need(w.dim() == 1 && w.is_contiguous() && w.device() == x.device() && w.numel() == x.size(x.dim() - 1));
  need(w.numel() <= INT32_MAX);
}

// x, weight, eps
PyObject* rmsnorm_fwd(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded(n, 3, [&]() -> PyObject* {
    const at::Tensor &x = tensor(p[0]), &w = tensor(p[1]);
    b200attn_rmsnorm_fwd_args a = {};
    int64_t xs;
    const int64_t rows = rows_of(x, xs);
    rms_types(x, w, a.x_dtype, a.w_dtype);
    a.eps = real(p[2]);
    const c10::cuda::CUDAGuard device(x.device());
    at::Tensor y = fresh(x.sizes(), x);
    at::Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat).requires_grad(false));
    a.x = x.data_ptr(); a.weight = w.data_ptr(); a.y = y.data_ptr(); a.rstd = rstd.data_ptr<float>();
    a.rows = rows; a.dim = (int)w.numel(); a.x_stride_row = xs; a.y_stride_row = w.numel();
    long long launches;
    const int st = call(L.rmsnorm_fwd, a, x, launches);
    return answer(st, launches, {y, rstd});
  });
}

// dy, x, weight, rstd
PyObject* rmsnorm_bwd(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded(n, 4, [&]() -> PyObject* {
    const at::Tensor &g = tensor(p[0]), &x = tensor(p[1]), &w = tensor(p[2]), &rstd = tensor(p[3]);
    b200attn_rmsnorm_bwd_args a = {};
    int64_t xs, gs;
    const int64_t rows = rows_of(x, xs);
    need(g.scalar_type() == x.scalar_type() && g.device() == x.device() && g.sizes() == x.sizes());
    need(rows_of(g, gs) == rows);
    rms_types(x, w, a.x_dtype, a.w_dtype);
    need(rstd.scalar_type() == at::kFloat && rstd.numel() == rows && rstd.is_contiguous() && rstd.device() == x.device());
    const c10::cuda::CUDAGuard device(x.device());
    at::Tensor dx = fresh(x.sizes(), x), dw = fresh(w.sizes(), w);
    a.dy = g.data_ptr(); a.x = x.data_ptr(); a.weight = w.data_ptr(); a.rstd = rstd.data_ptr<float>();
    a.dx = dx.data_ptr(); a.dweight = dw.data_ptr();
    a.rows = rows; a.dim = (int)w.numel();
    a.dy_stride_row = gs; a.x_stride_row = xs; a.dx_stride_row = w.numel();
    at::Tensor ws = scratch(L.rmsnorm_bwd_workspace_bytes(&a), x);
    a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
    long long launches;
    const int st = call(L.rmsnorm_bwd, a, x, launches);
    return answer(st, launches, {dx, dw});
  });
}

template <typename F>
bool bind(void* h, const char* name, F& fn) {
  fn = reinterpret_cast<F>(dlsym(h, name));
  if (!fn) PyErr_Format(PyExc_RuntimeError, "libb200attn.so lacks %s; rebuild it", name);
  return fn != nullptr;
}

// init(path of libb200attn.so, sizes of the argument structs as the caller knows them): resolve its
// entry points
PyObject* init(PyObject*, PyObject* const* x, Py_ssize_t n) {
  const size_t sizes[] = {sizeof(b200attn_prefill_args), sizeof(b200attn_prefill_bwd_args), sizeof(b200attn_decode_args),
                          sizeof(b200attn_paged_decode_args), sizeof(b200attn_kv_append_args),
                          sizeof(b200attn_topk_blocks_args), sizeof(b200attn_rmsnorm_fwd_args),
                          sizeof(b200attn_rmsnorm_bwd_args)};
  constexpr Py_ssize_t kStructs = sizeof(sizes) / sizeof(sizes[0]);
  bool same = n == 1 + kStructs;
  for (Py_ssize_t i = 0; same && i < kStructs; ++i) same = PyLong_AsSize_t(x[1 + i]) == sizes[i];
  if (!same) {
    PyErr_Clear();
    return PyErr_Format(PyExc_RuntimeError, "the native call path was built with other argument structs; rebuild it");
  }
  const char* p = PyUnicode_AsUTF8(x[0]);
  if (!p) return nullptr;
  void* h = dlopen(p, RTLD_NOW | RTLD_LOCAL);
  if (!h) return PyErr_Format(PyExc_RuntimeError, "%s", dlerror());
#define B(field, name) bind(h, "b200attn_" #name, L.field)
  if (!(B(last_launch_count, last_launch_count) && B(prefill_fwd, prefill_fwd) &&
        B(sparse_prefill_fwd, sparse_prefill_fwd) && B(prefill_bwd_workspace_bytes, prefill_bwd_workspace_bytes) &&
        B(prefill_bwd, prefill_bwd) && B(decode_workspace_bytes, decode_workspace_bytes) &&
        B(decode_fwd, decode_fwd) && B(sparse_decode_fwd, sparse_decode_fwd) &&
        B(paged_decode_workspace_bytes, paged_decode_workspace_bytes) && B(paged_decode_fwd, paged_decode_fwd) &&
        B(kv_append, kv_append) && B(topk_blocks, topk_blocks) && B(rmsnorm_fwd, rmsnorm_fwd) &&
        B(rmsnorm_bwd_workspace_bytes, rmsnorm_bwd_workspace_bytes) && B(rmsnorm_bwd, rmsnorm_bwd)))
    return nullptr;
#undef B
  ready = true;
  Py_RETURN_NONE;
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(prefill), FAST(prefill_bwd), FAST(decode), FAST(paged_decode), FAST(append_kv),
                         FAST(topk_blocks), FAST(rmsnorm_fwd), FAST(rmsnorm_bwd),
                         FAST(init), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200host(void) { return PyModule_Create(&module); }
