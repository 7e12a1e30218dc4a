// The per-call host work of tyr_b200/nn.py in native code: reads sizes, strides and pointers out of
// torch tensors, applies the argument checks, allocates the outputs and calls the C ABI of
// include/tyr_b200_attn.h on torch's current stream.
//
// A single-token step or a short prompt is a few microseconds of device work, and building the
// argument structures from Python cost 14 to 38 us per call (ctypes fields, a device context
// manager, tensor attributes one by one): the host set the pace.  Host time of a pass with the GPU idle, before ->
// after: three prologues and a dense decode 79 -> 23 us, the typed call on a 517-row prompt 21 -> 5.5 us, forward and
// backward 81 -> 18 us, a single-row typed call 35 -> 9.5 us.
// Nothing is cached here: every call reads its tensors anew.
//
// The Python functions keep names, defaults and results; they hand their arguments over by position.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <stdexcept>

#include "../../include/tyr_b200_attn.h"

namespace {

using at::Tensor;

PyObject* g_attn_error = nullptr;  // tyr_b200._lib.AttnError, handed over at import

struct ValueError : std::runtime_error { using std::runtime_error::runtime_error; };
struct CallError { int code; };  // a status of the C ABI

// lets other Python threads run while this one allocates and launches
struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

template <class F>
PyObject* guarded(F&& f) {
  HANDLE_TH_ERRORS
  try {
    return f();
  } catch (const ValueError& e) {
    PyErr_SetString(PyExc_ValueError, e.what());
  } catch (const CallError& e) {
    PyObject* x = g_attn_error ? PyObject_CallFunction(g_attn_error, "i", e.code) : nullptr;
    if (x) {
      PyErr_SetObject(g_attn_error, x);
      Py_DECREF(x);
    } else if (!PyErr_Occurred()) {
      PyErr_SetString(PyExc_RuntimeError, tyr_b200_attn_strerror(e.code));
    }
  }
  return nullptr;
  END_HANDLE_TH_ERRORS
}

void check_rc(int rc) {
  if (rc != 0) throw CallError{rc};
}

const Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) throw ValueError(std::string(what) + " must be a torch tensor");
  return THPVariable_Unpack(o);
}
// nullptr for None
const Tensor* maybe(PyObject* o, const char* what) { return o == Py_None ? nullptr : &tensor(o, what); }

int64_t integer(PyObject* o) {  // as int(o)
  PyObject* l = PyLong_CheckExact(o) ? Py_NewRef(o) : PyNumber_Long(o);
  if (!l) throw python_error();
  const int64_t v = PyLong_AsLongLong(l);
  Py_DECREF(l);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
float scale_of(PyObject* o) {  // None selects the default in the library
  if (o == Py_None) return 0.0f;
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return static_cast<float>(v);
}

// the launcher checks of Tyr/GPU/Codegen/Attribute.lean:333-336, as exceptions
void require_cuda(const Tensor& t) {
  if (!t.is_cuda()) throw ValueError("tensor must be on a CUDA device");
  if (t.dim() > 4) throw ValueError("tensor rank must be <= 4");
  if (t.dim() < 1 || t.stride(-1) != 1) throw ValueError("tensor must have unit stride on the head dimension");
}
void require_count(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) throw ValueError("wrong number of arguments");
}

void strides3(int64_t* s, const Tensor& t) {
  s[0] = t.stride(0);
  s[1] = t.stride(1);
  s[2] = t.stride(2);
}
int32_t i32(int64_t v) { return static_cast<int32_t>(v); }

Tensor new_tensor(at::IntArrayRef size, at::ScalarType dt, at::Device dev) {
  return at::detail::empty_cuda(size, dt, dev, c10::nullopt);
}
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// The mask as the C ABI takes it, one byte per key; checked only, other types are converted by the Python caller.
Tensor key_bytes(const Tensor& m, int64_t batch, int64_t kv_seq) {
  const bool byte = m.scalar_type() == at::kBool || m.scalar_type() == at::kByte;
  if (!m.is_cuda() || !byte || m.dim() != 2 || m.stride(1) != 1 || m.size(0) != batch || m.size(1) != kv_seq)
    throw ValueError("key_mask must be a uint8/bool CUDA tensor [batch, kv_seq]");
  return m;
}

void fill_prefill(TyrAttnPrefillArgs& a, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor* o) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) throw ValueError("q, k, v must be [batch, heads, seq, head_dim]");
  if (v.sizes() != k.sizes() || k.size(0) != q.size(0) || k.size(3) != q.size(3) || (o && o->sizes() != q.sizes()))
    throw ValueError("shape mismatch among q, k, v, out");
  const at::ScalarType dt = q.scalar_type();
  if (k.scalar_type() != dt || v.scalar_type() != dt || (o && o->scalar_type() != dt))
    throw ValueError("q, k, v and out must share one dtype");
  if (dt != at::kBFloat16 && dt != at::kFloat) throw ValueError("dtype must be bfloat16 (float32 in check mode)");
  std::memset(&a, 0, sizeof(a));
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.batch = i32(q.size(0));
  a.n_head = i32(q.size(1));
  a.n_kv_head = i32(k.size(1));
  a.q_seq = i32(q.size(2));
  a.kv_seq = i32(k.size(2));
  a.head_dim = i32(q.size(3));
  strides3(a.q_stride, q);
  strides3(a.k_stride, k);
  strides3(a.v_stride, v);
  a.dtype = dt == at::kBFloat16 ? TYR_ATTN_BF16 : TYR_ATTN_F32;
}

// q, k, v, is_causal, scale, out, lse, return_lse, check_mode, window_size, key_mask, workspace -> (out, lse)
PyObject* attention_fwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    require_count(n, 12);
    const Tensor &q = tensor(args[0], "q"), &k = tensor(args[1], "k"), &v = tensor(args[2], "v");
    require_cuda(q);
    require_cuda(k);
    require_cuda(v);
    const bool causal = truth(args[3]), return_lse = truth(args[7]), check_mode = truth(args[8]);
    const Tensor *out_in = maybe(args[5], "out"), *lse_in = maybe(args[6], "lse"), *mask = maybe(args[10], "key_mask");
    const bool never_split = args[11] == Py_False;
    const Tensor* ws_in = never_split ? nullptr : maybe(args[11], "workspace");
    TyrAttnPrefillArgs a;
    fill_prefill(a, q, k, v, out_in);
    if (out_in) require_cuda(*out_in);
    a.is_causal = causal;
    a.scale = scale_of(args[4]);
    a.check_mode = check_mode;
    a.window_size = i32(integer(args[9]));
    if (lse_in && (lse_in->scalar_type() != at::kFloat || !lse_in->is_contiguous() || lse_in->dim() != 3 ||
                   lse_in->size(0) != q.size(0) || lse_in->size(1) != q.size(1) || lse_in->size(2) != q.size(2)))
      throw ValueError("lse must be a contiguous float32 [batch, n_head, q_seq] tensor");
    if (mask) {
      const Tensor m = key_bytes(*mask, k.size(0), k.size(2));
      a.key_mask = static_cast<const uint8_t*>(m.data_ptr());
      a.key_mask_stride = m.stride(0);
    }
    Tensor out, lse, ws;
    {
      NoGil no_gil;
      c10::cuda::OptionalCUDAGuard guard(q.device());
      out = out_in ? *out_in : new_tensor(q.sizes(), q.scalar_type(), q.device());
      if (lse_in) lse = *lse_in;
      else if (return_lse) lse = new_tensor(q.sizes().slice(0, 3), at::kFloat, q.device());
      a.o = out.data_ptr();
      strides3(a.o_stride, out);
      a.lse = lse.defined() ? static_cast<float*>(lse.data_ptr()) : nullptr;
      // only unmasked, non-causal calls are ever split: no query for the others
      if (!never_split && !causal && a.window_size == 0 && !mask && !check_mode) {
        const int64_t need = tyr_b200_attn_prefill_workspace_bytes(&a);
        if (need > 0) {
          ws = ws_in ? *ws_in : new_tensor({need}, at::kByte, q.device());
          if (ws.scalar_type() != at::kByte || !ws.is_contiguous() || ws.device() != q.device() ||
              reinterpret_cast<uintptr_t>(ws.data_ptr()) % 256 != 0)
            throw ValueError("workspace must be a contiguous uint8 CUDA tensor on q's device, 256-byte aligned");
          a.workspace = ws.data_ptr();
          a.workspace_bytes = ws.numel();
        }
      }
      check_rc(tyr_b200_attn_prefill(&a, stream_of(q)));
    }
    PyObject* t = PyTuple_New(2);
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(out)));
    if (lse.defined()) {
      PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(lse)));
    } else {
      Py_INCREF(Py_None);
      PyTuple_SET_ITEM(t, 1, Py_None);
    }
    return t;
  });
}

// an uninitialised tensor with t's sizes and, where they are dense, its strides
Tensor like(const Tensor& t) {
  return t.is_contiguous() ? new_tensor(t.sizes(), t.scalar_type(), t.device()) : at::empty_like(t);
}

// q, k, v, o, lse, d_o, is_causal, scale, workspace, window_size, key_mask -> (d_q, d_k, d_v)
PyObject* attention_bwd(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    require_count(n, 11);
    const Tensor &q = tensor(args[0], "q"), &k = tensor(args[1], "k"), &v = tensor(args[2], "v"), &o = tensor(args[3], "o"),
                 &lse = tensor(args[4], "lse"), &d_o = tensor(args[5], "d_o");
    for (const Tensor* t : {&q, &k, &v, &o, &d_o, &lse}) require_cuda(*t);
    if (q.dim() != 4 || k.dim() != 4) throw ValueError("q, k, v must be [batch, heads, seq, head_dim]");
    if (v.sizes() != k.sizes() || k.size(0) != q.size(0) || k.size(3) != q.size(3) || o.sizes() != q.sizes() ||
        d_o.sizes() != q.sizes() || lse.sizes() != q.sizes().slice(0, 3))
      throw ValueError("shape mismatch among q, k, v, o, d_o, lse");
    for (const Tensor* t : {&q, &k, &v, &o, &d_o})
      if (t->scalar_type() != at::kBFloat16) throw ValueError("q, k, v, o, d_o must be bfloat16");
    if (lse.scalar_type() != at::kFloat || !lse.is_contiguous())
      throw ValueError("lse must be a contiguous float32 [batch, n_head, q_seq] tensor");
    const Tensor *ws_in = maybe(args[8], "workspace"), *mask = maybe(args[10], "key_mask");
    TyrAttnBackwardArgs a;
    std::memset(&a, 0, sizeof(a));
    a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = o.data_ptr(); a.d_o = d_o.data_ptr();
    a.lse = static_cast<const float*>(lse.data_ptr());
    a.batch = i32(q.size(0)); a.n_head = i32(q.size(1)); a.n_kv_head = i32(k.size(1));
    a.q_seq = i32(q.size(2)); a.kv_seq = i32(k.size(2)); a.head_dim = i32(q.size(3));
    strides3(a.q_stride, q); strides3(a.k_stride, k); strides3(a.v_stride, v); strides3(a.o_stride, o);
    strides3(a.do_stride, d_o);
    a.dtype = TYR_ATTN_BF16;
    a.is_causal = truth(args[6]);
    a.scale = scale_of(args[7]);
    a.window_size = i32(integer(args[9]));
    if (mask) {
      const Tensor m = key_bytes(*mask, k.size(0), k.size(2));
      a.key_mask = static_cast<const uint8_t*>(m.data_ptr());
      a.key_mask_stride = m.stride(0);
    }
    const int64_t need = (int64_t)tyr_b200_attn_backward_workspace_bytes(a.batch, a.n_head, a.q_seq);
    Tensor ws, d_q, d_k, d_v;
    {
      NoGil no_gil;
      c10::cuda::OptionalCUDAGuard guard(q.device());
      ws = ws_in ? *ws_in : new_tensor({need / 4}, at::kFloat, q.device());
      if (ws.scalar_type() != at::kFloat || !ws.is_contiguous() || ws.numel() * 4 < need)
        throw ValueError("workspace must be a contiguous float32 CUDA tensor of the required size");
      d_q = like(q);
      d_k = like(k);
      d_v = like(v);
      a.d_q = d_q.data_ptr(); a.d_k = d_k.data_ptr(); a.d_v = d_v.data_ptr();
      strides3(a.dq_stride, d_q); strides3(a.dk_stride, d_k); strides3(a.dv_stride, d_v);
      a.workspace = ws.data_ptr();
      a.workspace_bytes = (uint64_t)ws.numel() * 4;
      check_rc(tyr_b200_attn_backward(&a, stream_of(q)));
    }
    PyObject* t = PyTuple_New(3);
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(d_q)));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(d_k)));
    PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(std::move(d_v)));
    return t;
  });
}

// The [batch, heads, head_dim] query of a single-token call, given as such or as [batch, heads, 1, head_dim].
struct QueryRows {
  int64_t batch, heads, d, stride_b, stride_h;
};
QueryRows query_rows(const Tensor& q) {
  if (q.dim() != 3 && q.dim() != 4) throw ValueError("q must be bf16 [batch, n_head, head_dim]");
  require_cuda(q);
  return {q.size(0), q.size(1), q.size(-1), q.stride(0), q.stride(1)};
}
PyObject* out_and_lse(Tensor& out, Tensor& lse, bool unsqueeze) {
  PyObject* t = PyTuple_New(2);
  if (!t) throw python_error();
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(unsqueeze ? out.unsqueeze(2) : std::move(out)));
  if (lse.defined()) {
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(unsqueeze ? lse.unsqueeze(2) : std::move(lse)));
  } else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(t, 1, Py_None);
  }
  return t;
}

// q, (batch, n_head, n_kv_head, max_kv_seq, head_dim, max_splits, total_kv_len), k_ptrs, v_ptrs, kv_lens, head_strides,
// workspace or None (the library's own array), workspace_bytes, scale, out, lse, return_lse -> (out, lse)
PyObject* decode_ragged(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    require_count(n, 18);
    const Tensor& q = tensor(args[0], "q");
    const QueryRows r = query_rows(q);
    TyrAttnDecodeArgs a;
    std::memset(&a, 0, sizeof(a));
    a.batch = i32(integer(args[1]));
    a.n_head = i32(integer(args[2]));
    a.n_kv_head = i32(integer(args[3]));
    a.max_kv_seq = i32(integer(args[4]));
    a.head_dim = i32(integer(args[5]));
    a.max_splits = i32(integer(args[6]));
    a.total_kv_len = integer(args[7]);
    if (q.scalar_type() != at::kBFloat16 || r.batch != a.batch || r.heads != a.n_head || r.d != a.head_dim)
      throw ValueError("q must be bf16 [batch, n_head, head_dim]");
    a.k_ptrs = static_cast<const void* const*>(tensor(args[8], "k_ptrs").data_ptr());
    a.v_ptrs = static_cast<const void* const*>(tensor(args[9], "v_ptrs").data_ptr());
    a.kv_lens = static_cast<const int32_t*>(tensor(args[10], "kv_lens").data_ptr());
    a.kv_head_strides = static_cast<const int64_t*>(tensor(args[11], "head_strides").data_ptr());
    const Tensor* ws = maybe(args[12], "workspace");
    a.workspace = ws ? ws->data_ptr() : nullptr;
    a.workspace_bytes = (size_t)integer(args[13]);
    a.scale = scale_of(args[14]);
    const Tensor *out_in = maybe(args[15], "out"), *lse_in = maybe(args[16], "lse");
    const bool return_lse = truth(args[17]);
    a.q = q.data_ptr();
    a.q_stride[0] = r.stride_b;
    a.q_stride[1] = r.stride_h;
    a.k_stride[2] = a.v_stride[2] = a.head_dim;
    Tensor out, lse;
    {
      NoGil no_gil;
      c10::cuda::OptionalCUDAGuard guard(q.device());
      out = out_in ? *out_in : new_tensor({r.batch, r.heads, r.d}, at::kBFloat16, q.device());
      if (lse_in) lse = *lse_in;
      else if (return_lse) lse = new_tensor({r.batch, r.heads}, at::kFloat, q.device());
      a.o = out.data_ptr();
      a.o_stride[0] = out.stride(0);
      a.o_stride[1] = out.stride(1);
      a.lse = lse.defined() ? static_cast<float*>(lse.data_ptr()) : nullptr;
      check_rc(ws ? tyr_b200_attn_decode(&a, stream_of(q)) : tyr_b200_attn_decode_static(&a, stream_of(q)));
    }
    return out_and_lse(out, lse, ws && q.dim() == 4);
  });
}

// q, k_cache, v_cache, kv_lens, kv_len, scale, workspace, max_splits -> (out, lse)
PyObject* decode_dense(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    require_count(n, 8);
    const Tensor &q = tensor(args[0], "q"), &k = tensor(args[1], "k_cache"), &v = tensor(args[2], "v_cache");
    const QueryRows r = query_rows(q);
    require_cuda(k);
    require_cuda(v);
    if (k.dim() != 4 || v.dim() != 4) throw ValueError("k_cache and v_cache must be [batch, n_kv_head, cap, head_dim]");
    const Tensor *lens = maybe(args[3], "kv_lens"), *ws_in = maybe(args[6], "workspace");
    TyrAttnDecodeArgs a;
    std::memset(&a, 0, sizeof(a));
    a.q = q.data_ptr();
    a.k = k.data_ptr();
    a.v = v.data_ptr();
    a.kv_lens = lens ? static_cast<const int32_t*>(lens->data_ptr()) : nullptr;
    a.batch = i32(r.batch);
    a.n_head = i32(r.heads);
    a.n_kv_head = i32(k.size(1));
    a.max_kv_seq = i32(args[4] == Py_None ? k.size(2) : integer(args[4]));
    a.head_dim = i32(r.d);
    a.q_stride[0] = r.stride_b;
    a.q_stride[1] = r.stride_h;
    strides3(a.k_stride, k);
    strides3(a.v_stride, v);
    a.scale = scale_of(args[5]);
    a.max_splits = i32(integer(args[7]));
    a.total_kv_len = 0;  // a shared length is known as it is; per-sequence lengths live on the device
    Tensor out, lse, ws;
    {
      NoGil no_gil;
      c10::cuda::OptionalCUDAGuard guard(q.device());
      out = new_tensor({r.batch, r.heads, r.d}, q.scalar_type(), q.device());
      lse = new_tensor({r.batch, r.heads}, at::kFloat, q.device());
      a.o = out.data_ptr();
      a.o_stride[0] = r.heads * r.d;
      a.o_stride[1] = r.d;
      a.lse = static_cast<float*>(lse.data_ptr());
      if (ws_in) {
        ws = *ws_in;
      } else {
        const size_t need = tyr_b200_attn_decode_workspace_bytes(a.batch, a.n_head, a.head_dim, a.max_kv_seq, a.max_splits);
        ws = new_tensor({(int64_t)(need > 16 ? need : 16)}, at::kByte, q.device());
      }
      a.workspace = ws.data_ptr();
      a.workspace_bytes = (size_t)ws.numel();
      check_rc(tyr_b200_attn_decode(&a, stream_of(q)));
    }
    return out_and_lse(out, lse, false);
  });
}

// x, out, norm_weight, cos, sin, positions, position0, eps, pe, out_at_row0 -> None
PyObject* qk_prologue(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    require_count(n, 10);
    const Tensor &x = tensor(args[0], "x"), &out = tensor(args[1], "out");
    require_cuda(x);
    require_cuda(out);
    if (x.dim() != 4 || out.dim() != 4 || x.scalar_type() != at::kBFloat16 || out.scalar_type() != at::kBFloat16)
      throw ValueError("x must be bf16 [B,S,H,D] and out bf16 [B,H,cap,D]");
    const int64_t B = x.size(0), S = x.size(1), H = x.size(2), D = x.size(3), cap = out.size(2);
    if (out.size(0) != B || out.size(1) != H || out.size(3) != D) throw ValueError("out does not match x");
    const Tensor *w = maybe(args[2], "norm_weight"), *cos = maybe(args[3], "cos"), *sin = maybe(args[4], "sin"),
                 *pos = maybe(args[5], "positions"), *pe = maybe(args[8], "pe");
    for (const Tensor* t : {w, cos, sin, pe})
      if (t && (t->scalar_type() != at::kFloat || !t->is_contiguous() || !t->is_cuda()))
        throw ValueError("norm_weight / cos / sin / pe must be contiguous float32 CUDA tensors");
    if (pe) {
      if (cos || sin) throw ValueError("pass either cos/sin or pe");
      if (pe->dim() != 5 || pe->size(2) != D / 2 || pe->size(3) != 2 || pe->size(4) != 2 ||
          (pe->size(0) != 1 && pe->size(0) != B))
        throw ValueError("pe must be [B or 1, max_pos, D/2, 2, 2]");
    }
    if (cos && (!sin || cos->sizes() != sin->sizes() || cos->dim() != 2 || cos->size(1) != D / 2))
      throw ValueError("cos and sin must both be [max_pos, D/2]");
    const int64_t max_pos = pe ? pe->size(1) : (cos ? cos->size(0) : 0);
    const int64_t position0 = integer(args[6]);
    const bool row0 = truth(args[9]);
    if (row0 && S > cap) throw ValueError(std::to_string(S) + " rows do not fit the " + std::to_string(cap) + " rows of out");
    if (!pos) {
      if (position0 < 0 || (!row0 && position0 + S > cap))
        throw ValueError("rows " + std::to_string(position0) + ".." + std::to_string(position0 + S - 1) + " do not fit the " +
                         std::to_string(cap) + " rows of out");
      if (max_pos && position0 + S > max_pos)
        throw ValueError("positions up to " + std::to_string(position0 + S - 1) + " exceed the " + std::to_string(max_pos) +
                         " rows of the rotary table");
    } else if (pos->scalar_type() != at::kInt || !pos->is_cuda()) {
      throw ValueError("positions must be an int32 CUDA tensor");
    }
    TyrAttnPrologueArgs a;
    std::memset(&a, 0, sizeof(a));
    auto f32 = [](const Tensor* t) { return t ? static_cast<const float*>(t->data_ptr()) : nullptr; };
    a.x = x.data_ptr();
    a.out = out.data_ptr();
    a.norm_weight = f32(w);
    a.cos = f32(cos);
    a.sin = f32(sin);
    a.pe = f32(pe);
    a.positions = pos ? static_cast<const int32_t*>(pos->data_ptr()) : nullptr;
    a.position0 = i32(position0);
    a.batch = i32(B);
    a.seq = i32(S);
    a.n_head = i32(H);
    a.head_dim = i32(D);
    strides3(a.x_stride, x);
    strides3(a.out_stride, out);
    const double eps = PyFloat_AsDouble(args[7]);
    if (eps == -1.0 && PyErr_Occurred()) throw python_error();
    a.eps = static_cast<float>(eps);
    a.cap = i32(cap);
    a.max_pos = i32(max_pos);
    a.out_at_row0 = row0;
    a.pe_batch_stride = (pe && pe->size(0) > 1) ? pe->stride(0) : 0;
    {
      NoGil no_gil;
      c10::cuda::OptionalCUDAGuard guard(x.device());
      check_rc(tyr_b200_attn_qk_prologue(&a, stream_of(x)));
    }
    Py_RETURN_NONE;
  });
}

PyObject* set_error(PyObject*, PyObject* cls) {
  Py_XINCREF(cls);
  Py_XSETREF(g_attn_error, cls);
  Py_RETURN_NONE;
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST(attention_fwd), FAST(attention_bwd), FAST(decode_ragged), FAST(decode_dense), FAST(qk_prologue),
                           {"set_error", set_error, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) { return PyModule_Create(&g_module); }
