// Native front end of the Python operator layer: torch tensors in, one C-ABI call, torch tensors out.
//
// A call of the small cases is bound by the host, not by the device: with ctypes descriptors,
// torch.empty and the stream looked up in Python, plain attention took the host 25 us and H2O with
// its selection 39-43 us a call (128 rows, 2 heads, calls back to back).  Here the descriptors are
// filled from the tensor objects directly and the outputs come straight from the caching
// allocator: 7.7 and 13-15 us, most of it the launches themselves.  Nothing is cached between calls.  The interpreter lock is released around the C-ABI call, as ctypes does.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <initializer_list>
#include <optional>

#include "../../include/asuka_b200.h"

namespace {

PyObject* g_check = nullptr;  // flashtensor_b200._lib.check: raises AsukaError

// ---- arguments ---------------------------------------------------------------------------------
struct BadArg {};  // a Python exception has been set

const at::Tensor& tensor_arg(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "expected a torch.Tensor, got %s", Py_TYPE(o)->tp_name);
    throw BadArg();
  }
  return THPVariable_Unpack(o);
}
at::Tensor optional_tensor(PyObject* o) { return o == Py_None ? at::Tensor() : tensor_arg(o); }
bool bool_arg(PyObject* o) {
  const int r = PyObject_IsTrue(o);
  if (r < 0) throw BadArg();
  return r != 0;
}
double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw BadArg();
  return v;
}
// like int(o) stored into a C integer of fewer bits
uint64_t int_arg(PyObject* o) {
  PyObject* n = PyLong_Check(o) ? (Py_INCREF(o), o) : PyNumber_Long(o);
  if (n == nullptr) throw BadArg();
  const uint64_t v = PyLong_AsUnsignedLongLongMask(n);
  Py_DECREF(n);
  if (PyErr_Occurred()) throw BadArg();
  return v;
}
void want_args(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    throw BadArg();
  }
}

// ---- descriptors and outputs ---------------------------------------------------------------------
asuka_tensor desc(const at::Tensor& t) {
  asuka_tensor d;
  std::memset(&d, 0, sizeof(d));
  if (!t.defined()) return d;
  switch (t.scalar_type()) {
    case at::kHalf: d.dtype = ASUKA_F16; break;
    case at::kBFloat16: d.dtype = ASUKA_BF16; break;
    case at::kFloat: d.dtype = ASUKA_F32; break;
    case at::kInt: d.dtype = ASUKA_I32; break;
    case at::kByte:
    case at::kBool: d.dtype = ASUKA_U8; break;
    default:
      PyErr_Format(PyExc_TypeError, "unsupported dtype %s", c10::toString(t.scalar_type()));
      throw BadArg();
  }
  const auto sizes = t.sizes();
  const auto strides = t.strides();
  if (sizes.size() > 5) {
    PyErr_SetString(PyExc_ValueError, "at most 5 dimensions");
    throw BadArg();
  }
  d.ptr = t.data_ptr();
  d.ndim = static_cast<int32_t>(sizes.size());
  for (size_t i = 0; i < sizes.size(); ++i) {
    d.shape[i] = sizes[i];
    d.stride[i] = strides[i];
  }
  return d;
}

// the 2-D [S, H*128] layout of cases/attn.py as [1, S, H, 128] (same memory)
at::Tensor as4d(const at::Tensor& t) {
  if (t.defined() && t.dim() == 2) return t.view({1, t.size(0), t.size(1) / 128, 128});
  return t;
}

at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, const at::Tensor& like) {
  return at::detail::empty_cuda(shape, dtype, like.device(), std::nullopt);
}

// All tensors on one CUDA device, which becomes current for the call if it is not already.
struct OnDevice {
  c10::cuda::OptionalCUDAGuard guard;
  asuka_stream stream;
  explicit OnDevice(std::initializer_list<const at::Tensor*> ts) {
    const at::Tensor& first = **ts.begin();
    for (const at::Tensor* t : ts) {
      if (!t->defined()) continue;
      if (!t->is_cuda()) {
        PyErr_SetString(PyExc_RuntimeError, "asuka_b200 kernels run on CUDA tensors only; there is no CPU path");
        throw BadArg();
      }
      if (t->device() != first.device()) {
        PyErr_SetString(PyExc_RuntimeError, "all tensors must be on the same device");
        throw BadArg();
      }
    }
    if (c10::cuda::current_device() != first.get_device()) guard.set_index(first.get_device());
    stream = c10::cuda::getCurrentCUDAStream(first.get_device()).stream();
  }
};

// Runs a C-ABI call without the interpreter lock; a non-zero status raises AsukaError(name).
template <typename F>
void call(const char* name, F&& f) {
  int status;
  PyThreadState* save = PyEval_SaveThread();
  status = f();
  PyEval_RestoreThread(save);
  if (status != ASUKA_OK) {
    PyObject* r = PyObject_CallFunction(g_check, "si", name, status);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed: %d", name, status);
    throw BadArg();
  }
}
// (workspace queries only compute)
void query(const char* name, int status) {
  if (status != ASUKA_OK) call(name, [status] { return status; });
}

PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
PyObject* none_or(const at::Tensor& t) {
  if (t.defined()) return wrap(t);
  Py_RETURN_NONE;
}
PyObject* tuple(std::initializer_list<PyObject*> items) {
  PyObject* r = PyTuple_New(static_cast<Py_ssize_t>(items.size()));
  Py_ssize_t i = 0;
  for (PyObject* o : items) PyTuple_SET_ITEM(r, i++, o);
  return r;
}

// ---- entry points --------------------------------------------------------------------------------
// (q, k, v, causal, softmax_scale, return_lse, out, softcap) -> out | (out, lse)
PyObject* attn_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 8);
    const at::Tensor& q0 = tensor_arg(a[0]);
    const at::Tensor q = as4d(q0), k = as4d(tensor_arg(a[1])), v = as4d(tensor_arg(a[2]));
    at::Tensor out = optional_tensor(a[6]), lse;
    OnDevice on({&q, &k, &v, &out});
    if (!out.defined()) out = empty(q.sizes(), q.scalar_type(), q);
    const bool want_lse = bool_arg(a[5]);
    if (want_lse) lse = empty({q.size(0), q.size(2), q.size(1)}, at::kFloat, q);
    asuka_attn_params p;
    std::memset(&p, 0, sizeof(p));
    p.q = desc(q);
    p.k = desc(k);
    p.v = desc(v);
    p.out = desc(as4d(out));
    p.lse = desc(lse);
    p.softmax_scale = static_cast<float>(float_arg(a[4]));
    p.causal = bool_arg(a[3]) ? 1 : 0;
    p.softcap = static_cast<float>(float_arg(a[7]));
    size_t nbytes = 0;
    query("asuka_b200_attn_workspace_bytes", asuka_b200_attn_workspace_bytes(&p, &nbytes));
    at::Tensor ws;
    if (nbytes > 0) {
      ws = empty({static_cast<int64_t>(nbytes)}, at::kByte, q);
      p.workspace = ws.data_ptr();
      p.workspace_bytes = nbytes;
    }
    call("asuka_b200_attn_fwd", [&] { return asuka_b200_attn_fwd(&p, on.stream); });
    if (q0.dim() == 2) out = out.view(q0.sizes());
    return want_lse ? tuple({wrap(out), wrap(lse)}) : wrap(out);
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (kind, q, k, v, causal, softmax_scale, exp_rand, tau, seed, k_keep, recent, n_idx, workspace,
//  out, score, score_sq, idx, roco_mean, roco_std, unit_offset)
//   -> (out, score, score_sq, idx, roco_mean, roco_std)
// kind: 0 H2O, 1 RoCo, 2 Keyformer; roco_mean / roco_std: a tensor, None, or True to allocate it
PyObject* run_case(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 20);
    const int kind = static_cast<int>(int_arg(a[0]));
    const at::Tensor& q0 = tensor_arg(a[1]);
    const at::Tensor q = as4d(q0), k = as4d(tensor_arg(a[2])), v = as4d(tensor_arg(a[3]));
    const at::Tensor exp_rand = optional_tensor(a[6]);
    const int64_t n_idx = static_cast<int64_t>(int_arg(a[11]));
    at::Tensor ws = optional_tensor(a[12]), out = optional_tensor(a[13]), score = optional_tensor(a[14]),
               score_sq = optional_tensor(a[15]), idx = optional_tensor(a[16]), stats[2];
    for (int i = 0; i < 2; ++i)
      if (a[17 + i] != Py_True) stats[i] = optional_tensor(a[17 + i]);
    OnDevice on({&q, &k, &v, &exp_rand, &ws, &out, &score, &score_sq, &idx, &stats[0], &stats[1]});
    // scores and indices are per key/value head (with grouped-query attention: the group mean)
    const int64_t B = k.size(0), Skv = k.size(1), H = k.size(2);
    if (!out.defined()) out = empty(q.sizes(), q.scalar_type(), q);
    if (!score.defined()) score = empty({B, H, Skv}, at::kFloat, q);
    if (kind == 1 && !score_sq.defined()) score_sq = empty(score.sizes(), at::kFloat, q);
    if (n_idx > 0 && !idx.defined()) idx = empty({B, H, n_idx}, at::kInt, q);
    asuka_case_params p;
    std::memset(&p, 0, sizeof(p));
    p.q = desc(q);
    p.k = desc(k);
    p.v = desc(v);
    p.out = desc(as4d(out));
    p.score = desc(score);
    p.score_sq = desc(score_sq);
    p.exp_rand = desc(exp_rand);
    p.idx = desc(idx);
    p.softmax_scale = static_cast<float>(float_arg(a[5]));
    p.tau = static_cast<float>(float_arg(a[7]));
    p.seed = int_arg(a[8]);
    p.causal = bool_arg(a[4]) ? 1 : 0;
    p.k_keep = static_cast<int32_t>(int_arg(a[9]));
    p.recent = static_cast<int32_t>(int_arg(a[10]));
    for (int i = 0; i < 2; ++i)
      if (a[17 + i] == Py_True) stats[i] = empty({B, q.size(2), Skv}, at::kFloat, q);
    p.roco_mean = desc(stats[0]);
    p.roco_std = desc(stats[1]);
    p.seed_unit_offset = static_cast<uint32_t>(int_arg(a[19]));
    if (!ws.defined()) {
      size_t nbytes = 0;
      query("asuka_b200_case_workspace_bytes_split", asuka_b200_case_workspace_bytes_split(&p, &nbytes));
      ws = empty({static_cast<int64_t>(nbytes < 16 ? 16 : nbytes)}, at::kByte, q);
    }
    void* wp = ws.data_ptr();
    const size_t wn = static_cast<size_t>(ws.numel());
    const char* const names[3] = {"asuka_b200_h2o", "asuka_b200_roco", "asuka_b200_keyformer"};
    int (*const entries[3])(const asuka_case_params*, void*, size_t, asuka_stream) = {
        asuka_b200_h2o, asuka_b200_roco, asuka_b200_keyformer};
    if (kind < 0 || kind > 2) {
      PyErr_SetString(PyExc_ValueError, "unknown case");
      throw BadArg();
    }
    call(names[kind], [&] { return entries[kind](&p, wp, wn, on.stream); });
    if (q0.dim() == 2) {
      // the 2-D scripts return out [q_len, H*128] and per-key tensors [Hkv, kv_len] (cases/attn_h2o.py:47)
      out = out.view(q0.sizes());
      for (at::Tensor* t : {&score, &score_sq, &idx})
        if (t->defined()) *t = t->select(0, 0);
    }
    return tuple({wrap(out), wrap(score), none_or(score_sq), none_or(idx), none_or(stats[0]), none_or(stats[1])});
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (q, k, v, out (None: allocated, of q's type), ea) -> out
PyObject* linear_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 5);
    const at::Tensor& q0 = tensor_arg(a[0]);
    const at::Tensor q = as4d(q0), k = as4d(tensor_arg(a[1])), v = as4d(tensor_arg(a[2]));
    at::Tensor out = optional_tensor(a[3]);
    OnDevice on({&q, &k, &v, &out});
    const bool ea = bool_arg(a[4]);
    if (!out.defined()) out = empty(q.sizes(), q.scalar_type(), q);
    asuka_sima_params p;
    p.q = desc(q);
    p.k = desc(k);
    p.v = desc(v);
    p.out = desc(out);
    size_t nbytes = 0;
    query("asuka_b200_sima_workspace_bytes", asuka_b200_sima_workspace_bytes(&p, &nbytes));
    const at::Tensor ws = empty({static_cast<int64_t>(nbytes < 16 ? 16 : nbytes)}, at::kByte, q);
    void* wp = ws.data_ptr();
    const size_t wn = static_cast<size_t>(ws.numel());
    if (ea)
      call("asuka_b200_ea_fwd", [&] { return asuka_b200_ea_fwd(&p, wp, wn, on.stream); });
    else
      call("asuka_b200_sima_fwd", [&] { return asuka_b200_sima_fwd(&p, wp, wn, on.stream); });
    if (q0.dim() == 2) out = out.view(q0.sizes());
    return wrap(out);
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (q, k, v, ea, out) -> out
PyObject* linattn32_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 5);
    const at::Tensor &q = tensor_arg(a[0]), &k = tensor_arg(a[1]), &v = tensor_arg(a[2]);
    at::Tensor out = optional_tensor(a[4]);
    OnDevice on({&q, &k, &v, &out});
    if (!out.defined()) out = empty(q.sizes(), at::kFloat, q);
    asuka_linattn32_params p;
    p.q = desc(q);
    p.k = desc(k);
    p.v = desc(v);
    p.out = desc(out);
    p.ea = bool_arg(a[3]) ? 1 : 0;
    call("asuka_b200_linattn32_fwd", [&] { return asuka_b200_linattn32_fwd(&p, on.stream); });
    return wrap(out);
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// x w^T + bias into a new [M, N] tensor
at::Tensor linear_f32(const at::Tensor& x, const at::Tensor& w, const at::Tensor& bias, asuka_stream stream) {
  const at::Tensor out = empty({x.size(0), w.size(0)}, at::kFloat, x);
  asuka_linear_params p;
  p.x = desc(x);
  p.w = desc(w);
  p.bias = desc(bias);
  p.out = desc(out);
  call("asuka_b200_linear_f32", [&] { return asuka_b200_linear_f32(&p, stream); });
  return out;
}

// `t` as the kernels read it: contiguous from a 16-byte boundary on.  A copy where it is not (a slice of a
// flat parameter buffer may start anywhere); the caching allocator's blocks start on such a boundary.
at::Tensor dense(const at::Tensor& t) {
  const at::Tensor c = t.contiguous().resolve_neg();
  return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15u) == 0 ? c : c.clone(at::MemoryFormat::Contiguous);
}

// (x [M, K], w [N, K], bias [N]) -> out [M, N]
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 3);
    const at::Tensor &x = tensor_arg(a[0]), &w = tensor_arg(a[1]), &bias = tensor_arg(a[2]);
    OnDevice on({&x, &w, &bias});
    return wrap(linear_f32(x, w, bias, on.stream));
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// From how many rows of a batch on its core is folded into the output projection.  Folding spares the core a pass over
// the queries and its output, which grow with the rows; it costs C x C weights for every batch, written, read and split
// by a CTA of the projection that has nothing but that batch's rows, and scratch of that size.  Folded / not, us, SimA at
// C 128 (B 512 N 16 takes 93 / 56, B 4096 N 49 777 / 406):
//   N      100        128        160        192        224        256        320        400        500
//   B 2    22.0/22.1  22.1/22.4  24.2/23.8  24.2/23.9  24.7/25.1  24.8/25.2  24.9/26.7  26.0/29.3  26.2/30.7
//   16     25.3/23.1  25.9/23.2  26.7/24.9  27.0/26.3  28.0/28.1  31.7/32.7  32.2/34.4  35.1/40.9  37.1/44.2
//   64     32.4/31.3  32.5/32.3  33.7/34.9  34.4/34.1  37.3/38.8  38.2/39.1  45.3/47.3  48.8/55.4  53.5/61.9
//   148    42.2/42.3  47.7/43.5  50.0/51.4  53.5/55.6  59.0/64.2  61.5/67.6  70.2/76.6  92.2/96.3  99.8/116
//   512    135/105    154/114    168/140    185/151    200/175    206/190    242/224    284/278    328/339
// (EA: B 16 N 192 28.8/27.4, N 256 33.2/35.4, B 512 N 256 219/213, N 400 294/318.  C 64: B 64 N 128 22.0/22.1, N 256
// 27.0/28.0, B 512 N 256 108/105.)  Above the line the scratch is smaller than the output of the core that the other way
// needs.
int64_t fold_from(int64_t B) {
  return B <= at::cuda::getCurrentDeviceProperties()->multiProcessorCount ? 224 : 384;
}

// The whole block of bench/sima.mlir / bench/ea.mlir: (x [B, N, C], w_qkv, b_qkv, w_o, b_o, ea) -> [B, N, C];
// the core reads q, k, v as strided views of the projection's output [B*N, 3, C/32, 32].
PyObject* linattn_block(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 6);
    const at::Tensor x = dense(tensor_arg(a[0])), w_qkv = dense(tensor_arg(a[1])), b_qkv = dense(tensor_arg(a[2])),
                     w_o = dense(tensor_arg(a[3])), b_o = dense(tensor_arg(a[4]));
    // (the core's views of the projection below take its rows to be 3 C long)
    const int64_t C = x.dim() == 3 ? x.size(2) : -1;
    if (C < 0 || C % 32 != 0 || !w_qkv.sizes().equals({3 * C, C}) || !b_qkv.sizes().equals({3 * C}) ||
        !w_o.sizes().equals({C, C}) || !b_o.sizes().equals({C})) {
      PyErr_SetString(PyExc_RuntimeError,
                      "expected x [B, N, C], w_qkv [3C, C], b_qkv [3C], w_o [C, C], b_o [C] with C a multiple of 32");
      throw BadArg();
    }
    OnDevice on({&x, &w_qkv, &b_qkv, &w_o, &b_o});
    const int64_t B = x.size(0), N = x.size(1);
    const at::Tensor qkv = linear_f32(x.view({B * N, C}), w_qkv, b_qkv, on.stream);
    asuka_linattn32_proj_params p;
    p.q = desc(qkv);  // [B, N, C / 32, 32], strided over the fused rows
    p.q.ndim = 4;
    p.q.shape[0] = B; p.q.shape[1] = N; p.q.shape[2] = C / 32; p.q.shape[3] = 32;
    p.q.stride[0] = N * 3 * C; p.q.stride[1] = 3 * C; p.q.stride[2] = 32; p.q.stride[3] = 1;
    p.k = p.q;
    p.k.ptr = static_cast<float*>(p.q.ptr) + C;
    p.v = p.q;
    p.v.ptr = static_cast<float*>(p.q.ptr) + 2 * C;
    p.ea = bool_arg(a[5]) ? 1 : 0;
    if (N < fold_from(B)) {
      const at::Tensor core = empty({B, N, C / 32, 32}, at::kFloat, x);
      asuka_linattn32_params c;
      c.q = p.q;
      c.k = p.k;
      c.v = p.v;
      c.out = desc(core);
      c.ea = p.ea;
      call("asuka_b200_linattn32_fwd", [&] { return asuka_b200_linattn32_fwd(&c, on.stream); });
      return wrap(linear_f32(core.view({B * N, C}), w_o, b_o, on.stream).view({B, N, C}));
    }
    const at::Tensor out = empty({B, N, C}, at::kFloat, x), scratch = empty({B, C + 1, C}, at::kFloat, x);
    p.w = desc(w_o);
    p.bias = desc(b_o);
    p.out = desc(out);
    p.scratch = desc(scratch);
    call("asuka_b200_linattn32_proj", [&] { return asuka_b200_linattn32_proj(&p, on.stream); });
    return wrap(out);
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (score, kernel_size) -> pooled score
PyObject* pool_scores(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 2);
    const at::Tensor& score = tensor_arg(a[0]);
    OnDevice on({&score});
    const int32_t ks = static_cast<int32_t>(int_arg(a[1]));
    const at::Tensor out = empty(score.sizes(), score.scalar_type(), score);
    const asuka_tensor s = desc(score), o = desc(out);
    call("asuka_b200_pool_scores", [&] { return asuka_b200_pool_scores(&s, &o, ks, on.stream); });
    return wrap(out);
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (k, v, idx) -> (k rows, v rows)
PyObject* gather_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 3);
    const at::Tensor &k = tensor_arg(a[0]), &v = tensor_arg(a[1]), &idx = tensor_arg(a[2]);
    OnDevice on({&k, &v, &idx});
    const at::Tensor ko = empty({k.size(0), idx.size(2), k.size(2), k.size(3)}, k.scalar_type(), k);
    const at::Tensor vo = empty(ko.sizes(), k.scalar_type(), k);
    asuka_gather_params p;
    p.k = desc(k);
    p.v = desc(v);
    p.idx = desc(idx);
    p.k_out = desc(ko);
    p.v_out = desc(vo);
    call("asuka_b200_gather_kv", [&] { return asuka_b200_gather_kv(&p, on.stream); });
    return tuple({wrap(ko), wrap(vo)});
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (q, k, lse, mode, causal, softmax_scale, exp_rand, tau, seed, corm_mask, unit_offset) -> (score, score_sq)
PyObject* col_scores(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 11);
    const at::Tensor q = as4d(tensor_arg(a[0])), k = as4d(tensor_arg(a[1]));
    const at::Tensor lse = optional_tensor(a[2]), exp_rand = optional_tensor(a[6]), corm_mask = optional_tensor(a[9]);
    OnDevice on({&q, &k, &lse, &exp_rand, &corm_mask});
    const int mode = static_cast<int>(int_arg(a[3]));
    const at::Tensor score = empty({k.size(0), k.size(2), k.size(1)}, mode == ASUKA_SCORE_CORM ? at::kBool : at::kFloat, q);
    at::Tensor score_sq;
    if (mode == ASUKA_SCORE_SUM_SQ) score_sq = empty(score.sizes(), score.scalar_type(), q);
    asuka_score_params p;
    std::memset(&p, 0, sizeof(p));
    p.q = desc(q);
    p.k = desc(k);
    p.lse = desc(lse);
    p.score = desc(score);
    p.score_sq = desc(score_sq);
    p.exp_rand = desc(exp_rand);
    p.softmax_scale = static_cast<float>(float_arg(a[5]));
    p.tau = static_cast<float>(float_arg(a[7]));
    p.seed = int_arg(a[8]);
    p.causal = bool_arg(a[4]) ? 1 : 0;
    p.mode = mode;
    p.corm_mask = desc(corm_mask);
    p.seed_unit_offset = static_cast<uint32_t>(int_arg(a[10]));
    size_t nbytes = 0;
    query("asuka_b200_col_scores_workspace_bytes", asuka_b200_col_scores_workspace_bytes(&p, &nbytes));
    at::Tensor ws;
    if (nbytes > 0) {
      ws = empty({static_cast<int64_t>(nbytes)}, at::kByte, q);
      p.workspace = ws.data_ptr();
      p.workspace_bytes = nbytes;
    }
    call("asuka_b200_col_scores", [&] { return asuka_b200_col_scores(&p, on.stream); });
    return tuple({wrap(score), none_or(score_sq)});
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// (score, score_sq, k_keep, mode, recent, n_out, q_len, all_rows, mean, std) -> idx
PyObject* select_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    want_args(n, 10);
    const at::Tensor& score = tensor_arg(a[0]);
    const at::Tensor score_sq = optional_tensor(a[1]), mean = optional_tensor(a[8]), std = optional_tensor(a[9]);
    OnDevice on({&score, &score_sq, &mean, &std});
    const at::Tensor idx = empty({score.size(0), score.size(1), static_cast<int64_t>(int_arg(a[5]))}, at::kInt, score);
    asuka_select_params p;
    std::memset(&p, 0, sizeof(p));
    p.score = desc(score);
    p.score_sq = desc(score_sq);
    p.idx = desc(idx);
    p.k_keep = static_cast<int32_t>(int_arg(a[2]));
    p.recent = static_cast<int32_t>(int_arg(a[4]));
    p.q_len = static_cast<int32_t>(int_arg(a[6]));
    p.mode = static_cast<int32_t>(int_arg(a[3]));
    p.all_rows = bool_arg(a[7]) ? 1 : 0;
    p.mean = desc(mean);
    p.std = desc(std);
    call("asuka_b200_select_topk", [&] { return asuka_b200_select_topk(&p, on.stream); });
    return wrap(idx);
  } catch (const BadArg&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define ENTRY(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {ENTRY(attn_fwd),    ENTRY(run_case),  ENTRY(linear_fwd), ENTRY(linattn32_fwd),
                           ENTRY(pool_scores), ENTRY(gather_kv), ENTRY(col_scores), ENTRY(select_topk),
                           ENTRY(linear),      ENTRY(linattn_block),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_bind", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__bind(void) {
  PyObject* lib = PyImport_ImportModule("flashtensor_b200._lib");
  if (lib == nullptr) return nullptr;
  g_check = PyObject_GetAttrString(lib, "check");
  Py_DECREF(lib);
  if (g_check == nullptr) return nullptr;
  return PyModule_Create(&g_module);
}
