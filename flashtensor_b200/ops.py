"""Operator layer: torch tensors in, C-ABI calls, torch tensors out.

Outputs are allocated with torch.empty on the inputs' device and the work is enqueued on torch's
current stream without synchronising -- the contract of the reference's generated callables
(lib/Translate/to_triton.cpp:579-609).  Shape/dtype problems raise (as the TensorRT back end's
closure does, python/asuka/backend/tensorrt/builder.py:104-111); nothing falls back to PyTorch.
"""
import contextlib
import ctypes

import torch

from . import _lib
from ._lib import AsukaError  # noqa: F401  (re-exported)

_DTYPES = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16, torch.float32: _lib.F32,
           torch.int32: _lib.I32, torch.uint8: _lib.U8, torch.bool: _lib.U8}


_native = None


def _bind():
  """The native front end (csrc/bind.cpp): descriptors, output allocation and the C-ABI call."""
  global _native
  if _native is None:
    _lib.load()
    try:
      from . import _bind as native
    except ImportError as e:
      raise ImportError(f"the native front end does not load ({e}): build it with `python -m flashtensor_b200.build` "
                        "(there is no Python fallback)") from e
    _native = native
  return _native


def _desc(t):
  """asuka_tensor descriptor of a torch tensor (None -> null descriptor)."""
  d = _lib.Tensor()
  if t is None:
    return d
  if t.dtype not in _DTYPES:
    raise TypeError(f"unsupported dtype {t.dtype}")
  if t.dim() > 5:
    raise ValueError("at most 5 dimensions")
  n = t.dim()
  d.ptr = t.data_ptr()
  d.dtype = _DTYPES[t.dtype]
  d.ndim = n
  d.shape[:n] = t.shape
  d.stride[:n] = t.stride()
  return d


_NO_SWITCH = contextlib.nullcontext()


def _on(dev):
  """Context that makes `dev` the current CUDA device (a no-op, and cheap, when it already is)."""
  return _NO_SWITCH if dev.index == torch.cuda.current_device() else torch.cuda.device(dev)


def _stream(t):
  if not t.is_cuda:
    raise RuntimeError("asuka_b200 kernels run on CUDA tensors only; there is no CPU path")
  return ctypes.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _as4d(t):
  """Accept the 2-D [S, H*D] layout of cases/attn.py as [1, S, H, 128] (same memory)."""
  if t.dim() == 2:
    return t.view(1, t.shape[0], t.shape[1] // 128, 128)
  return t


def _same_device(*ts):
  dev = ts[0].device
  for t in ts:
    if t is None:
      continue
    if not t.is_cuda:
      raise RuntimeError("asuka_b200 kernels run on CUDA tensors only; there is no CPU path")
    if t.device != dev:
      raise RuntimeError("all tensors must be on the same device")


def attn_fwd(q, k, v, causal=True, softmax_scale=0.0, return_lse=False, out=None, softcap=0.0):
  """out = softmax(q k^T * scale (+ causal mask)) v.  q: [B,Sq,H,128]; k, v: [B,Skv,H,128].
  softcap > 0 applies cap * tanh(logits / cap) before the mask (cases/kernels/gemma2.py:30-33)."""
  return _bind().attn_fwd(q, k, v, causal, softmax_scale, return_lse, out, softcap)


def col_scores(q, k, lse, mode=_lib.SCORE_SUM, causal=True, softmax_scale=0.0, exp_rand=None,
               tau=1.0, seed=0, corm_mask=None, unit_offset=0):
  """Per-key reductions over the query rows of the attention probabilities: [B,H,Skv] f32 sums
  (and sums of squares in mode SCORE_SUM_SQ); in mode SCORE_CORM a bool tensor that is True where
  some probability reaches its threshold in `corm_mask` [Sq, Skv]."""
  score, score_sq = _bind().col_scores(q, k, lse, mode, causal, softmax_scale, exp_rand, tau, seed, corm_mask,
                                       unit_offset)
  return score if score_sq is None else (score, score_sq)


def keyformer_rowstat(q, k, causal=True, softmax_scale=0.0, exp_rand=None, tau=1.5, seed=0, unit_offset=0):
  """Base-2 log-sum-exp per query row of the perturbed logits (s + g) / tau: [B,H,Sq] f32."""
  lib = _lib.load()
  q4, k4 = _as4d(q), _as4d(k)
  _same_device(q4, k4, exp_rand)
  with _on(q4.device):
    lse = torch.empty((q4.shape[0], q4.shape[2], q4.shape[1]), dtype=torch.float32, device=q4.device)
    p = _lib.ScoreParams(_desc(q4), _desc(k4), _desc(lse), _lib.Tensor(), _lib.Tensor(),
                         _desc(exp_rand), float(softmax_scale), float(tau), int(seed),
                         int(bool(causal)), _lib.SCORE_PERTURBED, _lib.Tensor(), None, 0, int(unit_offset))
    _lib.check("asuka_b200_keyformer_rowstat",
               lib.asuka_b200_keyformer_rowstat(ctypes.byref(p), _stream(q4)))
  return lse


def select_topk(score, k_keep, mode=_lib.SELECT_TOPK, recent=0, score_sq=None, q_len=0, causal=True,
                return_stats=False):
  """Kept key indices, ascending int32 [B,H,k_keep(+recent)].  Mode SELECT_ROCO ranks by the
  per-key mean (then standard deviation) of the probabilities over the rows that attend to the
  key -- all `q_len` rows when `causal` is False -- and with `return_stats` also returns
  (mean, std), both [B,H,S] f32."""
  _same_device(score, score_sq)
  n_out = k_keep + (recent if mode == _lib.SELECT_TOPK_RECENT else 0)
  stats = return_stats and mode == _lib.SELECT_ROCO
  mean = torch.empty_like(score) if stats else None
  std = torch.empty_like(score) if stats else None
  idx = _bind().select_topk(score, score_sq, k_keep, mode, recent, n_out, q_len, not causal, mean, std)
  return (idx, mean, std) if stats else idx


def pool_scores(score, kernel_size):
  """SnapKV smoothing: avg_pool1d(score, kernel_size, padding=kernel_size // 2, stride=1) over keys."""
  return _bind().pool_scores(score, kernel_size)


def gather_kv(k, v, idx):
  """Compact the KV cache to the kept keys: (k[b, idx[b,h,n], h, :], v alike) as [B, n, H, 128]."""
  return _bind().gather_kv(k, v, idx)


def sima_fwd(q, k, v, out_dtype=None):
  """SimA: out = L1norm_seq(q) (L1norm_seq(k)^T v), [B,S,H,128]."""
  return _linear(q, k, v, out_dtype, False)


def ea_fwd(q, k, v, out_dtype=None):
  """EA (bench/ea.mlir:13-17): out = softmax_features(q) (softmax_seq(k)^T v), [B,S,H,128]."""
  return _linear(q, k, v, out_dtype, True)


def _linear(q, k, v, out_dtype, ea):
  out = None
  if out_dtype is not None and out_dtype != q.dtype:
    out = torch.empty(_as4d(q).shape, dtype=out_dtype, device=q.device)
  return _bind().linear_fwd(q, k, v, out, ea)


def linattn32_fwd(q, k, v, ea=False, out=None):
  """SimA (ea=False) or EA (ea=True) attention core at head_dim 32 in f32 (bench/sima.mlir:13-17,
  bench/ea.mlir:13-17).  q, k, v: [B, N, H, 32] f32, possibly strided views of a fused QKV tensor."""
  return _bind().linattn32_fwd(q, k, v, ea, out)


def linear_f32(x, w, bias):
  """x w^T + bias with f32 accuracy on the tensor pipe: x [M, K], w [N, K], bias [N] -> [M, N], f32,
  contiguous, K a multiple of 8 and at most LINEAR_MAX_K."""
  return _bind().linear(x, w, bias)


LINEAR_MAX_K = 128


def linattn_block(x, w_qkv, b_qkv, w_o, b_o, ea=False):
  """The whole block of bench/sima.mlir (ea=False) or bench/ea.mlir (ea=True), f32: QKV projection,
  core, output projection in three launches.  x [B, N, C], C a multiple of 32 and at most LINEAR_MAX_K.
  The result has no graph, whatever the operands require (``blocks`` takes another way then)."""
  return _bind().linattn_block(x, w_qkv, b_qkv, w_o, b_o, ea)


_H2O, _ROCO, _KEYFORMER = 0, 1, 2   # case kinds of the native front end


def _case(kind, q, k, v, causal, softmax_scale, exp_rand=None, tau=1.0, seed=0, k_keep=0, recent=0, n_idx=0,
          workspace=None, out=None, score=None, score_sq=None, idx=None, roco_mean=None, roco_std=None,
          unit_offset=0):
  return _bind().run_case(kind, q, k, v, causal, softmax_scale, exp_rand, tau, seed, k_keep, recent, n_idx, workspace,
                          out, score, score_sq, idx, roco_mean, roco_std, unit_offset)


def h2o(q, k, v, causal=True, softmax_scale=0.0, k_keep=0, recent=0, **buffers):
  """(out, h2o_score[, idx]) -- cases/kernels/h2o.py:18-38 plus the optional keep set."""
  n_idx = k_keep + recent if k_keep > 0 else 0
  out, score, _, idx, _, _ = _case(_H2O, q, k, v, causal, softmax_scale, k_keep=k_keep,
                             recent=recent, n_idx=n_idx, **buffers)
  return (out, score, idx) if n_idx else (out, score)


def h2o_static(q, k, v, out, score, idx=None, causal=True, softmax_scale=0.0, k_keep=0, recent=0):
  """H2O through the entry point that allocates nothing: the caller supplies every output
  (`out`, `score`, optionally `idx`), and the scratch between the two kernels is the library's
  fixed device array.  For hosts that may not allocate on the call path (engine plug-ins, fully
  pre-reserved memory pools); limited to B*H*Sq <= 524288 rows, and calls on one device must not
  overlap.  This wrapper itself creates no tensors."""
  lib = _lib.load()
  q4, k4, v4 = _as4d(q), _as4d(k), _as4d(v)
  _same_device(q4, k4, v4, out, score, idx)
  with _on(q4.device):
    p = _lib.CaseParams(_desc(q4), _desc(k4), _desc(v4), _desc(_as4d(out)), _desc(score),
                        _lib.Tensor(), _lib.Tensor(), _desc(idx), float(softmax_scale), 1.0, 0,
                        int(bool(causal)), int(k_keep), int(recent), _lib.Tensor(), _lib.Tensor(), 0)
    _lib.check("asuka_b200_h2o_static", lib.asuka_b200_h2o_static(ctypes.byref(p), _stream(q4)))
  return (out, score, idx) if idx is not None else (out, score)


def roco(q, k, v, causal=True, softmax_scale=0.0, k_keep=0, return_stats=False, **buffers):
  """(out, roco_score, roco_sq_score[, idx[, mean, std]]) -- cases/kernels/roco.py:18-48; with a
  selection (`k_keep` > 0) and `return_stats`, also the per-key mean and standard deviation of the
  probabilities the selection ranks by, [B,H,Skv] f32."""
  stats = return_stats and k_keep > 0
  if stats:
    buffers.setdefault("roco_mean", True)
    buffers.setdefault("roco_std", True)
  out, score, sq, idx, mean, std = _case(_ROCO, q, k, v, causal, softmax_scale, k_keep=k_keep, n_idx=k_keep, **buffers)
  if stats:
    return out, score, sq, idx, mean, std
  return (out, score, sq, idx) if k_keep else (out, score, sq)


def keyformer(q, k, v, exp_rand=None, tau=1.5, seed=0, causal=True, softmax_scale=0.0, k_keep=0,
              **buffers):
  """(out, kf_score[, idx]) -- cases/kernels/kf.py:19-42; exp_rand=None uses the seeded noise
  (`unit_offset`: index of this call's first (batch, head) unit when it is a slice of a larger
  problem, so that the slice gets the noise the whole problem would have had)."""
  out, score, _, idx, _, _ = _case(_KEYFORMER, q, k, v, causal, softmax_scale,
                             exp_rand=exp_rand, tau=tau, seed=seed, k_keep=k_keep, n_idx=k_keep,
                             **buffers)
  return (out, score, idx) if k_keep else (out, score)


def device_status():
  """(count, last_site) of expired device-side waits since the last read; raises if non-zero."""
  lib = _lib.load()
  w = (ctypes.c_uint32 * 2)()
  st = lib.asuka_b200_device_status(w)
  _lib.check("asuka_b200_device_status", st)
  return int(w[0]), int(w[1])


def launch_count():
  return int(_lib.load().asuka_b200_launch_count())
