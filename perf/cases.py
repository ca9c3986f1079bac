"""The work this library is measured on: one pass each of the fused attention programs, called the
way a user's program calls them (the per-case classes and blocks), over the range of sizes, data
types and options they are used with.

Sizes are the benchmark's own configurations (C1-C5), the shapes of bench/*.mlir, the smoke check's
call, and generic serving shapes beside them (a decode step over a long cache, a chunk of a prefill
over a ragged cache, odd sequence lengths).  head_dim is 128 except for the whole blocks (32).
"""
import math

import torch

import flashtensor_b200 as ft
from flashtensor_b200.blocks import EABlock, SimABlock

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def listed():
  return [
      # plain causal attention, one short prompt: the benchmark's smallest configuration (C1)
      {"name": "attn_prefill_1k", "kind": "attn", "dtype": "f16", "B": 1, "H": 32, "Hkv": 32, "Sq": 1024, "Skv": 1024,
       "causal": True},
      # one decode step of a batch with grouped key/value heads over caches of an odd length
      {"name": "attn_decode_gqa", "kind": "attn", "dtype": "bf16", "B": 16, "H": 32, "Hkv": 8, "Sq": 1, "Skv": 4001,
       "causal": True},
      # the smoke check's call, the smallest with every step of H2O in it: latency and launches
      {"name": "h2o_select_small", "kind": "h2o_select", "dtype": "f16", "B": 1, "H": 4, "Sq": 512, "Skv": 512, "keep": 64,
       "recent": 32},
      # the headline configuration (C2): H2O prefill with the heavy-hitter selection
      {"name": "h2o_select_4k", "kind": "h2o_select", "dtype": "f16", "B": 1, "H": 32, "Sq": 4096, "Skv": 4096, "keep": 512,
       "recent": 256},
      # chunked prefill: a block of new queries over a long ragged cache with grouped key/value heads
      {"name": "h2o_chunk_gqa", "kind": "h2o", "dtype": "bf16", "B": 1, "H": 32, "Hkv": 8, "Sq": 500, "Skv": 5003},
      # soft-capped logits, grouped heads, a long prompt
      {"name": "gemma2_8k_gqa", "kind": "gemma2", "dtype": "bf16", "B": 1, "H": 16, "Hkv": 8, "Sq": 8192, "Skv": 8192},
      # Keyformer with the noise as an operand, as the reference's case has it (C3): the most bytes
      {"name": "keyformer_noise_2k", "kind": "keyformer", "dtype": "f16", "B": 4, "H": 32, "Sq": 2048, "Skv": 2048,
       "keep": 512},
      # Keyformer with the noise from a seed, an odd length
      {"name": "keyformer_seeded_1500", "kind": "keyformer_seeded", "dtype": "bf16", "B": 2, "H": 32, "Sq": 1501,
       "Skv": 1501, "keep": 375},
      # RoCo with mean/deviation and selection, 40 heads (C4): the most operations
      {"name": "roco_select_4k", "kind": "roco_select", "dtype": "bf16", "B": 2, "H": 40, "Sq": 4096, "Skv": 4096,
       "keep": 512},
      # softmax-free attention over long sequences (C5)
      {"name": "sima_8k", "kind": "sima", "dtype": "f16", "B": 8, "H": 32, "S": 8192},
      # EA with few (batch, head) units and an odd length
      {"name": "ea_5k_ragged", "kind": "ea", "dtype": "bf16", "B": 2, "H": 32, "S": 5003},
      # the whole block of bench/sima.mlir at its own shape, f32: projections and core
      {"name": "sima_block", "kind": "sima_block", "dtype": "f32", "B": 64, "N": 784, "C": 128},
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["attn", "attn", "decode", "h2o_select", "h2o", "gemma2", "keyformer", "keyformer_seeded",
                     "roco_select", "sima", "ea", "sima_block", "ea_block"])
  dtype = rng.choice(["f16", "bf16"])
  if kind in ("sima_block", "ea_block"):
    return {"kind": kind, "dtype": "f32", "B": _log_int(rng, 2, 64), "N": _log_int(rng, 100, 784), "C": 128}
  if kind in ("sima", "ea"):
    B, H = rng.choice([1, 2, 3, 4, 8]), rng.choice([8, 16, 32])
    return {"kind": kind, "dtype": dtype, "B": B, "H": H, "S": _log_int(rng, 700, 8192)}
  if kind == "decode":
    Hkv, group = rng.choice([8, 16, 32]), rng.choice([1, 2, 4])
    return {"kind": "attn", "dtype": dtype, "B": _log_int(rng, 1, 16), "H": Hkv * group, "Hkv": Hkv,
            "Sq": rng.choice([1, 1, 1, 2, 4]), "Skv": _log_int(rng, 300, 8192), "causal": True}
  if kind == "h2o":
    Hkv, group, Sq = rng.choice([4, 8]), rng.choice([2, 4]), _log_int(rng, 100, 1024)
    return {"kind": "h2o", "dtype": dtype, "B": rng.choice([1, 1, 2]), "H": Hkv * group, "Hkv": Hkv, "Sq": Sq,
            "Skv": Sq + _log_int(rng, 200, 8000)}
  if kind in ("attn", "gemma2"):
    S = _log_int(rng, 128, 8192)
    Hkv, group = rng.choice([4, 8, 16]), rng.choice([1, 2])
    case = {"kind": kind, "dtype": dtype, "B": rng.choice([1, 2, 4]) if S <= 2048 else 1, "H": Hkv * group, "Hkv": Hkv,
            "Sq": S, "Skv": S}
    if kind == "attn":
      case["causal"] = rng.random() < 0.75 or S > 4096
    return case
  B, H = rng.choice([1, 2]), rng.choice([4, 16, 32, 40])
  S = _log_int(rng, 300, 2048 if kind == "keyformer" else 4096)
  case = {"kind": kind, "dtype": dtype, "B": B, "H": H, "Sq": S, "Skv": S, "keep": S // rng.choice([4, 8])}
  if kind == "h2o_select":
    case["recent"] = S // 16
  return case


def _model(case):
  kind = case["kind"]
  if kind == "sima_block":
    return SimABlock()
  if kind == "ea_block":
    return EABlock()
  heads = {"head_num": case["H"], "kv_head_num": case.get("Hkv", case["H"])}
  if kind == "attn":
    return ft.Attn(causal=case["causal"], **heads)
  return {"h2o": ft.H2O, "h2o_select": ft.H2O, "gemma2": ft.Gemma2, "keyformer": ft.KeyFormer,
          "keyformer_seeded": ft.KeyFormer, "roco_select": ft.RoCo, "sima": ft.SimA, "ea": ft.EA}[kind](**heads)


def prepare(case, seed):
  g = torch.Generator(device="cuda").manual_seed(seed)
  dt, kind = DTYPES[case["dtype"]], case["kind"]

  def normal(*shape, dtype=dt):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)

  state = {"case": dict(case), "model": _model(case)}
  if kind.endswith("_block"):
    C = case["C"]
    state["args"] = (normal(case["B"], case["N"], C), normal(3 * C, C) / C ** 0.5, normal(3 * C) * 0.1,
                     normal(C, C) / C ** 0.5, normal(C) * 0.1)
    return state
  B, H = case["B"], case["H"]
  Hkv = case.get("Hkv", H)
  Sq, Skv = case.get("Sq", case.get("S")), case.get("Skv", case.get("S"))
  q, k = normal(B, Sq, H, 128), normal(B, Skv, Hkv, 128)
  if kind == "sima":  # V ~ U(-1, 1), as the configuration has it
    v = (torch.rand((B, Skv, Hkv, 128), generator=g, device="cuda") * 2 - 1).to(dt)
  else:
    v = normal(B, Skv, Hkv, 128)
  state["args"] = (q, k, v)
  if kind == "keyformer":  # the case's own noise
    state["args"] += (normal(B, H, Sq, Skv, dtype=torch.float32).abs_().add_(1),)
  if kind == "keyformer_seeded":
    state["noise_seed"] = seed
  return state


def run(state):
  case, model, args = state["case"], state["model"], state["args"]
  kind = case["kind"]
  if kind == "h2o_select":
    return model.select(*args, case["keep"], case["recent"])
  if kind == "keyformer":
    return model.select(*args, case["keep"])
  if kind == "keyformer_seeded":
    return model.seeded(*args, state["noise_seed"], k_keep=case["keep"])
  if kind == "roco_select":
    return model.select(*args, case["keep"], return_stats=True)
  return model(*args)


def work(case):
  kind = case["kind"]
  if kind.endswith("_block"):
    B, N, C = case["B"], case["N"], case["C"]
    rows, weights = B * N, 4 * C * C + 4 * C
    return {"bytes": 4 * (2 * rows * C + weights), "flops": 2 * rows * C * 4 * C + 4 * rows * C * 32}
  B, H = case["B"], case["H"]
  if kind in ("sima", "ea"):
    return {"bytes": 4 * B * H * case["S"] * 128 * 2, "flops": 4 * B * H * case["S"] * 128 * 128}
  Hkv, Sq, Skv = case.get("Hkv", H), case["Sq"], case["Skv"]
  # (query, key) pairs that the mask leaves
  pairs = Sq * (Skv - Sq) + Sq * (Sq + 1) // 2 if case.get("causal", True) else Sq * Skv
  nbytes = 2 * 128 * B * (2 * Sq * H + 2 * Skv * Hkv)
  if kind in ("h2o", "h2o_select", "keyformer", "keyformer_seeded"):
    nbytes += 4 * B * Hkv * Skv
  if kind == "roco_select":
    nbytes += 4 * 4 * B * H * Skv
  if kind == "keyformer":
    nbytes += 4 * B * H * pairs  # (masked noise need not be read)
  nbytes += 4 * B * Hkv * (case.get("keep", 0) + case.get("recent", 0))
  return {"bytes": nbytes, "flops": 4 * 128 * B * H * pairs}


def tolerance(case):
  if case["dtype"] == "f32":
    return {"rel": 2e-5}
  # 16-bit outputs (and probabilities rounded to 16 bits inside); kept indices may differ at ties
  t = {"rel": 2e-3 if case["dtype"] == "f16" else 1e-2}
  if "keep" in case:
    t["differ"] = 0.01
  return t
