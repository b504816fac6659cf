"""What a user of the splash attention library has it do, as measurable cases.

Every case goes through the public API (`make_splash_mha` / `make_splash_mqa`, the kernel object's
call, `torch.autograd.grad`).  The kernel object -- the processed mask and its schedules -- is what a
program builds once and keeps, so it is made in `prepare`.

A case is a dict of plain values:

  mode    "infer"  out = kernel(q, k, v), no gradients wanted
          "fwd"    out and logsumexp (save_residuals=True)
          "train"  forward and backward: out, dq, dk, dv
  mask    "full", "causal" (rows end at the last key: a chunk of queries against a longer cache when
          q_len < kv_len), "local" (sliding window to the left), "chunked", "mixed" (causal and
          chunked heads in turn), "blocks" (block-sparse boolean array), "holes" (causal boolean array
          with random elements off)
  docs    packed documents of docs_min..docs_max tokens as segment ids (docs_seed draws their lengths)
"""

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "pallas-mosaic-gpu_b200"))

import splash_attention_mgpu as sa  # noqa: E402

DEVICE = "cuda"


def _case(**kw):
  c = dict(mode="train", mask="causal", batch=1, heads=8, kv_heads=8, q_len=1024, kv_len=0, head_dim=128,
           dtype="bf16", cap=0.0, window=0, chunk=0, mask_seed=0, docs=False, docs_min=0, docs_max=0, docs_seed=0,
           mqa=False, block_q=0, block_kv=0)
  c.update(kw)
  c["kv_len"] = c["kv_len"] or c["q_len"]
  return c


def listed():
  return [
      # A toy or a unit of work per token group: one call is launches and host work.
      _case(name="tiny_infer_d64", mode="infer", heads=4, kv_heads=4, q_len=256, head_dim=64),
      # Fine-tuning on short sequences, grouped heads, a length that is an odd number of blocks.
      _case(name="short_gqa_train", batch=2, heads=8, kv_heads=2, q_len=1152),
      # A chunk of a prompt against the keys already cached (offset causal), grouped heads.
      _case(name="chunked_prefill", mode="infer", heads=32, kv_heads=8, q_len=256, kv_len=16640),
      # Prefill of a batch of prompts, and the same shape as a training step: the library's headline.
      _case(name="causal_prefill", mode="fwd", batch=2, heads=16, kv_heads=16, q_len=8192),
      _case(name="causal_train", batch=2, heads=16, kv_heads=16, q_len=8192),
      # Bidirectional attention over one long sequence.
      _case(name="full_long", mode="fwd", mask="full", heads=16, kv_heads=16, q_len=16384),
      # Sliding window, grouped heads, soft-capped logits: training at long context.
      _case(name="window_gqa_cap_train", mask="local", window=1024, heads=32, kv_heads=8, q_len=16384, cap=50.0),
      # Packed documents, bidirectional, f16 at head_dim 64 (encoder training).
      _case(name="packed_full_train_d64", mask="full", batch=4, heads=16, kv_heads=16, q_len=8192, head_dim=64,
            dtype="f16", docs=True, docs_min=256, docs_max=4096, docs_seed=7),
      # Causal and chunked heads side by side on packed documents, an odd length.
      _case(name="packed_mixed_train_d64", mask="mixed", chunk=1024, batch=2, heads=16, kv_heads=16, q_len=4224,
            head_dim=64, dtype="f16", docs=True, docs_min=256, docs_max=4096, docs_seed=8),
      # The ordinary training step of a model with head_dim 64.
      _case(name="causal_train_d64", batch=4, heads=16, kv_heads=16, q_len=8192, head_dim=64, dtype="f16"),
      # A mask given as an array: training through streamed mask blocks, grouped heads.
      _case(name="array_mask_gqa_train", mask="holes", mask_seed=3, batch=2, heads=16, kv_heads=4, q_len=4096),
      # Block-sparse attention with one shared key/value head, head_dim 256.
      _case(name="mqa_block_sparse_d256", mode="fwd", mask="blocks", mask_seed=5, heads=64, kv_heads=1, q_len=8192,
            head_dim=256, mqa=True, block_q=128, block_kv=64),
  ]


def _spread(rng, lo, hi):
  """Whole number in [lo, hi], spread over its logarithm."""
  return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
  family = rng.choice(("plain", "plain", "plain", "window", "packed", "prefill", "array", "blocks"))
  head_dim = rng.choice((64, 128))
  dtype = rng.choice(("bf16", "f16"))
  mode = rng.choice(("infer", "fwd", "train", "train"))
  kv_heads = rng.choice((1, 2, 4, 8, 16))
  group = rng.choice((1, 1, 2, 4))
  common = dict(mode=mode, head_dim=head_dim, dtype=dtype, kv_heads=kv_heads, heads=kv_heads * group,
                batch=rng.choice((1, 1, 2, 4)), q_len=128 * _spread(rng, 1, 128))
  if family == "plain":
    mask = rng.choice(("full", "causal", "causal", "chunked"))
    c = _case(**common, mask=mask, chunk=128 * _spread(rng, 2, 32) if mask == "chunked" else 0)
  elif family == "window":
    c = _case(**common, mask="local", window=_spread(rng, 100, 4096), cap=rng.choice((0.0, 30.0, 50.0)))
  elif family == "packed":
    mask = rng.choice(("full", "causal", "mixed"))
    c = _case(**common, mask=mask, chunk=1024 if mask == "mixed" else 0, docs=True, docs_min=rng.choice((64, 256)),
              docs_max=rng.choice((1024, 4096)), docs_seed=rng.randrange(1 << 20))
  elif family == "prefill":
    c = _case(**dict(common, mode="infer", q_len=128 * _spread(rng, 1, 16)))
    c["kv_len"] = max(c["q_len"], 128 * _spread(rng, 8, 256))
  elif family == "array":
    c = _case(**dict(common, q_len=128 * _spread(rng, 2, 32)), mask="holes", mask_seed=rng.randrange(1 << 20))
  else:
    c = _case(**dict(common, mode=rng.choice(("infer", "fwd")), head_dim=256, kv_heads=1, heads=8 * group,
                     q_len=128 * _spread(rng, 8, 64)),
              mask="blocks", mask_seed=rng.randrange(1 << 20), mqa=True, block_q=128, block_kv=64)
  # No drawn case costs more than the training steps above.
  while _flops(c, _spans(c)) > 1.9e12:
    if c["batch"] > 1:
      c["batch"] //= 2
    elif c["kv_heads"] > 1:
      c["kv_heads"] //= 2
      c["heads"] //= 2
    else:
      c["q_len"] = c["kv_len"] = 128 * (c["q_len"] // 256)
  return c


# ---------------------------------------------------------------------------
# Masks, in this file's own terms: for each head pattern the half-open span of visible keys of each row,
# and for array masks the array itself.
# ---------------------------------------------------------------------------


def _docs(c, batch_row):
  """Segment ids [q_len] of one batch row."""
  rng = np.random.default_rng((c["docs_seed"], batch_row))
  ids, pos, seg = np.zeros(c["q_len"], np.int32), 0, 0
  while pos < c["q_len"]:
    n = int(rng.integers(c["docs_min"], c["docs_max"] + 1))
    ids[pos:pos + n] = seg
    pos, seg = pos + n, seg + 1
  return ids


def _array_mask(c):
  s = c["q_len"]
  rng = np.random.default_rng(c["mask_seed"])
  if c["mask"] == "holes":
    m = np.tril(np.ones((s, s), bool)) & (rng.random((s, s), dtype=np.float32) > 0.3)
  else:
    kinds = rng.choice(3, size=(s // 128, s // 64), p=[0.70, 0.10, 0.20])  # empty, partial, full
    m = np.repeat(np.repeat(kinds == 2, 128, axis=0), 64, axis=1)
    for i, j in zip(*np.nonzero(kinds == 1)):
      m[i * 128:(i + 1) * 128, j * 64:(j + 1) * 64] = rng.random((128, 64), dtype=np.float32) < 0.5
  m[np.arange(s), np.arange(s)] = True  # every row sees itself
  return m


def _head_spans(c):
  """[(lo, hi) per head pattern]: visible keys of row i are lo[i] .. hi[i] - 1 (array masks: at most)."""
  q, kv = c["q_len"], c["kv_len"]
  i = np.arange(q)
  causal = (np.zeros(q, np.int64), i + 1 + (kv - q))
  if c["mask"] in ("full", "blocks"):
    return [(np.zeros(q, np.int64), np.full(q, kv))]
  if c["mask"] == "local":
    return [(np.maximum(0, i - c["window"]), i + 1)]
  if c["mask"] == "chunked":
    return [(i // c["chunk"] * c["chunk"], i + 1)]
  if c["mask"] == "mixed":
    return [causal, (i // c["chunk"] * c["chunk"], i + 1)]
  return [causal]


def _spans(c):
  """spans[batch row][head pattern] = (lo, hi), documents taken into account."""
  heads = _head_spans(c)
  if not c["docs"]:
    return [heads] * c["batch"]
  out = []
  for b in range(c["batch"]):
    ids = _docs(c, b)
    lo, hi = np.searchsorted(ids, ids, "left"), np.searchsorted(ids, ids, "right")
    out.append([(np.maximum(l, lo), np.minimum(h, hi)) for l, h in heads])
  return out


def _visible(c, spans):
  """Visible (row, key) pairs over batch and heads."""
  if c["mask"] == "blocks":
    return c["batch"] * c["heads"] * 0.25 * c["q_len"] * c["kv_len"]
  per = [sum(int((h - l).sum()) for l, h in row) / len(row) for row in spans]
  share = 0.7 if c["mask"] == "holes" else 1.0
  return c["heads"] * sum(per) * share


def _flops(c, spans):
  return (14 if c["mode"] == "train" else 4) * c["head_dim"] * _visible(c, spans)


def work(case):
  c = case
  q = c["batch"] * c["heads"] * c["q_len"] * c["head_dim"] * 2
  kv = c["batch"] * c["kv_heads"] * c["kv_len"] * c["head_dim"] * 2
  n = 2 * q + 2 * kv
  if c["mode"] == "fwd":
    n += c["batch"] * c["heads"] * c["q_len"] * 4
  if c["mode"] == "train":
    n += 2 * q + 2 * kv  # dO, dQ, dK, dV
  if c["docs"]:
    n += 2 * c["batch"] * c["q_len"] * 4
  return {"bytes": n, "flops": _flops(c, _spans(c))}


# ---------------------------------------------------------------------------


def _inputs(c, seed):
  g = torch.Generator(device=DEVICE).manual_seed(seed)
  dtype = torch.bfloat16 if c["dtype"] == "bf16" else torch.float16
  lead = (c["batch"],)
  kv = lead + (() if c["mqa"] else (c["kv_heads"],)) + (c["kv_len"], c["head_dim"])
  qs = lead + (c["heads"], c["q_len"], c["head_dim"])
  normal = lambda shape, scale=1.0: (torch.randn(shape, generator=g, device=DEVICE) * scale).to(dtype)
  # q arrives scaled by head_dim ** -0.5, as the library expects it.
  return normal(qs, c["head_dim"] ** -0.5), normal(kv), normal(kv), normal(qs)


def _mask(c):
  q, kv = c["q_len"], c["kv_len"]
  causal = sa.CausalMask((q, kv), offset=kv - q)
  if c["mask"] == "full":
    return sa.FullMask((q, kv))
  if c["mask"] == "causal":
    return causal
  if c["mask"] == "local":
    return sa.LocalMask((q, kv), (c["window"], 0), 0)
  if c["mask"] == "chunked":
    return sa.ChunkedCausalMask((q, kv), chunk_size=c["chunk"])
  if c["mask"] == "mixed":
    chunked = sa.ChunkedCausalMask((q, kv), chunk_size=c["chunk"])
    return sa.MultiHeadMask([causal if h % 2 == 0 else chunked for h in range(c["heads"])])
  return sa.NumpyMask(_array_mask(c))


def prepare(case, seed):
  c = case
  make = sa.make_splash_mqa if c["mqa"] else sa.make_splash_mha
  kernel = make(_mask(c), block_sizes=sa.BlockSizes(block_q=c["block_q"] or None, block_kv=c["block_kv"] or None),
                attn_logits_soft_cap=c["cap"] or None)
  q, k, v, d_out = _inputs(c, seed)
  if c["mode"] == "train":
    q, k, v = (x.requires_grad_(True) for x in (q, k, v))
  else:
    d_out = None
  seg = None
  if c["docs"]:
    ids = torch.from_numpy(np.stack([_docs(c, b) for b in range(c["batch"])])).to(DEVICE)
    seg = sa.SegmentIds(ids, ids)
  return {"mode": c["mode"], "kernel": kernel, "q": q, "k": k, "v": v, "d_out": d_out, "seg": seg}


def run(state):
  kernel, q, k, v, seg = (state[n] for n in ("kernel", "q", "k", "v", "seg"))
  if state["mode"] == "infer":
    return kernel(q, k, v, seg)
  if state["mode"] == "fwd":
    out, (lse,) = kernel(q, k, v, seg, save_residuals=True)
    return out, lse
  out = kernel(q, k, v, seg)
  return (out.detach(),) + torch.autograd.grad(out, (q, k, v), state["d_out"])


# About four times the largest error seen against `exact` over the listed cases and some drawn ones
# (bf16: relative 2.6e-3, single value 0.16 of the root mean square; f16: 3.2e-4 and 0.019): results
# and the probabilities between the two products are 16-bit numbers.
_REL = {"bf16": 1.0e-2, "f16": 1.3e-3}
_MAX = {"bf16": 0.6, "f16": 0.075}


def tolerance(case):
  return {"rel": _REL[case["dtype"]], "max": _MAX[case["dtype"]]}


def exact(case, seed):
  c = case
  train, cap, group = c["mode"] == "train", c["cap"], c["heads"] // c["kv_heads"]
  q, k, v, d_out = (x.double() for x in _inputs(c, seed))
  if c["mqa"]:
    k, v = k.unsqueeze(1), v.unsqueeze(1)
  array = torch.from_numpy(_array_mask(c)).to(DEVICE) if c["mask"] in ("blocks", "holes") else None
  spans = _spans(c)
  out, lse = torch.zeros_like(q), torch.zeros(q.shape[:3], dtype=torch.float64, device=DEVICE)
  dq, dk, dv = (torch.zeros_like(x) for x in (q, k, v)) if train else (None, None, None)
  step = 1024
  for b in range(c["batch"]):
    per_head = [tuple(torch.from_numpy(x).to(DEVICE) for x in s) for s in spans[b]]
    for h in range(c["heads"]):
      lo, hi = per_head[h % len(per_head)]
      lo_np, hi_np = spans[b][h % len(per_head)]
      kh = h // group
      for r0 in range(0, c["q_len"], step):
        rows = slice(r0, min(r0 + step, c["q_len"]))
        c0, c1 = int(lo_np[rows].min()), int(hi_np[rows].max())
        cols = torch.arange(c0, c1, device=DEVICE)
        kc, vc, qr = k[b, kh, c0:c1], v[b, kh, c0:c1], q[b, h, rows]
        s = qr @ kc.T
        if cap:
          t = torch.tanh(s / cap)
          s = t * cap
        seen = (cols >= lo[rows, None]) & (cols < hi[rows, None])
        if array is not None:
          seen &= array[rows, c0:c1]
        s = s.masked_fill(~seen, -math.inf)
        lse[b, h, rows] = torch.logsumexp(s, dim=-1)
        p = torch.exp(s - lse[b, h, rows, None])
        out[b, h, rows] = p @ vc
        if train:
          do = d_out[b, h, rows]
          ds = p * (do @ vc.T - (do * out[b, h, rows]).sum(-1, keepdim=True))
          if cap:
            ds = ds * (1 - t * t)
          dv[b, kh, c0:c1] += p.T @ do
          dk[b, kh, c0:c1] += ds.T @ qr
          dq[b, h, rows] = ds @ kc
  if c["mode"] == "infer":
    return out
  if c["mode"] == "fwd":
    return out, lse
  if c["mqa"]:
    dk, dv = dk.squeeze(1), dv.squeeze(1)
  return out, dq, dk, dv
