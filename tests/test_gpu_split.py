"""Forward calls whose q tiles are shared by several CTAs because they alone would leave SMs idle:
against the CPU oracle with the bars of the unshared kernels, at the smallest and odd share counts, with
shares left empty by segment skipping and rows that see no key."""

import ctypes

import numpy as np
import pytest
import torch

import splash_attention_mgpu as sa
from oracle import dense_attention as oracle
from splash_attention_mgpu import _ffi

from common import assert_forward_close, inputs

DEV = "cuda:0"


def _params(**kw):
  p = _ffi.SplashParams()
  for k, v in dict(dict(batch=1, heads=4, kv_heads=4, q_len=256, kv_len=8192, head_dim=128, head_dim_v=128, block_q=128,
                        block_kv=128, max_steps=64, mask_heads=1), **kw).items():
    setattr(p, k, v)
  return p


def test_forward_share_rule():
  """CPU: 0 bytes where one CTA per tile is kept, else splits * rows * (head_dim_v + 2) floats."""
  size = lambda **kw: _ffi.load().splash_fwd_split_bytes(ctypes.byref(_params(**kw)))
  rows = lambda h, q: h * q * (128 + 2) * 4
  assert size() == 16 * rows(4, 256)                              # 8 tiles on 148 SMs, 512 keys per share
  assert size(heads=32, q_len=256) == 2 * rows(32, 256)           # 64 tiles: two CTAs each
  assert size(heads=32, q_len=512) == 0                           # 128 tiles fill the GPU
  assert size(heads=32, q_len=512, block_kv=64, max_steps=128) == 2 * rows(32, 512)  # two CTAs per SM
  assert size(max_steps=16) == 0                                  # 2048 keys: less than that would come off
  assert size(max_steps=24) == 6 * rows(4, 256)
  assert size(heads=1, q_len=128, kv_len=1 << 20, max_steps=1 << 13) == 32 * rows(1, 128)


def test_forward_shares_count_the_ctas_that_an_sm_holds():
  """CPU: 128 tiles of 64-wide blocks get a second CTA each only where two CTAs' shared memory fits an SM."""
  size = lambda d, stages, **kw: _ffi.load().splash_fwd_split_bytes(ctypes.byref(_params(
      heads=32, q_len=512, block_kv=64, max_steps=128, **dict(dict(head_dim=d, head_dim_v=d, num_stages=stages), **kw))))
  assert size(128, 2) > 0 and size(128, 3) == 0
  assert size(64, 5) > 0 and size(64, 6) == 0
  assert size(128, 2, head_dim_v=64) > 0 and size(192, 2) == 0


def test_tiling_of_few_tiles():
  """CPU: 128-wide blocks for up to one tile per SM, up to 7/4 where row lengths differ; a tiling of which
  a part is given stays what it was."""
  tiling = lambda mask, tiles, d=128, **bs: (lambda r: (r.block_q, r.block_kv, r.num_stages))(
      sa.make_splash_mha(mask, block_sizes=sa.BlockSizes(**bs)).resolved_block_sizes(d, d, tiles=tiles))
  causal, local = sa.CausalMask((1024, 1024)), sa.LocalMask((2048, 2048), (512, 0), 0)
  for d in (64, 128):
    assert tiling(causal, 148, d) == (128, 128, 2) == tiling(causal, 259, d)
    assert tiling(causal, 260, d) == tiling(causal, None, d) == (128, 64, 2)
    assert tiling(local, 148, d) == (128, 128, 2) and tiling(local, 149, d) == (128, 64, 2)
  assert tiling(causal, 8, block_kv=64) == (128, 64, 2) == tiling(causal, None, block_kv=64)
  assert tiling(causal, 8, num_stages=3) == (128, 64, 3)


@pytest.mark.parametrize("d", [64, 128])
def test_short_rows_keep_their_tiling(d):
  """CPU: few tiles, but a single block a row or a narrow window: the tiling that does not depend on the call."""
  tiling = lambda mask, tiles: (lambda r: (r.block_q, r.block_kv, r.num_stages))(
      sa.make_splash_mha(mask).resolved_block_sizes(d, d, tiles=tiles))
  window = lambda w: sa.LocalMask((2048, 2048), (w, 0), 0)
  chunks = lambda c: sa.ChunkedCausalMask((2048, 2048), chunk_size=c)
  for mask in [sa.CausalMask((128, 128)), *map(window, (64, 128, 256, 320)), *map(chunks, (128, 256, 384))]:
    assert tiling(mask, 8) == tiling(mask, None) == (128, 64, 2)
  for mask in [sa.CausalMask((256, 256)), sa.CausalMask((384, 384)), window(384), window(512), chunks(512)]:
    assert tiling(mask, 8) == (128, 128, 2) != tiling(mask, None)


CASES = [
    dict(q=128, kv=2816),
    dict(q=128, kv=2944, d=64, dtype=torch.float16),
    dict(q=384, kv=3200, h=2, kvh=1, cap=20.0),
    dict(q=256, kv=4096, d=256, h=3, kvh=1, block_sizes=sa.BlockSizes(block_kv=64)),
    dict(q=256, kv=4096, block_sizes=sa.BlockSizes(block_q=256)),
    dict(q=256, kv=3072, d=64, mask="full", block_sizes=sa.BlockSizes(block_q=256)),
    dict(q=3072, kv=3072, h=2, mask="full", segs=256),      # shares that skipping leaves without a step
    dict(q=3072, kv=3072, h=2, mask="full", segs=3072, d=64),  # no shared id at all: rows without a key
    dict(q=256, kv=3072, mask="holes"),
    dict(q=256, kv=4096, d=128, b=2, h=4, kvh=2, dtype=torch.float16, block_sizes=sa.BlockSizes(block_kv=64)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("c", CASES, ids=lambda c: ",".join(f"{k}={v}" for k, v in c.items()))
def test_gpu_split_forward(c):
  q_len, kv_len, d, h = c["q"], c["kv"], c.get("d", 128), c.get("h", 2)
  b, kvh, dtype, cap = c.get("b", 1), c.get("kvh", c.get("h", 2)), c.get("dtype", torch.bfloat16), c.get("cap")
  rows, cols = np.arange(q_len)[:, None], np.arange(kv_len)[None]
  dense = np.ones((q_len, kv_len), bool) if c.get("mask") == "full" else cols <= rows + (kv_len - q_len)
  if c.get("mask") == "holes":
    dense = dense & (np.random.default_rng(0).random(dense.shape) > 0.4)
    dense[5] = False                                         # a row without a key
    mask = sa.NumpyMask(dense)
  elif c.get("mask") == "full":
    mask = sa.FullMask((q_len, kv_len))
  else:
    mask = sa.CausalMask((q_len, kv_len), offset=kv_len - q_len)
  kernel = sa.make_splash_mha(mask, block_sizes=c.get("block_sizes"), attn_logits_soft_cap=cap)
  g = torch.Generator().manual_seed(1)
  draw = lambda n, s: torch.randn(b, n, s, d, generator=g).to(dtype).to(DEV)
  q, k, v = draw(h, q_len) * d ** -0.5, draw(kvh, kv_len), draw(kvh, kv_len)
  seg = None
  if c.get("segs"):
    sq = torch.arange(q_len, dtype=torch.int32) // c["segs"]
    skv = torch.arange(kv_len, dtype=torch.int32) // c["segs"] + (c["segs"] == kv_len)
    seg = sa.SegmentIds(sq.to(DEV), skv.to(DEV))
  bs = kernel.resolved_block_sizes(d, d, has_segments=seg is not None, tiles=b * h * q_len // 128)
  sched = kernel.fwd_info(bs.block_q, bs.block_kv)
  assert _ffi.load().splash_fwd_split_bytes(ctypes.byref(_params(
      batch=b, heads=h, kv_heads=kvh, q_len=q_len, kv_len=kv_len, head_dim=d, head_dim_v=d, block_q=bs.block_q,
      block_kv=bs.block_kv, max_steps=sched.kv_block.shape[-1]))) > 0, "this case is meant to be shared"
  out, (lse,) = kernel(q, k, v, seg, save_residuals=True)
  sa.check_device_status()
  if c.get("segs") == kv_len:
    assert not out.any() and bool((lse == kernel.mask_value).all())
    return
  for i in range(b):
    ref, ref_lse = oracle.attention_forward(dense[None], q[i], k[i], v[i], None if seg is None else (sq.numpy(), skv.numpy()),
                                            attn_logits_soft_cap=cap)
    if c.get("mask") == "holes":                             # zeros and mask_value, as in the unshared kernel
      assert not out[i][:, 5].any() and bool((lse[i][:, 5] == kernel.mask_value).all())
      keep = np.arange(q_len) != 5
      assert_forward_close(out[i][:, keep], lse[i][:, keep], ref[:, keep], ref_lse[:, keep], dtype)
    else:
      assert_forward_close(out[i], lse[i], ref, ref_lse, dtype)


@pytest.mark.gpu
def test_gpu_calls_with_a_backward_do_not_share():
  """A unit's results are the same to the bit alone and among others, where gradients follow."""
  s, d = 4096, 64
  q, k, v = (torch.randn(2, 4, s, d, generator=torch.Generator().manual_seed(i)).to(torch.bfloat16).to(DEV) * 0.3
             for i in range(3))
  kernel = sa.make_splash_mha(sa.CausalMask((s, s)))

  def run(*x):
    x = [t.clone().requires_grad_(True) for t in x]
    out = kernel(*x)
    return (out.detach(),) + torch.autograd.grad(out, x[1:], torch.ones_like(out))

  whole, alone = run(q, k, v), run(q[1:, 2:3], k[1:, 2:3], v[1:, 2:3])
  for a, b in zip(whole, alone):
    assert torch.equal(a[1, 2], b[0, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_gpu_inputs_that_require_grad_without_a_gradient_to_come(mode):
  """Parameters used under no_grad: the call is the same as with inputs that require no gradient, shares included."""
  q, k, v = (torch.randn(1, 2, n, 128, generator=torch.Generator().manual_seed(n)).to(torch.bfloat16).to(DEV) * 0.3
             for n in (256, 4096, 4096))
  kernel = sa.make_splash_mha(sa.CausalMask((256, 4096), offset=4096 - 256))
  plain, with_lse = kernel(q, k, v), kernel(q, k, v, save_residuals=True)[0]
  leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
  with mode():
    out = kernel(*leaves)
  assert not out.requires_grad
  assert torch.equal(out, plain) and torch.equal(out, with_lse)


@pytest.mark.gpu
@pytest.mark.parametrize("d,bq,bkv", [(64, 128, 64), (128, 128, 128), (128, 256, 64)])
def test_gpu_tiling_given_in_full_keeps_a_units_bits(d, bq, bkv):
  """Few tiles, long rows: alone, in a batch, with and without gradients, and with the logsumexp."""
  g = lambda n: torch.randn(2, 4, n, d, generator=torch.Generator().manual_seed(n)).to(torch.bfloat16).to(DEV) * 0.3
  q, k, v = g(256), g(4096), g(4097)[:, :, 1:].contiguous()
  kernel = sa.make_splash_mha(sa.CausalMask((256, 4096), offset=4096 - 256),
                              block_sizes=sa.BlockSizes(block_q=bq, block_kv=bkv, num_stages=2))
  unit = [t[1:, 2:3] for t in (q, k, v)]
  whole, alone, (with_lse, _) = kernel(q, k, v), kernel(*unit), kernel(*unit, save_residuals=True)
  trained = kernel(*(t.clone().requires_grad_(True) for t in unit)).detach()
  for x in (alone, with_lse, trained):
    assert torch.equal(x[0, 0], whole[1, 2])


def _local(q, kv, window):
  return sa.LocalMask((q, kv), (window, 0), kv - q)


FORMS = [
    dict(mask=lambda q, kv: sa.CausalMask((q, kv), offset=kv - q), d=192, block_sizes=sa.BlockSizes(block_kv=64)),
    dict(mask=lambda q, kv: sa.CausalMask((q, kv), offset=kv - q), d=128, dv=64),
    dict(mask=lambda q, kv: sa.CausalMask((q, kv), offset=kv - q), d=64, dv=128, cap=10.0),
    dict(mask=lambda q, kv: _local(q, kv, 3000), kv=8192),
    dict(mask=lambda q, kv: sa.ChunkedCausalMask((q, kv), chunk_size=3072), q=6144, kv=6144, h=1),
    dict(mask=lambda q, kv: sa.MultiHeadMask([sa.CausalMask((q, kv), offset=kv - q), _local(q, kv, 700),
                                              sa.FullMask((q, kv))]), h=3, d=64),
    dict(mask=lambda q, kv: sa.CausalMask((q, kv), offset=kv - q), h=3, mqa=True, dtype=torch.float16),
]


@pytest.mark.gpu
@pytest.mark.parametrize("c", FORMS, ids=["d192", "d128-dv64", "d64-dv128-cap", "local", "chunked", "per-head", "mqa"])
def test_gpu_shares_by_plain_inference(c, monkeypatch):
  """The call that writes no logsumexp, for the masks and head dims that the cases above leave out: it takes shares,
  agrees with the oracle, and has the bits of the call with a logsumexp."""
  q_len, kv_len, h, d = c.get("q", 256), c.get("kv", 4096), c.get("h", 2), c.get("d", 128)
  dtype, cap, mqa = c.get("dtype", torch.bfloat16), c.get("cap"), c.get("mqa", False)
  mask = c["mask"](q_len, kv_len)
  heads = mask.masks if isinstance(mask, sa.MultiHeadMask) else [mask]
  dense = np.stack([np.asarray(m[:, :]) for m in heads])
  q, k, v = inputs(1, h, h, kv_len, d, c.get("dv", d), dtype, mqa, seed=2, device=DEV)
  q = (q[:, :, :q_len] * d ** -0.5).contiguous()
  kernel = (sa.make_splash_mqa if mqa else sa.make_splash_mha)(mask, block_sizes=c.get("block_sizes"),
                                                               attn_logits_soft_cap=cap)
  lib, shared = _ffi.load(), []
  entry = lib.splash_fwd_split
  monkeypatch.setattr(lib, "splash_fwd_split", lambda *a: shared.append(entry(*a)) or shared[-1])
  out = kernel(q, k, v)
  assert shared == [0]
  with_lse, (lse,) = kernel(q, k, v, save_residuals=True)
  sa.check_device_status()
  assert shared == [0, 0] and torch.equal(out, with_lse)
  ref, ref_lse = oracle.attention_forward(dense, q, k, v, is_mqa=mqa, attn_logits_soft_cap=cap)
  assert_forward_close(out, lse, ref, ref_lse, dtype)
