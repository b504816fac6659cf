"""The 128-row fused backward where its own branches can go wrong: the bits of dense partial blocks
(read per thread, straight from memory), the shortest and odd step counts of its rings, per-head
masks and grouped heads; against the CPU oracle with the bars of test_gpu_backward.py."""

import numpy as np
import pytest
import torch

import splash_attention_mgpu as sa
from oracle import dense_attention as oracle
from splash_attention_mgpu import splash_attention

from common import build_mask, inputs
from test_gpu_backward import _check_grads, _id

CASES = [
    dict(mask_name="dense", s=128, d=64),                                   # one step
    dict(mask_name="dense", s=128, d=128, cap=5.0),
    dict(mask_name="dense", s=384, d=64, h=4, kvh=2, segs=True, cap=5.0),   # odd, grouped
    dict(mask_name="dense", s=384, d=128, h=4, kvh=2, multi_head_mask=True),
    dict(mask_name="dense", s=640, d=64, h=5, multi_head_mask=True, dtype=torch.float16),
    dict(mask_name="full", s=256, d=64, h=3, mqa=True),                      # two steps per head, six in all
    dict(mask_name="causal", s=384, d=64, b=2, dtype=torch.float16),
]


@pytest.mark.gpu
@pytest.mark.parametrize("kwargs", CASES, ids=_id)
def test_gpu_wide_backward(kwargs):
  kwargs = dict(kwargs)
  _check_grads(kwargs.pop("mask_name"), scaled=True, **kwargs)


@pytest.mark.gpu
@pytest.mark.parametrize("mask_name,cap,h,kvh", [("dense", None, 2, 2), ("causal", None, 2, 2), ("full", 20.0, 4, 2)])
def test_gpu_f16_delta_beyond_the_range_of_f16(mask_name, cap, h, kvh):
  """Loss-scaled f16 gradients: rows whose delta = dO . O is above 65504 while every operand and gradient is
  finite.  delta comes from the output rounded to f16 (2^-11 of 200 a value, eight values' worth in the root of the
  64 terms), dP - delta from values 20 wide: that alone is 200 / 2^11 / sqrt(3) / 20 = 0.3 % of a score's gradient."""
  s, d = 384, 64
  mask, dense = build_mask(mask_name, s, h, False)
  kernel = sa.make_splash_mha(mask, attn_logits_soft_cap=cap)
  q, k, v = inputs(1, h, kvh, s, d, d, torch.float16, False, seed=3, device="cuda:0", scale=d ** -0.5)
  v = 200 + 20 * v
  g = torch.Generator().manual_seed(5)
  d_out = (40 + 8 * torch.randn(q.shape, generator=g)).to(torch.float16).to("cuda:0")
  qg, kg, vg = (x.clone().requires_grad_(True) for x in (q, k, v))
  out = kernel(qg, kg, vg)
  got = torch.autograd.grad(out, (qg, kg, vg), d_out)
  sa.check_device_status()
  assert float((d_out.float() * out.detach().float()).sum(-1).abs().min()) > 65504
  want = oracle.attention_backward(dense, q, k, v, d_out, attn_logits_soft_cap=cap)
  for name, x, r in zip("qkv", got, want):
    x = x.float().cpu().numpy()
    assert np.isfinite(x).all(), name
    assert np.abs(x - r).max() / np.abs(r).max() < 2e-2, name
    assert np.abs(x - r).mean() / np.abs(r).mean() <= 1e-2, name


def _takes_fused(d, dense, stages, **bs):
  q = torch.empty(1, 2, 128, d, dtype=torch.bfloat16)
  return splash_attention._use_fused_backward(q, q, sa.BlockSizes(num_stages_bwd=stages, **bs), dense, False)


def test_ring_depth_does_not_choose_the_backward():
  """CPU: the fused kernel's layout is fixed, so the depths that the split kernels hold run in it."""
  assert all(_takes_fused(d, dense, n) for d in (64, 128) for dense in (False, True) for n in (1, 2, 3))
  assert _takes_fused(128, False, 4) and not _takes_fused(128, True, 4)  # the latter is refused by the split kernels
  assert _takes_fused(128, False, 3, block_kv_dq=128) and not _takes_fused(128, True, 3, block_kv_dq=128)


@pytest.mark.gpu
@pytest.mark.parametrize("mask_name,stages", [("dense", 3), ("causal", 4)])
def test_gpu_deep_rings(mask_name, stages):
  _check_grads(mask_name, s=640, d=128, h=4, kvh=2, scaled=True, block_sizes=sa.BlockSizes(num_stages_bwd=stages))
