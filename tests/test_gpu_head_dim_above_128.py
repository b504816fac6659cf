"""The forward at head_dim 192 and 256 with 64-wide KV blocks, one softmax group where rows of up to 16 steps span
all keys, else two that take the steps in turn, with one CTA per SM: the fewest steps, odd counts, every
masking option (rows of two steps beside long ones in two groups: test_gpu_short_rows.py); against the CPU oracle with the bars of test_gpu_forward.py."""

import numpy as np
import pytest
import torch

import splash_attention_mgpu as sa
from oracle import dense_attention as oracle

from common import assert_forward_close, inputs
from test_gpu_forward import _check, _id

pytestmark = pytest.mark.gpu

B64 = sa.BlockSizes(block_q=128, block_kv=64)
CASES = [
    dict(mask_name="causal", s=128),
    dict(mask_name="full", s=384, b=2, dtype=torch.float16),
    dict(mask_name="local", s=640, segs=True, h=4, kvh=2),
    dict(mask_name="chunked", s=512, cap=5.0),
    dict(mask_name="dense", s=512, h=3, multi_head_mask=True),
    dict(mask_name="dense", s=512, h=4, mqa=True, segs=True),
]


@pytest.mark.parametrize("d", [192, 256])
@pytest.mark.parametrize("kwargs", CASES, ids=_id)
def test_gpu_forward_above_128(kwargs, d):
  kwargs = dict(kwargs)
  _check(kwargs.pop("mask_name"), d=d, block_sizes=B64, **kwargs)


@pytest.mark.parametrize("d,kv", [(192, 64), (192, 192), (256, 64), (256, 128), (256, 192)])
def test_gpu_few_steps(d, kv):
  q, _, _ = inputs(1, 2, 2, 128, d, d, torch.bfloat16, False, seed=1, device="cuda:0", scale=d ** -0.5)
  _, k, v = inputs(1, 2, 2, kv, d, d, torch.bfloat16, False, seed=2, device="cuda:0")
  kernel = sa.make_splash_mha(sa.FullMask((128, kv)), block_sizes=B64)
  out, (lse,) = kernel(q, k, v, save_residuals=True)
  sa.check_device_status()
  ref, ref_lse = oracle.attention_forward(np.ones((1, 128, kv), bool), q, k, v)
  assert_forward_close(out, lse, ref, ref_lse, torch.bfloat16)


def test_gpu_deepest_ring_that_one_group_had(monkeypatch):
  """head_dim 128, head_dim_v 64 with eight stages fills shared memory to 512 bytes: the library takes it
  (this package's own budget, the reference's formula, asks for more than the kernel uses)."""
  monkeypatch.setattr(sa.config, "SMEM_BYTES", 1 << 20)
  _check("causal", s=1024, d=128, dv=64, block_sizes=sa.BlockSizes(block_q=128, block_kv=64, num_stages=8))
