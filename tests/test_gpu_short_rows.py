"""The forward with 64-wide KV blocks on both sides of the line between one softmax group (head dims up to 128: rows of
up to 8 steps; above: up to 16 that span all keys) and two: against the CPU oracle with the bars of test_gpu_forward.py."""

import numpy as np
import pytest
import torch

import splash_attention_mgpu as sa
from oracle import dense_attention as oracle

from common import assert_forward_close, inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

MASKS = {
    "one-block": lambda: sa.CausalMask((128, 128)),                # 2 steps: one group
    "window-8": lambda: sa.LocalMask((1536, 1536), (384, 0), 0),   # 8 steps: one group up to head_dim 128
    "window-9": lambda: sa.LocalMask((1536, 1536), (448, 0), 0),   # 9: two
    "causal-16": lambda: sa.CausalMask((1024, 1024)),              # 16 steps, all keys: one above 128
    "causal-18": lambda: sa.CausalMask((1152, 1152)),              # 18: two, rows of 2 steps among them
    "offset-16": lambda: sa.CausalMask((256, 1088), offset=768),   # 16 of 17: two
}


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 64), (192, 192), (256, 256)])
@pytest.mark.parametrize("name,form", [(n, {}) for n in MASKS] + [
    ("window-8", dict(segs=True, dtype=torch.float16)), ("causal-16", dict(cap=5.0)), ("window-8", dict(array=True)),
    ("causal-18", dict(segs=True, cap=5.0)), ("one-block", dict(array=True, segs=True, dtype=torch.float16))],
    ids=lambda x: x if isinstance(x, str) else ",".join(x))
def test_gpu_both_sides_of_the_line(name, form, d, dv):
  mask = MASKS[name]()
  dense = np.asarray(mask[:, :])
  if form.get("array"):
    dense = dense & ((np.random.default_rng(1).random(dense.shape) > 0.3) | np.eye(*dense.shape, dtype=bool))
    mask = sa.NumpyMask(dense)
  q_len, kv_len = dense.shape
  dtype, cap, seg = form.get("dtype", torch.bfloat16), form.get("cap"), None
  kernel = sa.make_splash_mha(mask, block_sizes=sa.BlockSizes(block_q=128, block_kv=64, num_stages=2),
                              attn_logits_soft_cap=cap)
  q, k, v = inputs(1, 4, 2, kv_len, d, dv, dtype, False, seed=3, device=DEV)
  q = (q[:, :, :q_len] * d ** -0.5).contiguous()
  if form.get("segs"):
    ids = torch.arange(kv_len, dtype=torch.int32, device=DEV) // 200
    seg = sa.SegmentIds(ids[:q_len], ids)
  out, (lse,) = kernel(q, k, v, seg, save_residuals=True)
  sa.check_device_status()
  ref, ref_lse = oracle.attention_forward(dense[None], q, k, v, seg, attn_logits_soft_cap=cap)
  assert_forward_close(out, lse, ref, ref_lse, dtype)
  assert torch.equal(kernel(q, k, v, seg), out)
