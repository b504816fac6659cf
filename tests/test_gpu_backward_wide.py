"""The 128-row fused backward where its own branches can go wrong: the bits of dense partial blocks
(read per thread, straight from memory), the shortest and odd step counts of its rings, per-head
masks and grouped heads; against the CPU oracle with the bars of test_gpu_backward.py."""

import pytest
import torch

from test_gpu_backward import _check_grads, _id

pytestmark = pytest.mark.gpu

CASES = [
    dict(mask_name="dense", s=128, d=64),                                   # one step
    dict(mask_name="dense", s=128, d=128, cap=5.0),
    dict(mask_name="dense", s=384, d=64, h=4, kvh=2, segs=True, cap=5.0),   # odd, grouped
    dict(mask_name="dense", s=384, d=128, h=4, kvh=2, multi_head_mask=True),
    dict(mask_name="dense", s=640, d=64, h=5, multi_head_mask=True, dtype=torch.float16),
    dict(mask_name="full", s=256, d=64, h=3, mqa=True),                      # two steps per head, six in all
    dict(mask_name="causal", s=384, d=64, b=2, dtype=torch.float16),
]


@pytest.mark.parametrize("kwargs", CASES, ids=_id)
def test_gpu_wide_backward(kwargs):
  kwargs = dict(kwargs)
  _check_grads(kwargs.pop("mask_name"), scaled=True, **kwargs)
