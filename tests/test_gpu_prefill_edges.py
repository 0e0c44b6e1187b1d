"""Prefill-shaped attention at the edges of its number range, against an fp64 softmax.

Tolerances as in test_gpu_prefill_attention.py: bf16 in, bf16 out, and with
`dense_attention` a logit on a bf16 rounding boundary may fall to either side (2e-2 for
a single row, 5e-3 for all rows together)."""

import math

import pytest
import torch

from jetstream_pytorch_b200 import attention_kernel as ak

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(hq, hkv, t, s, seed=3):
  g = torch.Generator(device=DEV).manual_seed(seed)
  return [torch.randn((1, h, n, 128), generator=g, device=DEV, dtype=torch.bfloat16) for h, n in ((hq, t), (hkv, s), (hkv, s))]


def _softmax_rows(q, k, v, mask, rounded):
  """fp64 attention; `rounded`: the logit chain of `dense_attention` in bf16 steps."""
  b, hq, t, d = q.shape
  hkv = k.shape[1]
  lg = q.reshape(b, hkv, -1, d).double() @ k.double().transpose(2, 3)
  if rounded:
    lg = (lg.float().to(torch.bfloat16).double() / math.sqrt(d)).float().to(torch.bfloat16)
    lg = (lg.float() + mask.float()).to(torch.bfloat16).double()
  else:
    lg = lg / math.sqrt(d) + mask.double()
  return (torch.softmax(lg, -1) @ v.double()).reshape(b, hq, t, d)


def _check(got, want, row=2e-2, whole=5e-3):
  got = got.double()
  worst = float(((got - want).norm(dim=-1) / want.norm(dim=-1)).max())
  assert worst <= row and float((got - want).norm() / want.norm()) <= whole, worst


@pytest.mark.parametrize("value", [-1e4, -1e10, ak.DEFAULT_MASK_VALUE, float(torch.finfo(torch.bfloat16).min)])
@pytest.mark.parametrize("hq,hkv,t,s", [(8, 2, 100, 320), (2, 2, 130, 700)])  # (few K/V tiles: no classes; more: classes)
@pytest.mark.parametrize("rounded", [True, False])
def test_finite_large_masks(value, hq, hkv, t, s, rounded):
  """200 left-padded keys under a finite mask value (a row's first K/V tile lies wholly under it), and rows that are masked
  throughout: with one value for all keys those are the unmasked softmax, or uniform where the value swallows the logits."""
  q, k, v = _inputs(hq, hkv, t, s)
  m = torch.full((t, s), value, device=DEV).triu(1 + s - t)
  m[:, :200] = value
  m[t // 2] = value
  m[t - 1] = value
  mask = m.to(torch.bfloat16).repeat(hq // hkv, 1)[None, None]
  if rounded:
    out = ak.dense_attention(q, k, v, None, None, mask)
  else:
    out, _ = ak.flash_attention(q, k, v, 0, mask=mask)
  assert ak.kernel_status(DEV) == 0
  if not rounded:  # (logits are fp32 here: the sum with the mask is rounded to that)
    lg = ((q.reshape(1, hkv, -1, 128).float() @ k.float().transpose(2, 3)) / math.sqrt(128) + mask.float()).double()
    want = (torch.softmax(lg, -1) @ v.double()).reshape(q.shape)
  else:
    want = _softmax_rows(q, k, v, mask, True)
  _check(out, want)
