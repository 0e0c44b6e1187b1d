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


def test_probabilities_are_rounded_to_both_sides():
  """V is multiplied by probabilities in two bf16 parts: rounded, their error has no sign.  The mean signed error of the
  rows is compared with that of the scalar kernel (fp32 probabilities).  Well under 1 % of the N = 4 M rounded outputs differ
  between the two, by 2^-8 of their value, so chance keeps the means within 3 sqrt(N / 100) 2^-8 / N = 6e-7; parts that are
  cut instead of rounded shift one of them by 2^-18 = 4e-6."""
  from jetstream_pytorch_b200 import _lib

  t, hq, hkv = 1024, 32, 8
  q, k, v = _inputs(hq, hkv, t, t)
  mask = torch.full((t, t), float("-inf"), device=DEV).triu(1).to(torch.bfloat16).repeat(hq // hkv, 1)[None, None]
  want = _softmax_rows(q, k, v, mask, False)
  bias = []
  for force_generic in (0, 1):
    o, _, _ = ak._flash_decode(q, k, v, mask_mode=_lib.MASK_ADD, mask=mask, mask_strides=(0, t), sm_scale=1 / math.sqrt(128),
                               kv_strides=k.stride()[:3], n_kv_heads=hkv, seq=t, force_generic=force_generic)
    bias.append(float(((o.double() - want) * want.sign()).sum() / want.abs().sum()))
  assert abs(bias[0] - bias[1]) <= 1.5e-6, bias


@pytest.mark.parametrize("hq,hkv,t,s", [(8, 2, 100, 320), (2, 2, 130, 700)])
@pytest.mark.parametrize("rounded", [True, False])
@pytest.mark.parametrize("scaled", [False, True])
def test_values_that_are_not_finite(hq, hkv, t, s, rounded, scaled):
  """Masked keys may hold anything; an attended infinity or NaN reaches the rows that see it and no others.  Against the
  scalar kernel: the same rows finite, and within the tolerance where they are."""
  q, k, v = _inputs(hq, hkv, t, s)
  q = q.transpose(1, 2).contiguous().transpose(1, 2)  # (strided, as a model hands it over)
  from jetstream_pytorch_b200 import _lib

  m = torch.full((t, s), float("-inf"), device=DEV).triu(1 + s - t)
  m[:, :100] = float("-inf")
  mask = m.to(torch.bfloat16).repeat(hq // hkv, 1)[None, None]
  v[:, :, :60, 5] = float("nan")  # masked for every row, in a tile that the rows read
  v[:, :, 60:100] = float("inf")
  v[:, 0, s - 20, 70] = float("inf")  # seen by the last 20 queries of the first group
  v[:, 0, s - 10, 3] = float("nan")
  v[:, hkv - 1, s - 30, 100] = float("-inf")
  scales = (0.5 + torch.rand((2, 1, 1, s, 1), device=DEV)) if scaled else (None, None)
  outs = []
  for force_generic in (0, 1):
    o, _, _ = ak._flash_decode(q, k, v, k_scale=scales[0], v_scale=scales[1], scale_strides=(s, 1), mask_mode=_lib.MASK_ADD, mask=mask,
                               mask_strides=(0, s), sm_scale=1 / math.sqrt(128), kv_strides=k.stride()[:3], n_kv_heads=hkv, seq=s,
                               force_generic=force_generic, logit_rounding=rounded)
    outs.append(o.float())
  assert ak.kernel_status(DEV) == 0
  got, want = outs
  bad = ~torch.isfinite(want)
  assert 0 < int(bad.sum()) < want.numel() // 100
  assert torch.equal(torch.nan_to_num(got[bad], nan=7.0), torch.nan_to_num(want[bad], nan=7.0))
  assert bool(torch.isfinite(got[~bad]).all())
  _check(torch.where(bad, torch.zeros_like(got), got), torch.where(bad, torch.zeros_like(want), want).double())
