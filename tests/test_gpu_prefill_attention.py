"""Prefill-shaped attention (many query rows per KV head, bf16, head_dim 128) on
the tensor-core kernel against a plain fp32 reference of the same op.

Tolerance: q, K, V are bf16 and the result is rounded to bf16 (2^-9 relative).
With the logit roundings of `dense_attention` two implementations whose fp32 dot
products differ in the last bits may round a logit to neighbouring bf16 values.  A
logit of magnitude 2 .. 4 has a step of 2^-6, which changes its probability by
e^(2^-6) - 1 = 1.6 %, and with few keys a row hangs on one such probability: a single
row may be off by 2^-6 + 2^-8 = 2e-2 in the 2-norm.  Such flips are rare (the dot
products agree to 2^-20), so all rows together agree to 5e-3, the size of the
output's own rounding.  `flash_attention` has no such rounding: 6e-3 per row.
"""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(b, hq, hkv, t, s, seed, transposed):
  g = torch.Generator(device=DEV).manual_seed(seed)

  def heads(n, h):
    x = torch.randn((b, n, h, 128), generator=g, device=DEV, dtype=torch.bfloat16)
    return x.transpose(1, 2) if transposed else x.transpose(1, 2).contiguous()

  return heads(t, hq), heads(s, hkv), heads(s, hkv), g


def _check_rows(got, want, rel, rel_all=5e-3):
  got, want = got.double(), want.double()
  err = (got - want).norm(dim=-1)
  worst = float((err / (want.norm(dim=-1) + 1e-9)).max())
  whole = float((got - want).norm() / want.norm())
  assert worst <= rel and whole <= rel_all, (worst, whole)


def _mask(kind, rep, t, s, g):
  if kind == "none":
    return None
  if kind == "causal":  # the queries are the last t of s tokens
    m = torch.full((t, s), float("-inf"), device=DEV).triu(1 + s - t)
  elif kind == "random":
    m = torch.where(torch.rand((t, s), generator=g, device=DEV) < 0.5, float("-inf"), torch.randn((t, s), generator=g, device=DEV))
    m[:, 0] = 0
    m[t // 2] = float("-inf")  # a fully masked row gives zeros
  else:  # one broadcast row: zeros, then -inf
    m = torch.zeros((1, s), device=DEV)
    m[:, s // 3:] = float("-inf")
    return m.to(torch.bfloat16)[None, None]
  return m.to(torch.bfloat16).repeat(rep, 1)[None, None]


@pytest.mark.parametrize("b,hq,hkv,t,s,kind,transposed", [
    (1, 2, 1, 128, 128, "none", False),       # one item, one K/V tile
    (1, 32, 8, 1024, 1024, "causal", True),   # the tiled mask of a grouped model, classes and skipped tiles
    (1, 8, 8, 300, 300, "causal", True),      # one query head per KV head, ragged tiles
    (2, 4, 1, 129, 129, "causal", False),     # one row into the second tile, contiguous queries
    (1, 3, 1, 128, 641, "causal", False),     # odd number of row tiles, more keys than queries, one key into a tile
    (1, 8, 1, 17, 17, "causal", True),        # the smallest prompts, mask rows not 16-byte aligned
    (1, 4, 1, 520, 520, "random", True),      # mixed tiles everywhere, a row without a single key
    (2, 8, 2, 70, 600, "broadcast", True),    # one mask row for all
    (1, 40, 1, 1, 512, "none", False),        # many grouped heads, one token
    (10, 10, 10, 650, 650, "causal", True),   # more items than SMs, an odd number of row tiles of a head: neighbours share an item
    (1, 4, 4, 500, 500, "causal", True),      # four blocks of tokens of a head on its own: longest and shortest share an item
    (1, 3, 1, 300, 300, "causal", True),      # nine row tiles: the middle one is alone
])
@pytest.mark.parametrize("scales", ["none", "ones", "random", "random_f32"])
def test_dense_attention_matches_the_reference(b, hq, hkv, t, s, kind, transposed, scales):
  from jetstream_pytorch_b200 import attention_kernel as ak

  q, k, v, g = _inputs(b, hq, hkv, t, s, 7, transposed)
  mask = _mask(kind, hq // hkv, t, s, g)
  ks = vs = None
  if scales == "ones":
    ks = vs = torch.ones((b, 1, s, 1), dtype=torch.bfloat16, device=DEV)
  elif scales != "none":
    dt = torch.float32 if scales == "random_f32" else torch.bfloat16
    ks, vs = (0.5 + torch.rand((2, b, 1, s, 1), generator=g, device=DEV)).to(dt)
  out = ak.dense_attention(q, k, v, ks, vs, mask)
  assert out.is_contiguous() and out.shape == q.shape
  assert ak.kernel_status(DEV) == 0
  # reference: the logit chain in bf16 steps, the rest in fp32
  rep = hq // hkv
  qg = q.reshape(b, hkv, rep * t, 128).float()
  lg = (qg @ k.float().transpose(2, 3)).to(torch.bfloat16)
  lg = (lg.float() / math.sqrt(128)).to(torch.bfloat16)
  if ks is not None:
    lg = (lg.float() * ks.float().reshape(b, 1, 1, s)).to(torch.bfloat16)
  if mask is not None:
    lg = (lg.float() + mask.float()).to(torch.bfloat16)
  p = torch.nan_to_num(torch.softmax(lg.float(), dim=-1))
  if vs is not None:
    p = p * vs.float().reshape(b, 1, 1, s)
  want = (p @ v.float()).reshape(b, hq, t, 128)
  _check_rows(out, want, 2e-2)


@pytest.mark.parametrize("b,hq,hkv,t,s,kind", [(1, 16, 4, 256, 256, "causal"), (2, 6, 2, 200, 450, "random"), (1, 8, 1, 65, 130, "none")])
def test_flash_attention_statistics(b, hq, hkv, t, s, kind):
  """Without the logit roundings; m and l are those of the true row maximum although the kernel keeps a lazy one."""
  from jetstream_pytorch_b200 import attention_kernel as ak

  q, k, v, g = _inputs(b, hq, hkv, t, s, 11, True)
  q = q * 4  # spread the logits so that the running maximum moves a lot
  mask = _mask(kind, hq // hkv, t, s, g)
  out, (m, l) = ak.flash_attention(q, k, v, 0, mask=mask)
  assert ak.kernel_status(DEV) == 0
  lg = (q.reshape(b, hkv, -1, 128).float() @ k.float().transpose(2, 3)) / math.sqrt(128)
  if mask is not None:
    lg = lg + mask.float()
  want_m = lg.amax(-1)
  p = torch.exp(lg - want_m.clamp(min=-1e30)[..., None])
  want = torch.nan_to_num((p @ v.float()) / p.sum(-1, keepdim=True)).reshape(b, hq, t, 128)
  _check_rows(out, want, 6e-3)
  want_m, want_l = want_m.reshape(m.shape), p.sum(-1).reshape(l.shape)
  live = torch.isfinite(want_m)
  assert torch.allclose(m[live], want_m[live], atol=1e-3, rtol=1e-5)
  assert torch.allclose(l[live], want_l[live], rtol=1e-3)
  assert bool((l[~live] == 0).all()) and bool((m[~live] == float("-inf")).all())
