"""The int8 decode kernel's division of work: whole segments longest first with tickets, cut segments (one item per CTA, or more
than one), equal shares, one or two groups of 128 sequences, lengths around the 128-token tile and the 256-token round, rings that
wrap.  Each case runs three times with other lengths in between: the ticket counter has to come round to zero."""

import math

import pytest
import torch

from parity_tools import attention_close, describe

pytestmark = pytest.mark.gpu

DEV = "cuda"
EDGES = (0, 1, 127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512)


def _lengths(kind, b, s, g):
  if kind == "equal":
    return torch.full((b,), s)
  if kind == "one long":
    n = torch.randint(0, 3, (b,), generator=g)
    n[b // 2] = s
    return n
  if kind == "edges":
    return torch.tensor([min(EDGES[i % len(EDGES)], s) for i in range(b)])
  return torch.randint(0, s + 1, (b,), generator=g)


@pytest.mark.parametrize("kind,b,hq,hkv,s,ring", [
    ("spread", 96, 64, 8, 1024, False),   # more segments than CTAs: tickets
    ("spread", 60, 8, 8, 2048, False),    # a few more segments than CTAs, long ones cut
    ("equal", 60, 16, 8, 512, False),     # the same with one length: equal shares
    ("one long", 40, 8, 1, 4096, False),  # one segment cut into many pieces
    ("spread", 5, 32, 8, 2048, False),    # one item per CTA
    ("edges", 26, 64, 8, 512, False),
    ("edges", 130, 8, 2, 512, False),     # a second group of sequences
    ("spread", 257, 4, 1, 256, False),    # more sequences than are sorted
    ("one long", 3, 8, 1, 16640, False),  # more tiles than are sorted
    ("spread", 33, 32, 32, 640, True),
    ("edges", 13, 16, 8, 520, True),
])
def test_every_token_of_every_segment(kind, b, hq, hkv, s, ring):
  from jetstream_pytorch_b200 import attention_kernel as ak

  g = torch.Generator().manual_seed(b * hq + s)
  d, rep = 128, hq // hkv
  q = torch.randn(b, hq, 1, d, generator=g).to(torch.bfloat16).to(DEV)
  k, v = (torch.randint(-127, 128, (b, hkv, s, d), generator=g, dtype=torch.int8).to(DEV) for _ in range(2))
  ks, vs = ((torch.rand(b, 1, s, 1, generator=g) * 0.01 + 0.01).to(torch.bfloat16).to(DEV) for _ in range(2))
  for turn in range(3):
    n = _lengths(kind if turn != 1 else "spread", b, s, g)
    first = torch.randint(0, s, (b,), generator=g) if ring else torch.zeros(b, dtype=torch.int64)
    if ring:
      n = n.clamp(max=s - 1)
      start, end = first.to(torch.int32).to(DEV), ((first + n) % s).to(torch.int32).to(DEV)
    else:
      start, end = None, n.to(torch.int32).to(DEV)
    out, (m, l) = ak.ragged_mha(q, k, v, 0, start, end, None, None, ks, vs, ring=ring)
    at = torch.arange(s, device=DEV)[None, :]
    valid = ((at - first.to(DEV)[:, None]) % s < n.to(DEV)[:, None])[:, None, None, :]
    x = (q.float().reshape(b, hkv, rep, d) @ (k.float() * ks.float()).transpose(2, 3)) / math.sqrt(d)
    x = x.masked_fill(~valid, -math.inf)
    top = x.amax(-1, keepdim=True)
    p = torch.where(valid, torch.exp(x - torch.where(top == -math.inf, 0.0, top)), 0.0)
    den = p.sum(-1, keepdim=True)
    want = torch.where(den > 0, (p @ (v.float() * vs.float())) / den.clamp_min(1e-30), 0.0).reshape(b, hq, 1, d)
    assert attention_close(out.reshape(b, hq, 1, d), want), describe(out.reshape(b, hq, 1, d), want)
    empty = (n == 0).to(DEV)
    assert (m.reshape(b, hq)[empty] == -math.inf).all() and not l.reshape(b, hq)[empty].any()
    assert torch.allclose(l.reshape(b, hq), den.reshape(b, hq), rtol=1e-3, atol=1e-6)
    assert torch.allclose(m.reshape(b, hq)[~empty], top.reshape(b, hq)[~empty], rtol=1e-3, atol=1e-3)


def _copied_in_front(dst, src):
  """dst = src for int32 [B], by this package's copy kernel: it lets the next launch start before it writes."""
  from jetstream_pytorch_b200 import _lib

  rows = lambda t: t.view(torch.bfloat16).reshape(1, 1, 1, -1)
  spare = torch.empty_like(dst)
  assert _lib.native.insert_dense([(rows(src), rows(src))], [(rows(spare), rows(dst))], None, 0, 0, False, False)


@pytest.mark.parametrize("form", ["dense", "ring", "mask", "paged"])
@pytest.mark.parametrize("b,hq,hkv", [(40, 32, 8), (5, 8, 2), (150, 8, 1)])
def test_lengths_written_by_the_kernel_in_front(form, b, hq, hkv):
  """The list is made from the lengths as they are under the kernel in front and made again when that kernel changed them: other numbers of
  tiles, the same again, none.  Each call's rows equal those of a call whose lengths stood long before, bit for bit."""
  from jetstream_pytorch_b200 import attention_kernel as ak

  s, d, page = 1024, 128, 64
  g = torch.Generator(device=DEV).manual_seed(b)
  q = torch.randn(b, hq, 1, d, generator=g, device=DEV, dtype=torch.bfloat16)
  ks, vs = (torch.rand(b, 1, s, 1, generator=g, device=DEV).mul_(0.01).add_(0.01).to(torch.bfloat16) for _ in range(2))
  if form == "paged":
    k, v = (torch.randint(-127, 128, (hkv, b * s // page, page, d), generator=g, device=DEV, dtype=torch.int8) for _ in range(2))
    ks, vs = ks.reshape(1, -1, page, 1), vs.reshape(1, -1, page, 1)
    table = torch.randperm(b * s // page, generator=g, device=DEV).to(torch.int32).reshape(b, -1)
  else:
    k, v = (torch.randint(-127, 128, (b, hkv, s, d), generator=g, device=DEV, dtype=torch.int8) for _ in range(2))
  start = torch.full((b,), s // 3, dtype=torch.int32, device=DEV)
  mask = torch.empty(b, 1, 1, s, dtype=torch.bfloat16, device=DEV)
  at = torch.arange(s, device=DEV)

  def call(end):
    if form == "paged":
      return ak.call_paged_attention(None, q.squeeze(2), k, v, end, table, k_scaler=ks, v_scaler=vs)
    if form == "mask":
      return ak.dense_attention(q, k, v, ks, vs, mask)
    return ak.ragged_mha(q, k, v, 0, start, end, None, None, ks, vs, ring=form == "ring")[0]

  lens = [torch.randint(1, s + 1, (b,), generator=g, device=DEV, dtype=torch.int32) for _ in range(3)]
  lens += [lens[2].flip(0), torch.zeros_like(lens[0]) + (1 if form == "mask" else 0), torch.full_like(lens[0], s - 1)]
  masks = [torch.zeros_like(mask).masked_fill_((at >= n[:, None])[:, None, None, :], -math.inf) for n in lens]
  want = []
  for n, m in zip(lens, masks):
    mask.copy_(m)
    torch.cuda.synchronize()
    want.append(call(n))
    torch.cuda.synchronize()
  end = torch.empty_like(lens[0])
  got = []
  for turn in range(20):
    for n, m in zip(lens, masks):
      if form == "mask":
        mask.copy_(m)
      else:
        _copied_in_front(end, n)
      got.append(call(end))
  for i, o in enumerate(got):
    assert torch.equal(o, want[i % len(lens)]), i
  assert ak.kernel_status() == 0
