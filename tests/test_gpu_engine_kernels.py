"""The engine's bookkeeping launches against the tensor operations they stand for, the
inserts of scattered layers against the layers one by one, and the lazy step's token
against the two-partial merge."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _env(**kw):
  from jetstream_pytorch_b200.environment import JetEngineEnvironment, JetEngineEnvironmentData

  return JetEngineEnvironment(JetEngineEnvironmentData(**kw), device=DEV)


@pytest.mark.parametrize("b,s,bk", [(1, 64, 16), (7, 512, 128), (96, 2048, 512), (3, 100, 512), (5, 1000, 64)])
@pytest.mark.parametrize("ring", [False, True])
def test_block_tables_and_mask(b, s, bk, ring):
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200.engine import precompute_ragged_block_indices, update_mask

  env = _env(batch_size=b, cache_sequence_length=s, block_size=bk, ring_buffer=ring)
  g = torch.Generator().manual_seed(b * s)
  start = torch.randint(0, s, (b,), generator=g, dtype=torch.int32)
  pos = torch.randint(0, s, (b,), generator=g, dtype=torch.int32)
  pos[0] = 0
  want = precompute_ragged_block_indices(env, start, pos)  # (the tensor operations, on the CPU)
  for dt in (torch.bfloat16, torch.float32):
    mask = torch.full((b, s), float("-inf"), dtype=dt)
    dmask = mask.to(DEV)
    got = _lib.native.engine_begin(start.to(DEV), pos.to(DEV), s, bk, dmask, ring, s // 3)
    assert torch.equal(dmask.cpu(), update_mask(env, mask, s // 3, pos))
    for x, y in zip(got, want):
      assert x.shape == y.shape and torch.equal(x.cpu(), y)


@pytest.mark.parametrize("b,v", [(1, 5), (3, 1000), (96, 32001), (2, 128256)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_end_of_a_step(b, v, dt):
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200.engine import advance_positions

  g = torch.Generator().manual_seed(v)
  logits = torch.randn(b, 2, v, generator=g).to(dt)
  logits[0, 1, [v // 2, v - 1]] = 9.0  # a tie: the first wins
  if b > 2:
    logits[1, 1, v // 3] = float("nan")  # above everything
    logits[2, 1] = float("-inf")
  tokens, lens = (torch.randint(0, 3, (b, 1), generator=g, dtype=torch.int32) for _ in range(2))
  pos = torch.randint(0, 3, (b,), generator=g, dtype=torch.int32)
  for ring in (False, True):
    env = _env(batch_size=b, cache_sequence_length=64, ring_buffer=ring)
    nt, lo, po, data = _lib.native.engine_end(logits.to(DEV), tokens.to(DEV), lens.to(DEV), pos.to(DEV), 64, None, ring, 0)
    want_pos, want_lens = advance_positions(env, pos, lens)
    assert torch.equal(nt.cpu()[:, 0], torch.argmax(logits[:, 1].float(), dim=-1).to(torch.int32))
    assert torch.equal(po.cpu(), want_pos) and torch.equal(lo.cpu(), want_lens)
    assert torch.equal(data.cpu(), torch.cat([tokens, torch.ones_like(tokens), want_lens], dim=-1))


@pytest.mark.parametrize("nl,quant", [(1, True), (5, False), (50, True)])  # (48 layers are one launch)
@pytest.mark.parametrize("paged", [False, True])
def test_inserts_of_scattered_layers(nl, quant, paged):
  from jetstream_pytorch_b200 import _lib, insert
  from jetstream_pytorch_b200.page_attention_manager import PageAttentionManager

  g = torch.Generator(device=DEV).manual_seed(nl)
  h, n, d, s, ps, pages = 2, 37, 128, 64, 16, 9
  dt = torch.int8 if quant else torch.bfloat16
  prefix = [tuple(torch.randn((1, n, h, d), generator=g, device=DEV, dtype=torch.bfloat16).transpose(1, 2) for _ in range(2))
            for _ in range(nl)]

  def caches():
    shape, sshape = ((h, pages, ps, d), (1, pages, ps, 1)) if paged else ((3, h, s, d), (3, 1, s, 1))
    c = [tuple(torch.full(shape, 3, dtype=dt, device=DEV) for _ in range(2)) for _ in range(nl)][::-1]
    sc = [tuple(torch.ones(sshape, dtype=torch.bfloat16, device=DEV) for _ in range(2)) for _ in range(nl)]
    return c, sc if quant else None

  (ca, sa), (cb, sb) = caches(), caches()
  if paged:
    order = [7, 2, 5]
    PageAttentionManager(2, pages, ps, 4).insert_prefill_cache(prefix, ca, order, decode_scales=sa)
    for i in range(nl):
      PageAttentionManager(2, pages, ps, 4).insert_prefill_cache(prefix[i:i + 1], cb[i:i + 1], torch.tensor(order, device=DEV),
                                                                 decode_scales=sb[i:i + 1] if quant else None)
  else:
    before = _lib.lib().jpt_launch_count()
    assert _lib.native.insert_dense(prefix, ca, sa, 1, 50, True, False)
    assert _lib.lib().jpt_launch_count() - before == -(-nl // 48)
    for i in range(nl):
      insert.insert_dense(*prefix[i], *cb[i], 1, 50, wrap=True, k_scaler=sb[i][0] if quant else None, v_scaler=sb[i][1] if quant else None)
  for x, y in zip(ca + (sa or []), cb + (sb or [])):
    assert torch.equal(x[0], y[0]) and torch.equal(x[1], y[1])


def test_inserts_of_narrow_prefixes_take_no_longer_than_wide_ones():
  """A prefix of 1 or 2 KV heads has an eighth or a quarter of the bytes of one of 8 and about its time (1.1 of it: a CTA per token); 1.5 leaves
  room for the clock.  (With a wait at the start of each of those CTAs it was 2.2.)"""
  from jetstream_pytorch_b200 import _lib

  def best_time(h, n=1900, nl=32):
    prefix = [tuple(torch.randn(1, n, h, 128, device=DEV, dtype=torch.bfloat16).transpose(1, 2) for _ in range(2)) for _ in range(nl)]
    caches = [tuple(torch.zeros(1, h, 2048, 128, dtype=torch.int8, device=DEV) for _ in range(2)) for _ in range(nl)]
    scales = [tuple(torch.ones(1, 1, 2048, 1, dtype=torch.bfloat16, device=DEV) for _ in range(2)) for _ in range(nl)]
    times = []
    for _ in range(8):
      a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
      a.record()
      for _ in range(20):
        assert _lib.native.insert_dense(prefix, caches, scales, 0, 0, False, False)
      b.record()
      b.synchronize()
      times.append(a.elapsed_time(b))
    return min(times)

  wide = best_time(8)
  for h in (1, 2):
    assert best_time(h) < 1.5 * wide


@pytest.mark.parametrize("b,hq,hkv,d,dt", [(1, 4, 1, 128, torch.bfloat16), (3, 8, 8, 128, torch.bfloat16), (2, 6, 3, 20, torch.float32)])
@pytest.mark.parametrize("int8", [False, True])
def test_lazy_token_joins_the_cache(b, hq, hkv, d, dt, int8):
  """Against the formulas in fp32.  Tolerance: the attention rows over the cache are rounded to bf16 (2^-9 of a value
  of order one) before they are joined."""
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200 import attention_kernel as ak

  g = torch.Generator(device=DEV).manual_seed(hq)
  s = 200
  q, xk, xv = (torch.randn((b, n, 1, d), generator=g, device=DEV).to(dt) for n in (hq, hkv, hkv))
  k, v = (torch.randn((b, hkv, s, d), generator=g, device=DEV).to(dt) for _ in range(2))
  end = torch.tensor([0, s, 77][:b], dtype=torch.int32, device=DEV)  # an empty slot among them
  ks = vs = torch.ones(b, device=DEV)
  if int8:
    k, v, kq, vq = ((x.float() * 30).round().clamp(-127, 127).to(torch.int8) for x in (k, v, xk, xv))
    sc = torch.full((b, 1, s, 1), 1 / 30, device=DEV, dtype=dt)
    ks, vs = (torch.rand((2, b), generator=g, device=DEV) * 0.01 + 0.03).to(dt)
    out = _lib.native.attend_lazy_int8(q, (k, v, sc, sc), 0, end, kq, vq, ks.reshape(b, 1, 1, 1), vs.reshape(b, 1, 1, 1))
    o1, (m1, l1) = ak.ragged_mha(q, k, v, 0, None, end, None, None, sc, sc)
    xk, xv = kq, vq
  else:
    keep_k, keep_v = (torch.zeros((2, b, hkv, 1, d), dtype=dt, device=DEV) for _ in range(2))
    out = _lib.native.attend_lazy(q, xk, xv, torch.stack([k, k]), torch.stack([v, v]), 1, end, keep_k, keep_v)
    assert torch.equal(keep_k[1], xk) and torch.equal(keep_v[1], xv) and not keep_k[0].any()
    o1, (m1, l1) = ak.ragged_mha(q, k, v, 0, None, end)
  rep = hq // hkv
  o1, m1, l1 = o1.float().reshape(b, hq, 1, d), m1.reshape(b, hq, 1, 1), l1.reshape(b, hq, 1, 1)
  xk, xv = xk.float().repeat_interleave(rep, 1), xv.float().repeat_interleave(rep, 1)
  m2 = (q.float() * xk).sum(-1, keepdim=True) / math.sqrt(d) * ks.float().reshape(b, 1, 1, 1)
  top = torch.maximum(m1, m2)
  w1, w2 = torch.exp(m1 - top) * l1, torch.exp(m2 - top)
  want = (w1 * o1 + w2 * xv * vs.float().reshape(b, 1, 1, 1)) / (w1 + w2)
  assert torch.allclose(out, want, atol=1e-5, rtol=1e-4)
