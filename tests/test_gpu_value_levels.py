"""The fixed-point levels of the int8 decode kernel's probabilities: what their rounding leaves in float32 results."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("even,odd", [(0.03, 0.03), (0.03, 0.001), (0.001, 0.03)])
def test_each_tile_is_rounded_against_its_own_largest_value_scale(even, odd):
  """Queries of zeros: every probability is 1 and the only rounding left is that of scale / (tile's largest scale) to 16 bits: evenly
  distributed, so the error of an output element is Gaussian with the variance below, whatever scales the tile next to it has (one reference for two tiles of
  scales 30 apart: 1.41 of that deviation).  Enough segments that none is cut into single tiles; 65536 elements hardly correlated: the measured
  deviation is within 1 % of it, and float32 sums add less than 2 %."""
  from jetstream_pytorch_b200.cache_manager import Int8KVCacheGenerate
  from jetstream_pytorch_b200.environment import JetEngineEnvironment, JetEngineEnvironmentData

  g = torch.Generator(device=DEV).manual_seed(11)
  b, hkv, s, d = 64, 8, 1024, 128
  lens = 700 + torch.arange(b, device=DEV) * 5  # (six to nine tiles)
  lens[:8] = torch.tensor([1023, 897, 896, 895, 769, 768, 1000, 513], device=DEV)
  codes = torch.randint(-127, 128, (b, hkv, s, d), generator=g, device=DEV, dtype=torch.int8)
  at = torch.arange(s, device=DEV)
  tile = at // 128
  scales = ((torch.rand(b, s, generator=g, device=DEV) * 0.2 + 0.8) * torch.where(tile % 2 == 0, even, odd)).to(torch.bfloat16)
  data = JetEngineEnvironmentData(batch_size=b, cache_sequence_length=s, ring_buffer=False, testing=True, lazy_cache_update=True)
  data.quant_config.enable_kv_quantization = True
  cache = Int8KVCacheGenerate(codes, codes, scales.reshape(b, 1, s, 1), scales.reshape(b, 1, s, 1), lens, env=JetEngineEnvironment(data, device=DEV))
  zeros = torch.zeros(b, hkv, 1, d, dtype=torch.bfloat16, device=DEV)  # (the new token too: scale 0)
  q = torch.zeros(b, hkv, 1, d, dtype=torch.bfloat16, device=DEV)
  out = cache._fused_step(q, zeros, zeros, 0, torch.zeros_like(lens), lens, False, None, None, True)[4]
  assert out.dtype == torch.float32
  valid = (at < lens[:, None]).double()
  w = scales.double() * valid
  want = torch.stack([torch.einsum("s,hsd->hd", w[i], codes[i].double()) / (int(lens[i]) + 1) for i in range(b)])
  err = out[:, :, 0].double() - want
  largest = w.reshape(b, -1, 128).amax(-1)[:, tile] * valid
  square = codes[0].double().pow(2).mean()
  deviation = ((largest**2).sum(1) * square / 12).sqrt() / 65535 / (lens + 1)
  measured = (err / deviation[:, None, None]).pow(2).mean().sqrt()
  assert 0.8 < measured < 1.2, float(measured)


@pytest.mark.parametrize("hq", [1, 4, 8])
def test_dot_products_of_queries_within_a_factor_of_127_are_exact(hq):
  """The unrounded logits of one-token sequences, read from the row maximum: the integer sums are exact, what is left is the conversion and six
  float32 products (2^-24 each).  Rows whose largest value has the mantissa 255, 254 or 128, and scales over the range of bf16."""
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200 import attention_kernel as ak

  g = torch.Generator().manual_seed(hq)
  b, d = 96, 128
  q = torch.randn(b, hq, 1, d, generator=g).to(torch.bfloat16)
  q[0::4, :, :, 7], q[1::4, :, :, 7], q[2::4, :, :, 7] = 255 / 64, -254 / 64, 4.0  # (with mantissas 255, 254, 128: the largest of nearly all rows)
  q = torch.where(q.abs() * 127 < q.abs().amax(-1, keepdim=True), torch.zeros_like(q), q)
  q = (q.double() * 2.0 ** torch.linspace(-90, 60, b).round()[:, None, None, None]).to(torch.bfloat16)
  k = torch.randint(-127, 128, (b, 1, 1, d), generator=g, dtype=torch.int8)
  ks = (torch.rand(b, 1, 1, 1, generator=g) + 0.5).to(torch.bfloat16)
  _, m, _ = ak._flash_decode(q.to(DEV), k.to(DEV), k.to(DEV), k_scale=ks.to(DEV), v_scale=ks.to(DEV), scale_strides=(1, 1),
                             mask_mode=_lib.MASK_LENGTH, end=torch.ones(b, dtype=torch.int32), sm_scale=d**-0.5, kv_strides=(d, d, d),
                             n_kv_heads=1, seq=1)
  want = (q.double() * k.double()).sum(-1).reshape(b, hq) * ks.double().reshape(b, 1) * d**-0.5
  err = (m.reshape(b, hq).double().cpu() - want).abs()
  assert (err <= 7 * 2.0**-24 * want.abs()).all(), float((err / want.abs()).max())
