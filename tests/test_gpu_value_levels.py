"""The fixed-point levels of the int8 decode kernel's probabilities: what their rounding leaves in float32 results."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("even,odd", [(0.03, 0.03), (0.03, 0.001), (0.001, 0.03)])
def test_each_tile_is_rounded_against_its_own_largest_value_scale(even, odd):
  """Queries of zeros: every probability is 1 and the only rounding left is that of scale / (tile's largest scale) to 16 bits: evenly
  distributed, so the error of an output element is Gaussian with the variance below, whatever scales the tile next to it has (one reference for two tiles of
  scales 30 apart: 1.41 of that deviation).  896 elements hardly correlated: the measured deviation is within 3 % of it; float32 sums add less than 2 %."""
  from jetstream_pytorch_b200.cache_manager import Int8KVCacheGenerate
  from jetstream_pytorch_b200.environment import JetEngineEnvironment, JetEngineEnvironmentData

  g = torch.Generator().manual_seed(11)
  lens = torch.tensor([2047, 1920, 1664, 1536, 1281, 1100, 2000])
  b, hkv, s, d = len(lens), 1, 2048, 128
  codes = torch.randint(-127, 128, (b, hkv, s, d), generator=g, dtype=torch.int8)
  tile = torch.arange(s) // 128
  scales = ((torch.rand(b, s, generator=g) * 0.2 + 0.8) * torch.where(tile % 2 == 0, even, odd)).to(torch.bfloat16)
  data = JetEngineEnvironmentData(batch_size=b, cache_sequence_length=s, ring_buffer=False, testing=True, lazy_cache_update=True)
  data.quant_config.enable_kv_quantization = True
  cache = Int8KVCacheGenerate(codes.to(DEV), codes.to(DEV), scales.reshape(b, 1, s, 1).to(DEV), scales.reshape(b, 1, s, 1).to(DEV),
                              lens.to(DEV), env=JetEngineEnvironment(data, device=DEV))
  zeros = torch.zeros(b, hkv, 1, d, dtype=torch.bfloat16, device=DEV)  # (the new token too: scale 0)
  q = torch.zeros(b, 8, 1, d, dtype=torch.bfloat16, device=DEV)
  out = cache._fused_step(q, zeros, zeros, 0, torch.zeros_like(lens).to(DEV), lens.to(DEV), False, None, None, True)[4]
  assert out.dtype == torch.float32
  valid = (torch.arange(s) < lens[:, None]).double()
  w = scales.double() * valid
  want = torch.einsum("bs,bsd->bd", w, codes[:, 0].double()) / (lens[:, None] + 1)
  err = out[:, 0, 0].double().cpu() - want
  largest = w.reshape(b, -1, 128).amax(-1)[:, tile] * valid
  deviation = ((largest**2).sum(1) * codes.double().pow(2).mean() / 12).sqrt() / 65535 / (lens + 1)
  measured = (err / deviation[:, None]).pow(2).mean().sqrt()
  assert measured < 1.2, float(measured)
