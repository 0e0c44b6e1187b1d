"""The decode form of the weight-only int8 layer at the sizes where its tiles, halves, pairs and K splits end."""

import pytest
import torch

from oracle import linear as ol

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows: edges of the groups of 8 and of the padded 16; channels: one, a tile with a few, odd counts, one and two halves, a last
# pair with an empty CTA, several waves; K: one step, fewer steps than splits, splits of unequal length
@pytest.mark.parametrize("m", [1, 8, 9, 17, 96, 127, 128])
@pytest.mark.parametrize("k,n", [(128, 1), (256, 33), (384, 257), (640, 4099), (1152, 1280), (128, 38000), (256, 80001), (2176, 10240)])
def test_rows_channels_and_splits(m, k, n):
  from jetstream_pytorch_b200.layers import WeightOnlyPerChannelQuantizedLinear

  g = torch.Generator().manual_seed(m + n)
  w, s = ol.quantize_weight(torch.randn(n, k, generator=g) * 0.03)
  lin = WeightOnlyPerChannelQuantizedLinear(k, n, device=DEV)
  lin._load_quantized_weights(w, s)
  x = torch.randn(m, k, generator=g).to(torch.bfloat16)
  if m > 1:
    x[m // 2] = 0
  y = lin(x.to(DEV)).cpu()
  assert lin.kernel_status() == 0
  exp = ol.w8a16_linear(x, w, s)
  err = (y.double() - exp.double()).abs()
  assert (err <= ol.w8a16_tolerance(x, w, s)).all(), float(err.max())
  assert m == 1 or not y[m // 2].any()
