"""The weight-only int8 layers on prompts (more than 128 rows: the tile kernel)
against the oracle, within the layer's own tolerance."""

import pytest
import torch

from oracle import linear as ol

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(n, k, g):
  from jetstream_pytorch_b200.layers import WeightOnlyPerChannelQuantizedLinear

  w, s = ol.quantize_weight(torch.randn(n, k, generator=g) * 0.03)
  lin = WeightOnlyPerChannelQuantizedLinear(k, n, device=DEV)
  lin._load_quantized_weights(w, s)
  return lin, w, s


# one row into a second block, row counts that are no multiple of eight, a channel tile with one channel, the shortest K
@pytest.mark.parametrize("m,k,n", [(129, 128, 256), (130, 384, 257), (257, 640, 100), (1000, 256, 520), (200, 4096, 1280), (1000, 128, 5121)])  # (the last: 168 tiles, more than one of some CTAs)
def test_many_rows_match_the_oracle(m, k, n):
  g = torch.Generator().manual_seed(m + n)
  lin, w, s = _layer(n, k, g)
  x = torch.randn(m, k, generator=g).to(torch.bfloat16)
  x[5] = 0
  y = lin(x.to(DEV)).cpu()
  assert lin.kernel_status() == 0
  exp = ol.w8a16_linear(x, w, s)
  err = (y.double() - exp.double()).abs()
  assert (err <= ol.w8a16_tolerance(x, w, s)).all(), float(err.max())
  assert (y == exp).float().mean() > 0.95
  assert not y[5].any()


@pytest.mark.parametrize("m,dim,hidden", [(129, 256, 384), (333, 512, 200 * 128), (700, 384, 128)])
def test_gate_of_a_prompt_equals_the_layers_one_by_one(m, dim, hidden):
  """The fused projections and gate against the two layers (each checked above) followed by the gate kernel: the same
  sums, the same roundings, the same bits."""
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200.layers import silu_mul

  g = torch.Generator().manual_seed(m)
  w1, w3 = _layer(hidden, dim, g)[0], _layer(hidden, dim, g)[0]
  x = torch.randn(m, dim, generator=g).to(torch.bfloat16).to(DEV)
  h, _ = _lib.native.gate(x, w1.weight, w1.weight_scaler, w3.weight, w3.weight_scaler)
  assert torch.equal(h, silu_mul(w1(x), w3(x)))


@pytest.mark.parametrize("m,k", [(296, 4096), (297, 8192), (1000, 264), (301, 5120)])
def test_rmsnorm_of_a_prompt(m, k):
  """Equal to a neighbouring bf16 value at most (the fp32 sum is taken in another order)."""
  from jetstream_pytorch_b200.layers import RMSNorm

  g = torch.Generator().manual_seed(k)
  norm = RMSNorm(k, device=DEV)
  w = (1 + 0.1 * torch.randn(k, generator=g)).to(torch.bfloat16)
  norm.weight.data.copy_(w)
  x = torch.randn(m, k, generator=g).to(torch.bfloat16)
  y, exp = norm(x.to(DEV)).cpu(), ol.rmsnorm(x, w, norm.eps)
  assert torch.allclose(y.float(), exp.float(), rtol=2.0 ** -6, atol=0)
  assert (y == exp).float().mean() > 0.99


def test_a_prompt_leaves_no_scratch_behind():
  """What a layer keeps is the workspace of at most 128 rows, whatever came before; its status word reports the last call."""
  from jetstream_pytorch_b200 import _lib, layers

  k, n = 512, 640
  block = layers.FeedForward(k, n, device="cuda")
  most = {m: _lib.lib().jpt_w8a16_linear_workspace_bytes(128, m.out_features, m.in_features) for m in (block.w1, block.w2, block.w3)}
  small, large = (torch.randn(rows, k, device="cuda").to(torch.bfloat16) for rows in (5, 3000))
  want = block.w1(small)
  for x in (large, small, large):
    assert block(x).shape == x.shape
    assert block.w1(x).shape == (x.shape[0], n)
    for layer, limit in most.items():
      assert layer._workspace is None or layer._workspace.numel() <= limit
    assert block.w1.kernel_status() == 0 and block.w2.kernel_status() == 0
  assert torch.equal(block.w1(small), want)  # (the short call grows what a prompt left it)


def test_levels_outlive_another_call_of_a_layer_that_read_them():
  """One level split for two layers, with a call on other activations in between."""
  from jetstream_pytorch_b200 import layers

  g = torch.Generator().manual_seed(3)
  w1, w3 = (_layer(320, 256, g)[0] for _ in range(2))
  x, other = (torch.randn(9, 256, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
  want = w3(x)
  levels = layers.ActivationLevels.of(x)
  w1(x, levels=levels)
  assert w1.kernel_status() == 0
  w1(other)
  assert torch.equal(w3(x, levels=levels), want)
