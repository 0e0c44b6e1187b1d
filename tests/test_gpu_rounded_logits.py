"""The logit chain of dense_attention on bf16 tensors (dot product, / sqrt(D), * K scale, + mask, each rounded to bf16) in the int8
decode kernel, read from the row maximum of sequences of one token: bit for bit where the dot product is exact in float32."""

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
D, ROWS = 128, 8


def _row_maxima(x, codes, sm_scale=1.0 / math.sqrt(D)):
  """x [B, 8]: query rows of one value each; codes [B, 128] int8: the token of each sequence.  The logits as the kernel has them."""
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200 import attention_kernel as ak

  b = x.shape[0]
  q = x[:, :, None, None].expand(b, ROWS, 1, D).contiguous().to(DEV)
  k = codes.reshape(b, 1, 1, D).to(DEV)
  one = torch.ones(b, 1, 1, 1, dtype=torch.bfloat16, device=DEV)
  _, m, _ = ak._flash_decode(q, k, k, k_scale=one, v_scale=one, scale_strides=(1, 1), mask_mode=_lib.MASK_LENGTH,
                             end=torch.ones(b, dtype=torch.int32), sm_scale=sm_scale, kv_strides=(D, D, D), n_kv_heads=1, seq=1,
                             logit_rounding=True)
  return m.reshape(b, ROWS).to(torch.bfloat16).cpu()  # (held as a base-2 logarithm: back within 3e-7)


def _codes_of_sum(total, rng):
  """128 codes of the given sum: equal ones, then pairs moved against each other."""
  c = np.full(D, total // D)
  c[: total - c.sum()] += 1
  move = rng.integers(0, 127 - c.max() + 1, D // 2)
  c[0::2] += move
  c[1::2] -= move
  return c


def test_exact_dot_products_next_to_a_tie_are_rounded_as_the_reference_rounds_them():
  # x m-th of 128 .. 255, codes of sum t: the product m t (below 2^22, exact in float32) lies above a tie of its bf16 rounding by 1e-6 ..
  # 8e-6 of itself: more than float32 loses on the way (four roundings: 2.4e-7), less than query levels that do not hold the
  # row's amax exactly.
  rng = np.random.default_rng(5)
  m = np.arange(128, 256)
  xs, codes = [], []
  while len(xs) < 64:
    t = int(rng.integers(2000, 12000))
    p = (m * t).astype(np.int64)
    ulp = 1 << (np.floor(np.log2(p)).astype(np.int64) - 7)
    over = p % ulp - ulp // 2
    near = m[(over > 1e-6 * p) & (over < 8e-6 * p)]
    if near.size:
      xs.append(rng.choice(near, ROWS))
      codes.append(_codes_of_sum(t, rng))
  x = torch.from_numpy(np.stack(xs)).to(torch.bfloat16)
  c = torch.from_numpy(np.stack(codes))
  assert c.abs().max() <= 127
  dot = (x.float() * c.sum(1, keepdim=True)).to(torch.bfloat16)
  want = (dot.float() / math.sqrt(D)).to(torch.bfloat16)
  got = _row_maxima(x, c.to(torch.int8))
  assert torch.equal(got, want), f"{int((got != want).sum())} of {want.numel()} logits differ"


@pytest.mark.parametrize("sm_scale", [1.0 / math.sqrt(D), 1.0 / math.sqrt(96), 1.0 / math.sqrt(160), 0.3, 1.0, 1.7, 3e-3])
def test_the_quotient_is_the_division(sm_scale):
  """Every bf16 mantissa at exponents over the range where the quotient is a normal number, both signs."""
  m = torch.arange(128, 256, dtype=torch.float64)
  exponents = torch.tensor([-100, -31, -9, -8, -7, -1, 0, 3, 30, 60], dtype=torch.float64)
  x = (m[None, :] * 2.0 ** exponents[:, None]).to(torch.bfloat16).reshape(-1, ROWS)
  x[::3] *= -1
  codes = torch.zeros(x.shape[0], D, dtype=torch.int8)
  codes[:, 5] = 1  # the dot product is x itself
  by = np.float32(1) / np.float32(sm_scale)
  want = torch.from_numpy(x.float().numpy() / by).to(torch.bfloat16)
  got = _row_maxima(x, codes, sm_scale)
  assert torch.equal(got, want), f"{int((got != want).sum())} of {want.numel()} logits differ"


@pytest.mark.parametrize("rounded", [True, False])
def test_a_dot_product_beyond_the_range_is_a_logit_of_minus_infinity(rounded):
  """Two tokens, one with a dot product below -3.4e38: it has no weight, and the row is the other token's, whatever the launches before left
  where a second tile's sums would be."""
  from jetstream_pytorch_b200 import attention_kernel as ak

  one = torch.ones(1, 1, 512, 1, dtype=torch.bfloat16, device=DEV)
  for turn in range(3):
    k = torch.zeros(1, 1, 2, D, dtype=torch.int8, device=DEV)
    k[0, 0, 0] = -127
    v = torch.randint(-127, 128, (1, 1, 2, D), dtype=torch.int8, device=DEV)
    q = torch.full((1, 4, 1, D), 3e38, dtype=torch.bfloat16, device=DEV)
    if rounded:
      out = ak.dense_attention(q, k, v, one[:, :, :2], one[:, :, :2], torch.zeros(1, 1, 1, 2, dtype=torch.bfloat16, device=DEV))
    else:
      out = ak.ragged_mha(q, k, v, 0, None, torch.full((1,), 2, dtype=torch.int32, device=DEV), None, None, one[:, :, :2], one[:, :, :2])[0]
    assert torch.equal(out.reshape(4, D), v[0, 0, 1:].to(torch.bfloat16).expand(4, D)), turn
    # sums of full tiles in every column of every SM
    full = torch.full((64, 8, 512, D), 127, dtype=torch.int8, device=DEV)
    ones = one.expand(64, 1, 512, 1).contiguous()
    ak.ragged_mha(torch.ones(64, 64, 1, D, dtype=torch.bfloat16, device=DEV), full, full, 0, None,
                  torch.full((64,), 512, dtype=torch.int32, device=DEV), None, None, ones, ones)
