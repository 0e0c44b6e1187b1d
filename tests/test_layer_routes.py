"""CPU: which launches the layers ask for, with the native host side replaced by a recorder."""

from types import SimpleNamespace

import pytest
import torch

BF = torch.bfloat16


@pytest.fixture
def calls(monkeypatch):
  from jetstream_pytorch_b200 import _lib

  names = []

  def record(name, result):
    def call(*args):
      names.append(name)
      return result(*args)

    return call

  fake = SimpleNamespace(
      gate=record("gate", lambda x, w1, *a: (x.new_zeros(*x.shape[:-1], w1.shape[0]), None)),
      linear=record("linear", lambda x, w, *a: (x.new_zeros(*x.shape[:-1], w.shape[0]), None)),
      silu_mul=record("silu_mul", lambda a, b, levels: (a, None)))
  monkeypatch.setattr(_lib, "native", fake)
  return names


def _block():
  from jetstream_pytorch_b200 import layers

  return layers.FeedForward(128, 256, device="cpu"), torch.zeros(200, 128, dtype=BF)


def test_a_prompt_takes_the_fused_gate(calls):
  block, x = _block()
  block(x)
  assert calls == ["gate", "linear"]


@pytest.mark.parametrize("change", ["hook", "pre_hook", "global_hook", "subclass", "forward"])
def test_projections_that_do_more_are_called(calls, change):
  from jetstream_pytorch_b200 import layers

  block, x = _block()
  seen, handle = [], None
  if change == "hook":
    block.w1.register_forward_hook(lambda m, a, y: seen.append("w1"))
  elif change == "pre_hook":
    block.w3.register_forward_pre_hook(lambda m, a: seen.append("w3"))
  elif change == "global_hook":
    handle = torch.nn.modules.module.register_module_forward_hook(lambda m, a, y: seen.append("any"))
  elif change == "subclass":

    class Adapted(layers.WeightOnlyPerChannelQuantizedLinear):
      def forward(self, x, **kw):
        seen.append("adapted")
        return super().forward(x, **kw)

    block.w3 = Adapted(128, 256, device="cpu")
  else:
    inner = block.w1.forward
    block.w1.forward = lambda x, **kw: (seen.append("w1"), inner(x, **kw))[1]
  try:
    block(x)
  finally:
    if handle:
      handle.remove()
  assert seen and calls == ["linear", "linear", "silu_mul", "linear"]


def test_activations_of_another_width_are_refused(calls):
  from jetstream_pytorch_b200 import layers

  layer = layers.WeightOnlyPerChannelQuantizedLinear(128, 64, device="cpu")
  for shape in [(2, 256), (256, 64), (3, 100)]:
    with pytest.raises(RuntimeError, match="128 input features"):
      layer(torch.zeros(shape, dtype=BF))
  assert not calls
  assert layer(torch.zeros(3, 0, 128, dtype=BF)).shape == (3, 0, 64)
  assert layer(torch.zeros(5, 4, 128, dtype=BF)).shape == (5, 4, 64) and calls == ["linear"]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
def test_kept_token_has_the_default_type(dtype):
  from jetstream_pytorch_b200.cache_manager import Int8KVCacheGenerate

  env = SimpleNamespace(generate_cache_stacked=True, lazy_cache_update=True, new_cache_stacked=True, default_type=dtype)
  cache, scales = torch.zeros(2, 3, 4, 16, 128, dtype=torch.int8), torch.ones(2, 3, 1, 16, 1, dtype=dtype)
  kept = Int8KVCacheGenerate(cache, cache.clone(), scales, scales.clone(), None, env=env)
  assert kept.new_ks.shape == kept.new_vs.shape == (2, 3, 4, 1, 128) and kept.new_ks.dtype == torch.int8
  assert kept.new_k_scaler.shape == (2, 3, 1, 1, 1) and kept.new_k_scaler.dtype == kept.new_v_scaler.dtype == dtype
  assert not kept.new_ks.any() and not kept.new_v_scaler.any()


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("tokens", [1, 2])
def test_a_cache_of_one_token_keeps_its_mask(monkeypatch, int8, tokens):
  """A lazy step over a cache of one token is flash attention under the step's mask and not ragged attention up to `end`."""
  from jetstream_pytorch_b200 import _lib, layers

  env = SimpleNamespace(lazy_cache_update=True, ragged_mha=True, flash_attention=True, page_attention=False, shard_on_batch=False,
                        generate_cache_stacked=True, block_size=16)
  b, h, d = 2, 4, 16
  k = torch.zeros(1, b, h, tokens, d, dtype=torch.int8 if int8 else BF)
  out = torch.zeros(b, h, 1, d)
  native = []
  fake = lambda name: lambda *a: (native.append(name), out)[1]
  monkeypatch.setattr(_lib, "native", SimpleNamespace(attend_lazy=fake("lazy"), attend_lazy_int8=fake("lazy_int8")))
  cache = SimpleNamespace(cache_k=k, cache_v=k, new_ks=k, new_vs=k, keeps_stacked=lambda *a: True, fused_step_supported=lambda *a: False)
  cache.update = (lambda xk, xv, i: (k, k, xk, xv, None, None, None, None)) if int8 else (lambda xk, xv, i: (k[i], k[i]))
  kernel = (layers.Int8KVAttentionKernel if int8 else layers.AttentionKernel)(env, 0)
  masks = []

  def flash(xq, keys, values, layer, k_scaler, v_scaler, mask):
    masks.append(mask)
    return out.to(BF), (torch.zeros(b, h, 1, 1), torch.ones(b, h, 1, 1))

  kernel.flash_attention = flash
  kernel._merge = lambda *a: out
  x = torch.zeros(b, h, 1, d, dtype=BF)
  kernel(x, x, x, "mask", cache, start=torch.zeros(b, dtype=torch.int32), end=torch.ones(b, dtype=torch.int32))
  if tokens == 1:
    assert native == [] and masks[0] == "mask"
  else:
    assert native == ["lazy_int8" if int8 else "lazy"] and not masks
