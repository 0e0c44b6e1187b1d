"""CPU: the checks of the native host side.  Shapes are looked at before devices, so a CPU tensor of the right
shape is refused for its device and one of the wrong shape for its shape."""

import pytest
import torch

BF = torch.bfloat16
B, HQ, H, S, D = 3, 8, 2, 16, 128


def _native():
  from jetstream_pytorch_b200 import _lib

  return _lib.native


def _step(dtype=BF):
  return (torch.zeros(B, HQ, 1, D, dtype=BF), torch.zeros(B, H, 1, D, dtype=dtype), torch.zeros(B, H, 1, D, dtype=dtype))


def _calls():
  """name -> (call(q, xk, xv, batch, heads, dim, scale tokens, kept batch)), each with the shapes of the cache as given"""

  def int8_cache(b, h, d, s):
    return tuple(torch.zeros(b, h, S, d, dtype=torch.int8) for _ in range(2)) + tuple(torch.ones(b, 1, s, 1, dtype=BF) for _ in range(2))

  end = torch.zeros(B, dtype=torch.int32)

  def fused(q, xk, xv, b=B, h=H, d=D, s=S, kept=B):
    outs = tuple(torch.zeros(2, kept, H, 1, D, dtype=torch.int8) for _ in range(2)) + tuple(torch.zeros(2, kept, 1, 1, 1, dtype=BF) for _ in range(2))
    _native().update_attend(q, xk, xv, int8_cache(b, h, d, s), 0, None, end, False, 0, False, outs, True, None, None)

  def lazy(q, xk, xv, b=B, h=H, d=D, s=S, kept=B):
    keep = [torch.zeros(2, kept, H, 1, D, dtype=BF) for _ in range(2)]
    k, v = (torch.zeros(2, b, h, S, d, dtype=BF) for _ in range(2))
    _native().attend_lazy(q, xk, xv, k, v, 1, end, *keep)

  def lazy_int8(q, xk, xv, b=B, h=H, d=D, s=S, kept=B):
    scale = torch.ones(kept, dtype=BF)
    _native().attend_lazy_int8(q, int8_cache(b, h, d, s), 0, end, xk.to(torch.int8), xv.to(torch.int8), scale, scale)

  return {"update_attend": fused, "attend_lazy": lazy, "attend_lazy_int8": lazy_int8}


@pytest.mark.parametrize("name", ["update_attend", "attend_lazy", "attend_lazy_int8"])
def test_step_shapes(name):
  call = _calls()[name]
  q, xk, xv = _step()
  with pytest.raises(ValueError, match="CUDA tensors only"):
    call(q, xk, xv)  # all shapes agree
  for wrong in (dict(b=B - 1), dict(d=64)):
    with pytest.raises(AssertionError, match="batch or head_dim"):
      call(q, xk, xv, **wrong)
  with pytest.raises(ValueError, match="token must be"):
    call(q, xk, xv, h=H * 2)  # more KV heads than the token has
  with pytest.raises(ValueError, match="token must be"):
    call(q, xk[:1], xv[:1])
  with pytest.raises(ValueError, match="token must be"):
    call(q, xk, xv[:, :1])
  with pytest.raises(ValueError, match="one query token"):
    call(torch.zeros(B, HQ, 2, D, dtype=BF), xk, xv)
  with pytest.raises(ValueError):
    call(q, xk, xv, kept=B - 1)
  if name != "attend_lazy":
    with pytest.raises(AssertionError, match="scales"):
      call(q, xk, xv, s=S - 1)


def test_block_tables_need_one_row_per_slot():
  i32 = dict(dtype=torch.int32)
  begin = _native().engine_begin
  with pytest.raises(ValueError, match="one row per slot"):
    begin(torch.zeros(4, **i32), torch.zeros(1, **i32), 64, 16, None, False, 0)
  with pytest.raises(ValueError, match="one row per slot"):
    begin(torch.zeros(2, 2, **i32), torch.zeros(4, **i32), 64, 16, None, False, 0)
  with pytest.raises(ValueError, match="the mask is"):
    begin(torch.zeros(4, **i32), torch.zeros(4, **i32), 64, 16, torch.zeros(3, 64), False, 0)


def test_block_tables_of_a_broadcast_position_go_through_tensor_operations(monkeypatch):
  """One `input_pos` for all slots: the tensor operations broadcast it, the launch reads one per slot."""
  from types import SimpleNamespace

  from jetstream_pytorch_b200 import _lib, engine

  class OnGpu:  # (a CPU tensor that says that it lies on a GPU)
    def __init__(self, t):
      self.t = t

    is_cuda = True

    def __getattr__(self, name):
      return getattr(self.t, name)

    def __add__(self, other):
      return self.t + other.t

  taken = []
  monkeypatch.setattr(_lib, "native", SimpleNamespace(engine_begin=lambda *a: taken.append(a)))
  env = SimpleNamespace(cache_len=64, block_size=16)
  start, pos = torch.tensor([0, 5, 60], dtype=torch.int32), torch.tensor([7], dtype=torch.int32)
  got = engine.precompute_ragged_block_indices(env, OnGpu(start), OnGpu(pos))
  want = engine.precompute_ragged_block_indices(env, start, pos.expand(3).contiguous())
  assert not taken
  assert all(torch.equal(x, y) for x, y in zip(got, want))
  engine.precompute_ragged_block_indices(env, OnGpu(start), OnGpu(pos.expand(3).contiguous()))
  assert len(taken) == 1


def test_end_of_a_step_needs_a_token_of_logits():
  i32 = [torch.zeros(2, dtype=torch.int32) for _ in range(3)]
  with pytest.raises(ValueError, match="logits are"):  # (the row before the first one would be read)
    _native().engine_end(torch.zeros(2, 0, 5), *i32, 64, None, False, 0)
  with pytest.raises(ValueError, match="elsewhere"):
    _native().engine_end(torch.zeros(2, 1, 5), *(t.to("meta") for t in i32), 64, None, False, 0)


def test_exceptions_of_tensor_calls_keep_their_types():
  with pytest.raises(IndexError):
    _native().rmsnorm(torch.zeros((), dtype=BF), torch.zeros(8, dtype=BF), 1e-6, False)


@pytest.mark.gpu
def test_out_of_memory_is_torchs():
  """2 TB: refused by the allocator, nothing is launched."""
  x = torch.zeros(1, 8, dtype=BF, device="cuda").expand(1 << 37, 8)
  with pytest.raises(torch.OutOfMemoryError):
    _native().silu_mul(x, x, False)


def test_empty_extents_are_refused():
  """(an integer division by zero would end the process)"""
  n, e = _native(), torch.zeros(4, 0, dtype=BF)
  w, sc = torch.zeros(8, 0, dtype=torch.int8), torch.zeros(8, dtype=BF)
  for call in (lambda: n.rmsnorm(e, e[0], 1e-6, False), lambda: n.silu_mul(e, e, False), lambda: n.linear(e, w, sc, None),
               lambda: n.gate(e, w, sc, w, sc, None), lambda: n.linear_from_levels(e, e, w, sc)):
    with pytest.raises(ValueError, match="0 features"):
      call()
  q, k = torch.zeros(2, 8, 1, D, dtype=BF), torch.zeros(2, 0, S, D, dtype=BF)
  end, mask = torch.zeros(2, dtype=torch.int32), torch.zeros(2, 1, 1, S, dtype=BF)
  for call in (lambda: n.ragged(q, k, k, 0, None, end, None, None, True, False), lambda: n.dense(q, k, k, None, None, mask),
               lambda: n.paged(q[:, :, 0], k.reshape(0, 2, S, D), k.reshape(0, 2, S, D), end, end.reshape(2, 1), 1.0, None, None)):
    with pytest.raises(ValueError, match="without KV heads"):
      call()
  assert n.fused_ok(q, torch.zeros(2, 0, 1, D, dtype=BF), None) is False
  with pytest.raises(ValueError, match="blocks of 0"):
    n.engine_begin(end, end, 64, 0, None, False, 0)


def test_cpu_tensors_are_refused_with_one_message():
  n, x = _native(), torch.zeros(4, 128, dtype=BF)
  w, sc = torch.zeros(8, 128, dtype=torch.int8), torch.zeros(8, dtype=BF)
  for call in (lambda: n.rmsnorm(x, x[0], 1e-6, False), lambda: n.silu_mul(x, x, True), lambda: n.linear(x, w, sc, None)):
    with pytest.raises(ValueError, match="CUDA tensors only"):
      call()


def test_page_table_walk_takes_the_managers_extents(monkeypatch):
  """As many slots and pages as the manager has, not as many as the table happens to have rows and columns."""
  from types import SimpleNamespace

  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200.page_attention_manager import PageAttentionManager

  lens, table = torch.zeros(4, dtype=torch.int32), torch.zeros(3, 6, dtype=torch.int32)
  walk = _native().page_token_indices
  for few in ((lens[:2], table), (lens, table[:2])):
    with pytest.raises(ValueError, match="lengths of 3 slots"):
      walk(*few, 16, 3, 6)
  seen = []
  monkeypatch.setattr(_lib, "native", SimpleNamespace(page_token_indices=lambda *a: seen.append(a[2:])))
  PageAttentionManager(3, 20, 16, 6).get_page_token_indices_device(lens, table)
  assert seen == [(16, 3, 6)]


def test_stacked_insert_needs_a_scale_per_layer():
  """Scalers of fewer layers than the prefix: left to the loop over the layers, which raises IndexError for the missing one."""
  prefix = [(torch.zeros(1, H, 5, D, dtype=BF),) * 2 for _ in range(3)]
  caches = [(torch.zeros(3, B, H, S, D, dtype=torch.int8),) * 2]
  assert _native().insert_dense(prefix, caches, [(torch.ones(2, B, 1, S, 1, dtype=BF),) * 2], 0, 0, False, True) is False
  assert _native().insert_dense(prefix, caches, [(torch.ones(B, 1, S, 1, dtype=BF),) * 2], 0, 0, False, True) is False
