"""CPU: the plan of the int8 linear layer's GEMM.  The ranks of a row-parallel layer exchange
their partial sums by tile and split, so their plans must not depend on the GPU they run on."""

import ctypes

import pytest

# clusters that a GPU holds at once, [single CTAs, pairs] by K splits: of one B200, and with a group of SMs short
EVEN = [[0, 148, 74, 45, 33, 26, 22, 15, 15], [0, 74, 33, 22, 15, 0, 0, 0, 0]]
SHORT = [[0, 132, 64, 42, 30, 24, 20, 16, 12], [0, 60, 28, 16, 10, 0, 0, 0, 0]]


def _plan(m, n, k, row_parallel, slots):
  from jetstream_pytorch_b200 import _lib

  flat = (ctypes.c_int * 18)(*(x for row in slots for x in row))
  out = (ctypes.c_int * 5)()
  _lib.check(_lib.lib().jpt_w8a16_plan(m, n, k, row_parallel, flat, out))
  return tuple(out)


@pytest.mark.parametrize("m", [1, 7, 64, 96, 128])
def test_row_parallel_plan_does_not_depend_on_the_gpu(m):
  shapes = [(8192, 1024), (8192, 3584), (4096, 512), (28672, 1024), (1000, 2048), (256, 1024), (262144, 128)]
  for n, k in shapes:
    assert _plan(m, n, k, 1, EVEN) == _plan(m, n, k, 1, SHORT), (n, k)
    pair, split, tile, tiles, kb = _plan(m, n, k, 1, EVEN)
    assert tiles * tile >= n and tiles <= 1024 and (pair + 1) * split <= 8 and kb * split <= k // 128
  # (alone on its GPU the layer does follow it)
  assert any(_plan(m, n, k, 0, EVEN) != _plan(m, n, k, 0, SHORT) for n, k in shapes)
