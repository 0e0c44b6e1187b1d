"""CPU: which attention calls go to the prefill kernel (host code of the dispatch; nothing is launched)."""

import ctypes

import pytest


def _taken(b, hq, hkv, tq, s, rows_mask):
  from jetstream_pytorch_b200 import _lib

  p = _lib.AttnParams()
  p.q = p.k = p.v = p.o = p.mask = 1 << 20  # (aligned; never read)
  p.q_dtype = p.kv_dtype = _lib._DTYPES[__import__("torch").bfloat16]
  p.B, p.Hq, p.Hkv, p.Tq, p.D, p.S = b, hq, hkv, tq, 128, s
  p.kv_b, p.kv_h, p.kv_s = hkv * s * 128, s * 128, 128
  p.sm_scale = 128 ** -0.5
  if rows_mask:
    p.mask_mode, p.mk_r = _lib.MASK_ADD, s
  else:
    p.mask = None
  return bool(_lib.lib().jpt_flash_attend_strided_q_ok(ctypes.byref(p), hq * tq * 128, tq * 128, 128))


@pytest.mark.parametrize("rows_mask", [False, True])
def test_few_rows_over_many_keys_keep_the_split_kernel(rows_mask):
  for shape in [(1, 40, 1, 1, 8192), (1, 32, 1, 1, 65536), (1, 8, 1, 3, 4096), (1, 8, 1, 3, 16384)]:  # 1.2 to 2 times as slow there
    assert not _taken(*shape, rows_mask), shape
  for shape in [(1, 40, 1, 1, 512), (1, 8, 1, 3, 1024), (1, 64, 8, 4, 8192), (1, 64, 8, 4, 32768), (1, 32, 8, 5, 16384), (1, 8, 1, 64, 16384),
                (1, 32, 8, 1024, 1024), (1, 4, 1, 1024, 1024), (1, 8, 1, 17, 17), (1, 4, 1, 128, 65536)]:
    assert _taken(*shape, rows_mask), shape
