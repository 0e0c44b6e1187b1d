"""The attention scratch of CUDA graphs."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(b, hq, hkv, s, seed):
  g = torch.Generator(device=DEV).manual_seed(seed)
  q = torch.randn((b, hq, 1, 128), generator=g, device=DEV, dtype=torch.bfloat16)
  k, v = (torch.randn((b, hkv, s, 128), generator=g, device=DEV, dtype=torch.bfloat16) for _ in range(2))
  return q, k, v, torch.randint(1, s, (b,), generator=g, device=DEV, dtype=torch.int32)


def test_a_graph_keeps_the_scratch_it_was_captured_with():
  """Captured, then outgrown by an eager call: the replay still writes into its own scratch and not into what was allocated
  since."""
  from jetstream_pytorch_b200 import _lib
  from jetstream_pytorch_b200 import attention_kernel as ak

  q, k, v, end = _case(9, 32, 8, 1500, 1)
  want, _ = ak.ragged_mha(q, k, v, 0, None, end)
  torch.cuda.synchronize()
  graph = torch.cuda.CUDAGraph()
  with torch.cuda.graph(graph):
    out, _ = ak.ragged_mha(q, k, v, 0, None, end)
  held = [t.data_ptr() for _, stream, t in _lib.native.attention_workspaces() if stream is None]
  biggest = max(t.numel() for _, stream, t in _lib.native.attention_workspaces() if stream is None)
  # a call of the scalar kernel whose partial sums need more than that: rows x splits x (D + 2) floats
  g = torch.Generator(device=DEV).manual_seed(5)
  s, rows = 2048, 4
  while True:
    big_q = torch.randn((1, 1, rows, 96), generator=g, device=DEV)
    k2 = torch.randn((1, 1, s, 96), generator=g, device=DEV)
    splits = biggest // (rows * 98 * 4) + 2
    if splits <= 2048:
      break
    rows *= 4
  ak._flash_decode(big_q, k2, k2, sm_scale=0.1, kv_strides=(s * 96, s * 96, 96), n_kv_heads=1, seq=s, num_splits=splits)
  now = {t.data_ptr(): t for _, stream, t in _lib.native.attention_workspaces() if stream is None}
  assert len(now) == len(held) + 1 and set(held) <= set(now)  # outgrown, and still held
  sizes = sorted(t.numel() for t in now.values())
  assert sizes[-1] >= 2 * sizes[-2]
  fill = [torch.full((sizes[-2],), 7, dtype=torch.uint8, device=DEV) for _ in range(4)]
  for _ in range(2):
    graph.replay()
  torch.cuda.synchronize()
  assert torch.equal(out, want) and ak.kernel_status(DEV) == 0
  assert all(bool((f == 7).all()) for f in fill)


_FIRST = """
import torch
from jetstream_pytorch_b200 import attention_kernel as ak
g = torch.Generator(device="cuda").manual_seed(0)
q, k, v = (torch.randn((1, 700, h, 128), generator=g, device="cuda", dtype=torch.bfloat16).transpose(1, 2) for h in (16, 4, 4))
mask = torch.full((700, 700), float("-inf"), device="cuda").triu(1).to(torch.bfloat16).repeat(4, 1)[None, None]
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
  out = ak.dense_attention(q, k, v, None, None, mask)
graph.replay()
torch.cuda.synchronize()
got = out.clone()
assert torch.equal(got, ak.dense_attention(q, k, v, None, None, mask)) and ak.kernel_status("cuda") == 0
print("captured first")
"""


def test_a_prompt_can_be_captured_before_anything_ran():
  import os
  import subprocess
  import sys

  root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
  run = subprocess.run([sys.executable, "-c", _FIRST], cwd=root, capture_output=True, text=True, timeout=300)
  assert run.returncode == 0 and "captured first" in run.stdout, run.stderr[-2000:]
