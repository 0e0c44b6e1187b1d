"""The int8 decode kernel with its cache rows copied by the threads (layouts that no tensor map describes; JPT_NO_TMA=1, read once per process,
takes every layout there): the tests of its steps, lengths and divisions again, in a process of their own."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("tests", ["test_gpu_fused_step.py", "test_gpu_decode_work_list.py", "test_gpu_random_shapes.py"])
def test_rows_copied_by_the_threads(tests):
  r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", os.path.join(HERE, tests)], cwd=os.path.dirname(HERE),
                     env=dict(os.environ, JPT_NO_TMA="1"), capture_output=True, text=True, timeout=300)
  assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
