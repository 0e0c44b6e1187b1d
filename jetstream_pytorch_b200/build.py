"""Builds libjpt_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m jetstream_pytorch_b200.build [--force]
"""

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libjpt_b200.so")
NATIVE = os.path.join(HERE, "_native.so")  # the host side of the calls, a Python extension module on top of LIB

SOURCES = [
    "kv_update.cu",
    "prefill_insert.cu",
    "attention_generic.cu",
    "attention_mma.cu",
    "attention_umma.cu",
    "attention_prefill.cu",
    "w8a16_linear.cu",
    "engine_step.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]

# The quantisers must round exactly like the reference: never fast math, and no
# fused multiply-add contraction across the rounding steps in those two files.
EXTRA_FLAGS = {
    "kv_update.cu": ["--fmad=false"],
    "prefill_insert.cu": ["--fmad=false"],
}


def _stale():
  if not os.path.exists(LIB) or not os.path.exists(NATIVE):
    return True
  t = min(os.path.getmtime(LIB), os.path.getmtime(NATIVE))
  deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
  deps += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
  deps.append(os.path.abspath(__file__))
  return any(os.path.getmtime(d) > t for d in deps)


def build_library(force=False, verbose=False):
  """Compiles every .cu under csrc/ into one shared library and host.cpp into the extension module on top of it; returns the library's path."""
  if not force and not _stale():
    return LIB
  nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
  objs = []
  build_dir = os.path.join(HERE, "build")
  os.makedirs(build_dir, exist_ok=True)
  procs = [("host.cpp", _compile_host(os.path.join(build_dir, "host.o")))]
  for src in SOURCES:
    obj = os.path.join(build_dir, src.replace(".cu", ".o"))
    cmd = [nvcc, *NVCC_FLAGS, *EXTRA_FLAGS.get(src, []), *os.environ.get("JPT_NVCC_FLAGS", "").split(), "-I", INCLUDE, "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
    if verbose:
      cmd += ["-Xptxas", "-v"]
    procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    objs.append(obj)
  for src, pr in procs:
    out, _ = pr.communicate()
    if verbose and out:
      print(out)
    if pr.returncode != 0:
      raise RuntimeError(f"nvcc failed on {src}:\n{out}")
  cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
  out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
  if out.returncode != 0:
    raise RuntimeError(f"link failed:\n{out.stdout}")
  _link_host(os.path.join(build_dir, "host.o"))
  return LIB


def _compile_host(obj):
  import sysconfig

  import torch
  from torch.utils import cpp_extension

  cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-w",
         f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I", INCLUDE,
         "-isystem", sysconfig.get_paths()["include"], "-isystem", "/usr/local/cuda/include"]
  for d in cpp_extension.include_paths():
    cmd += ["-isystem", d]
  cmd += ["-c", os.path.join(CSRC, "host.cpp"), "-o", obj]
  return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _link_host(obj):
  import torch

  libs = os.path.join(os.path.dirname(torch.__file__), "lib")
  cmd = [os.environ.get("CXX", "g++"), "-shared", "-o", NATIVE, obj, "-L", libs, "-L", HERE, "-L", "/usr/local/cuda/lib64",
         "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-lcudart", "-l:libjpt_b200.so",
         "-Wl,-rpath,$ORIGIN"]
  out = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
  if out.returncode != 0:
    raise RuntimeError(f"link failed:\n{out.stdout}")


if __name__ == "__main__":
  print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
