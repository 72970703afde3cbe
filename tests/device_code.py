"""Compiles a piece of CUDA that includes the library's headers, for tests of
single device functions."""
import ctypes
import os
import subprocess

from conftest import ROOT
from ntustcfdlab_b200 import build


def compile_cuda(tmp_path, source: str) -> ctypes.CDLL:
    cu, so = tmp_path / "device_code.cu", tmp_path / "device_code.so"
    cu.write_text(source)
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "ntustcfdlab_b200", "csrc"), "-cudart", "static", "-o", str(so), str(cu)],
                   check=True)
    return ctypes.CDLL(str(so))
