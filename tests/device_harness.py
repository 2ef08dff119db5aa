"""Compiles a few lines of CUDA against the library's device headers, for tests
of device functions that no entry point reaches by itself."""
import ctypes
import importlib.util
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "genericlinearalgebra.jl_gb300")


def compile_cuda(source, directory, link=()):
    """The shared library of `source` (a .cu text that may include the csrc headers), loaded."""
    spec = importlib.util.spec_from_file_location("gla_build", os.path.join(PKG, "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    cu, so = os.path.join(str(directory), "harness.cu"), os.path.join(str(directory), "harness.so")
    with open(cu, "w") as f:
        f.write(source)
    r = subprocess.run([b.nvcc(), *b.FLAGS, *b.ARCH, "-I", b.CSRC, "-shared", "-o", so, cu, *link],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)
