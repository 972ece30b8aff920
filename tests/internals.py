"""tests/cpp/internals.cu as a ctypes library: internal functions of libgreen_b200.so."""
import ctypes
import functools
import os
import subprocess
import tempfile

from green_gpu_b200 import build, native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@functools.lru_cache(None)
def load():
    native.load()
    lib = build.build()
    out = os.path.join(tempfile.mkdtemp(prefix="internals_"), "internals.so")
    cmd = [build.nvcc(), *build.ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I",
           os.path.join(ROOT, "include"), "-I", build.CSRC, "-shared", "-o", out,
           os.path.join(ROOT, "tests", "cpp", "internals.cu"), "-L", os.path.dirname(lib), "-lgreen_b200",
           "-Xlinker", "-rpath=" + os.path.dirname(lib)]
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return ctypes.CDLL(out)
