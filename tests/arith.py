"""tests/arith_host.cpp built with the host compiler and called through ctypes."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def build(tmp):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    so = os.path.join(str(tmp), "libarith.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(HERE, "..", "av1gpu_b200", "csrc"),
                    os.path.join(HERE, "arith_host.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    vp = C.c_void_p
    L.quant_check.argtypes = [vp, C.c_int, C.c_uint, C.c_int]
    return L

