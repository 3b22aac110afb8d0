"""tests/arith_host.cpp built with the host compiler and called through ctypes, and streams of symbol words for it."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ADAPT, BIT, SPLIT_H, SPLIT_V = 0, 1, 2, 3


def build(tmp):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    so = os.path.join(str(tmp), "libarith.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(HERE, "..", "av1gpu_b200", "csrc"),
                    os.path.join(HERE, "arith_host.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    vp, ln = C.c_void_p, C.c_long
    L.serial_code.argtypes, L.serial_code.restype = [vp, ln, vp, ln, vp, ln], ln
    L.parallel_code.argtypes, L.parallel_code.restype = [vp, ln, vp, ln, ln, vp, ln], ln
    L.spec_decode.argtypes, L.spec_decode.restype = [vp, ln, vp, ln, vp, ln], ln
    L.quant_check.argtypes = [vp, C.c_int, C.c_uint, C.c_int]
    return L


def serial(L, words, cdf):
    out = np.zeros(2 * len(words) + 64, np.uint8)
    n = L.serial_code(words.ctypes.data, len(words), cdf.ctypes.data, len(cdf), out.ctypes.data, out.size)
    assert n > 0
    return out[:n].tobytes()


def parallel(L, words, cdf, chunk):
    out = np.zeros(2 * len(words) + 64, np.uint8)
    n = L.parallel_code(words.ctypes.data, len(words), cdf.ctypes.data, len(cdf), chunk, out.ctypes.data, out.size)
    assert n > 0, "parallel form refused: %d" % n
    return out[:n].tobytes()


def decoded(L, data, words, cdf):
    return L.spec_decode(data, len(data), words.ctypes.data, len(words), cdf.ctypes.data, len(cdf))


def words(rng, off, alphabet, n, kind):
    """n symbol words over the CDFs at off with the alphabets given.  kind: "mixed" (every CDF, bits, frame-edge splits),
    "first" (long stretches of symbol 0), "one" (one CDF has nearly all), "bits", "last" (the least probable symbols)."""
    off, alphabet = np.asarray(off), np.asarray(alphabet)
    k = rng.integers(0, len(off), n)
    if kind == "one":
        k = np.where(rng.random(n) < 0.97, rng.integers(0, len(off)), k)
    N = alphabet[k].astype(np.int64)
    s = np.minimum((rng.random(n) ** rng.uniform(1, 4) * N).astype(np.int64), N - 1)
    if kind == "first":
        s[rng.random(n) < 0.997] = 0
        for _ in range(3):
            a = int(rng.integers(0, n))
            s[a:a + int(rng.integers(1, 5000))] = 0
    if kind == "last":
        s = N - 1
    w = ADAPT | (N - 1) << 2 | s << 6 | off[k].astype(np.int64) << 16
    b = rng.random(n) < (1.0 if kind == "bits" else 0.0 if kind == "first" else 0.15)
    w = np.where(b, BIT | 1 << 2 | rng.integers(0, 2, n) << 6, w)
    part = off[alphabet == 10]
    if len(part) and kind == "mixed":
        e = rng.random(n) < 0.03
        w = np.where(e, rng.choice([SPLIT_H, SPLIT_V], n) | 1 << 2 | rng.integers(0, 2, n) << 6 | rng.choice(part, n).astype(np.int64) << 16, w)
    return w.astype(np.uint32)
