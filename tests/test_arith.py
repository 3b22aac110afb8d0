"""The kernels' table-free arithmetic on the CPU (tests/arith_host.cpp): packed levels against their definition, the parallel
range coder against a serial one and against the decoder of spec 8.2.  Integers and bytes: equal."""
import ctypes as C

import numpy as np
import pytest

import arith


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    return arith.build(tmp_path_factory.mktemp("arith"))


def test_packed_rows_have_the_coefficients_rate(L):
    """row_bits over the six small sizes and three classes: levels up to the largest, dense and sparse, any scan."""
    assert L.levels_check(C.c_uint(1), C.c_int(20000)) == 0


def test_levels_without_division(L):
    """quant_level at the thresholds of every level up to 400 and at random values, for the steps of the qindex extremes."""
    steps = np.array([4, 5, 7, 8, 9, 31, 63, 64, 65, 127, 255, 342, 1023, 1336, 1828, 4 * 1336, 4 * 1828], np.int32)
    assert L.quant_check(steps.ctypes.data, len(steps), 3, 200000) == 0


def test_carries_of_32_digits(L):
    assert L.carry_check(C.c_uint(5), C.c_int(200000)) == 0


def _cdfs(rng):
    """CDFs of every alphabet from 2 to 16 symbols, a skewed and a flat one each, in the spec's form, at their own offsets."""
    off, alphabet, data = [], [], [0, 0, 0]
    for n in list(range(2, 17)) * 3:
        p = rng.random(n) ** rng.choice([0.3, 1, 6, 20]) + 1e-3
        c = np.maximum(np.round(np.cumsum(p) / p.sum() * (32768 - 33 * n)) + 32 * np.arange(1, n + 1), 1).astype(int)
        c[-1] = 32768
        off.append(len(data))
        alphabet.append(n)
        data += list(c) + [0]
    return np.array(off), np.array(alphabet), np.array(data, np.uint16)


@pytest.mark.parametrize("kind", ["mixed", "first", "one", "bits", "last"])
def test_parallel_coder_equals_the_serial_one(L, kind):
    """Also with chunks that hardly hold a step, streams around a chunk's edges, and a single symbol."""
    rng = np.random.default_rng([ord(c) for c in kind])
    for chunk, lengths in ((1024, (1, 2, 31, 1023, 1024, 1025, 2049, 9000)), (64, (63, 64, 65, 128, 3000)), (7, (700,)), (32, tuple(rng.integers(1, 600, 40)))):
        for n in lengths:
            off, alphabet, cdf = _cdfs(rng)
            w = arith.words(rng, off, alphabet, int(n), kind)
            want = arith.serial(L, w, cdf)
            assert arith.decoded(L, want, w, cdf) == n
            assert arith.parallel(L, w, cdf, chunk) == want, "%d symbols in chunks of %d" % (n, chunk)
