"""The kernels' table-free arithmetic on the CPU (tests/arith_host.cpp): packed levels and
quantisation against their definition.  Integers: equal."""
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
