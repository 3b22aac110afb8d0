"""The entropy coder's kernels on symbol streams of their own, without the reference: the payloads against a serial coder and the
decoder of spec 8.2 (tests/arith_host.cpp), over the CDFs the library holds.  Bytes: equal."""
import numpy as np
import pytest

import arith
from av1gpu_b200 import isearch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    return arith.build(tmp_path_factory.mktemp("arith"))


@pytest.mark.parametrize("kind", ["mixed", "first", "one", "bits", "last"])
def test_payloads_equal_the_serial_coder(enc, L, kind):
    """Tiles around the edges of a chunk (1024 steps), of a batch (4096 symbols) and of a CDF's first 32 symbols, many tiles in
    one call, and one long one; four q-contexts."""
    rng = np.random.default_rng([ord(c) for c in kind])
    for qctx, lengths in enumerate(((1, 2, 15, 16, 17, 31, 32, 33, 34), (1023, 1024, 1025, 2047, 2049), (4095, 4096, 4097, 8193, 12289),
                                    (200000,) + tuple(rng.integers(1, 3000, 60)))):
        cdf, off, alphabet = isearch.test_cdfs(qctx)
        tiles = [arith.words(rng, off, alphabet, int(n), kind) for n in lengths]
        for w, got in zip(tiles, enc.test_code_symbols(tiles, qctx)):
            assert arith.decoded(L, got, w, cdf) == len(w)
            assert got == arith.serial(L, w, cdf), "%d symbols, q-context %d" % (len(w), qctx)


def test_refusals(enc):
    cdf, off, alphabet = isearch.test_cdfs(0)
    good = arith.words(np.random.default_rng(1), off, alphabet, 8, "last")
    for w in (good[:0], good | 3 << 2, (good & 0xFFFF) | (int(off[0]) + 1) << 16, np.full(3, 1 | 1 << 2 | 2 << 6, np.uint32)):
        with pytest.raises(Exception):
            enc.test_code_symbols([w.astype(np.uint32)], 0)
