"""The committed records of the oracle (tests/golden), without the oracle library: the GPU reproduces them where the library
holds av1core's own tables."""
import glob
import os

import numpy as np
import pytest

from av1gpu_b200 import isearch

pytestmark = pytest.mark.gpu
HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


@pytest.fixture(autouse=True)
def av1core_tables():
    if not isearch.build_info().endswith("checkout"):
        pytest.skip("the library was compiled from headers that are not a checkout of av1core: " + isearch.build_info())


@pytest.mark.parametrize("name", sorted(os.path.basename(p) for p in glob.glob(os.path.join(HERE, "oracle_*.npz"))))
def test_golden_records(enc, name):
    z = np.load(os.path.join(HERE, name))
    r = enc.encode((z["y"], z["u"], z["v"]), int(z["q"]))
    assert np.array_equal(r.blocks.view(np.uint8).ravel(), z["blocks"].ravel()) and np.array_equal(r.block_txb, z["block_txb"])
    assert np.array_equal(r.txb.view(np.uint8).ravel(), z["txb"].ravel()) and np.array_equal(r.coeffs, z["coeffs"])
    assert all(np.array_equal(r.recon[p], z["recon_" + k]) for p, k in enumerate("yuv"))


def test_golden_reference_picture(enc):
    z = np.load(os.path.join(HERE, "gate_cfl_edge_211x149.npz"))
    for q in (int(v) for v in z["qs"]):
        r = enc.encode((z["y"], z["u"], z["v"]), q)
        assert np.array_equal(r.blocks.view(np.uint8), z["blocks_%d" % q]) and np.array_equal(r.block_txb, z["block_txb_%d" % q])
        assert np.array_equal(r.txb.view(np.uint8), z["txb_%d" % q]) and np.array_equal(r.coeffs, z["coeffs_%d" % q])
        assert all(np.array_equal(r.recon[p], z["recon_%s_%d" % (k, q)]) for p, k in enumerate("yuv"))
