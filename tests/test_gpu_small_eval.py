"""The evaluations of the small tx sizes with a different tx type in every task of a warp, as the closed loop and the learned
analysis run them, against the evaluation of one block a warp and against each other.  Integers: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TX = [(0, 4, 4), (1, 8, 8), (5, 4, 8), (6, 8, 4), (13, 4, 16), (14, 16, 4)]
SET1 = [0, 1, 2, 3, 9, 10, 11]


def _blocks(rng, n, w, h, bd):
    """Sources and predictions: full-range noise, small residuals, single spikes, sparse columns and rows, flat ones."""
    top = (1 << bd) - 1
    src, pred = rng.integers(0, top + 1, (n, h, w)), rng.integers(0, top + 1, (n, h, w))
    kind = rng.integers(0, 6, n)
    small = np.clip(pred + np.round(rng.normal(0, top / 60, (n, h, w))).astype(int), 0, top)
    src = np.where((kind == 1)[:, None, None], small, src)
    one = pred.copy()
    one[np.arange(n), rng.integers(0, h, n), rng.integers(0, w, n)] = rng.integers(0, top + 1, n)
    src = np.where((kind == 2)[:, None, None], one, src)
    lines = np.where((rng.integers(0, 2, (n, 1, w)) * (kind == 3)[:, None, None] + rng.integers(0, 2, (n, h, 1)) * (kind == 4)[:, None, None]) > 0,
                     src, pred)
    src = np.where(((kind == 3) | (kind == 4))[:, None, None], lines, src)
    src = np.where((kind == 5)[:, None, None], pred, src)
    src[0], pred[0] = top, 0
    src[1], pred[1] = 0, top
    return src, pred


@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("tx", TX, ids=["%dx%d" % (t[1], t[2]) for t in TX])
def test_mixed_types_in_a_warp(enc, tx, bd):
    t, w, h = tx
    rng = np.random.default_rng(70 + t + bd)
    for q in (1, 25, 60, 121, 255):
        for plane in (0, 1):
            n = 403   # the last warp of either form has blocks to spare
            src, pred = _blocks(rng, n, w, h, bd)
            types = rng.choice(SET1, n)
            ctx = (int(rng.integers(0, 13)), int(rng.integers(0, 3)), int(rng.integers(0, 13)))
            pair = enc.test_eval_mixed(0, src, pred, t, types, plane, q, ctx, bd)
            thread = enc.test_eval_mixed(1, src, pred, t, types, plane, q, ctx, bd)
            for a, b, name in zip(pair[1:], thread[1:], ("D", "R", "eob")):
                assert np.array_equal(a, b), "%s: two lanes a block and a thread a block differ at %s" % (name, np.nonzero(a != b)[0][:4])
            if w * h == 64:
                assert np.array_equal(pair[0], thread[0])
            assert np.any(np.abs(pair[0]) > 14) or q > 25
            for tt in SET1:   # the same blocks, one type a warp
                m = types == tt
                alone = enc.test_eval_mixed(0, src[m], pred[m], t, types[m], plane, q, ctx, bd)
                for a, b in zip(pair, alone):
                    assert np.array_equal(a[m], b)
                if bd == 8:   # and one block a warp, through the evaluation of run-time sizes
                    _, lv, D, R, eob = enc.test_fwd_quant(src[m] - pred[m], t, tt, plane, q, ctx)
                    assert np.array_equal(pair[0][m], lv), "levels differ (type %d, qindex %d)" % (tt, q)
                    assert np.array_equal(pair[1][m], D) and np.array_equal(pair[3][m], eob)
                    assert np.array_equal(pair[2][m], R), "rates differ (type %d, qindex %d, blocks %s)" % (tt, q, np.nonzero(pair[2][m] != R)[0][:4])


def test_refusals(enc):
    z = np.zeros((1, 4, 4), np.uint16)
    for kw in (dict(tx_size=2), dict(types=[4]), dict(ctx=(13, 0, 0)), dict(src=z + 256)):
        with pytest.raises(Exception):
            enc.test_eval_mixed(0, kw.get("src", z), z, kw.get("tx_size", 0), kw.get("types", [0]), 0, 100, kw.get("ctx", (0, 0, 0)))
