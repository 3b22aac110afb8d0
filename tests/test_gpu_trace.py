"""The closed loop's leaf trace (is_set_trace / is_get_trace): every leaf has all its stamps, in order."""
import numpy as np
import pytest

from av1gpu_b200 import leaftrace

pytestmark = pytest.mark.gpu


def _picture(w, h, bd, c444):
    """A flat left half (blocks of 32 and 64 samples a side, whose tx sizes have DCT_DCT only), noise over ramps on the
    right (small blocks, and the sizes between)."""
    dt, top = (np.uint16, 1023) if bd == 10 else (np.uint8, 255)
    rng = np.random.default_rng(w + h)
    out = []
    for ph, pw in ((h, w),) + (((h, w) if c444 else ((h + 1) // 2, (w + 1) // 2)),) * 2:
        p = np.full((ph, pw), top // 3, np.float64)
        p[:, pw // 2:] = (np.arange(ph)[:, None] + 2 * np.arange(pw - pw // 2)[None, :]) % (top // 2)
        p[:, pw // 2:] += rng.normal(0, top / 40, (ph, pw - pw // 2)) * (np.arange(ph)[:, None] > ph // 2)
        out.append(np.clip(np.round(p), 0, top).astype(dt))
    return tuple(out)


@pytest.mark.parametrize("w,h,q,bd,c444,rd_k", [(448, 320, 120, 8, False, 4), (320, 200, 200, 10, True, 4), (448, 320, 220, 8, False, 1)])
def test_every_leaf_has_its_stamps_in_order(enc, w, h, q, bd, c444, rd_k):
    """Also for the leaves that skip a pass (a tx size of DCT_DCT only has no pass 2; a single candidate with DCT_DCT, as
    with rd_k 1, has no pass 1): a pass that does not run takes no time.  Leaves without chroma have stamps 6 and 7 zero."""
    im = _picture(w, h, bd, c444)
    enc.set_search_options(rd_k=rd_k, tx_keep=0)
    enc.set_trace(True)
    try:
        enc.encode(tuple(p[::-1].copy() for p in im), q)   # another picture first: what it leaves in the trace is old
        old = enc.trace().astype(np.int64)
        r = enc.encode(im, q)
        t = enc.trace().astype(np.int64)
    finally:
        enc.set_trace(False)
        enc.set_search_options()
    ids = t[:, 9]
    assert len(t) == len(r.blocks) and len(np.unique(ids)) == len(t)
    t0 = old[:, 8].max()
    luma = t[:, [0, 1, 2, 3, 4, 5, 8]]
    assert np.all(luma[:, 0] > t0) and np.all(np.diff(luma, axis=1) >= 0), "a luma stamp is missing or stale"
    has = t[:, 6] != 0
    assert np.all(np.diff(t[has][:, [5, 6, 7, 8]], axis=1) >= 0) and np.all(t[~has][:, 7] == 0), "a chroma stamp is missing or stale"
    leaves = {}
    for sb in np.unique((ids >> 8) & 0xFFFFFF):
        leaves[int(sb)] = enc.debug_leaves(int(sb))
    bs = np.array([leaves[int(v >> 8) & 0xFFFFFF][0][int(v) & 255] for v in ids])
    if not c444:
        # 4:2:0: a block of 4 samples a side carries chroma only at odd 4x4 rows / columns
        x4 = np.array([leaves[int(v >> 8) & 0xFFFFFF][1][int(v) & 255] for v in ids])
        y4 = np.array([leaves[int(v >> 8) & 0xFFFFFF][2][int(v) & 255] for v in ids])
        n4w, n4h = np.isin(bs, [0, 1, 16]), np.isin(bs, [0, 2, 17])
        assert np.array_equal(has, (~n4w | (x4 & 1 == 1)) & (~n4h | (y4 & 1 == 1)))
    else:
        assert has.all()
    big = np.isin(bs, [9, 10, 11, 12, 7, 8, 18, 19, 20, 21])   # a side of 32 or 64: no pass 2
    assert big.any() and np.isin(bs, [0, 1, 2, 3]).any()
    assert np.all(t[big][:, 3] == t[big][:, 4])
    if rd_k == 1:   # a single candidate: no pass 1 for them either
        assert np.median(t[big][:, 3] - t[big][:, 2]) < 1000
    rows, per, _, span = leaftrace.summarise(enc, enc.trace())
    assert all(np.isfinite(v).all() and min(v) >= 0 and max(v) <= span * 1e3 for v in rows.values())
    assert all(min(v) >= 0 and max(v[1:]) <= span * 1e3 for v in per.values())
