"""Performance cases: what a program built on this library has it do, through its public entry points.

Every case is one of five kinds of work, over the sizes, formats and options of the repository's own configurations:

  encode   one image searched (planes in host or device memory), its DecisionRecord and reconstruction read back
  batch    a list of images of uneven size, format and qindex searched in one call, every record read back
  obu      the records of the handle's last search entropy-coded on the device into OBU streams
  avif     planes to AVIF file: search, deblocking and CDEF, entropy coding, container
  train    one training step of the shortlist network on rows of a search

listed() names the cases that are measured, draw(rng) gives further ones of the same ranges, prepare(case, seed) makes
what a program has in hand before the call, run(state) is one pass, work(case) the bytes and operations it cannot do
without, exact(case, seed) a float64 restatement of the outputs that are computed in floating point.
"""
import math
import os

import numpy as np
import torch

import av1gpu_b200
from av1gpu_b200 import Encoder
from av1gpu_b200 import isearch, shortlist

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(av1gpu_b200.__file__)), "shortlist_weights.npz")
FORMATS = ((8, False), (8, True), (10, False), (10, True))


def listed():
    return [
        # the smallest call: a thumbnail, where the dependency chain and the launches count
        dict(name="thumb_160x120", kind="encode", width=160, height=120, bit_depth=8, chroma_444=False, qindex=120, device=False,
             pruning="none"),
        # a picture of a web page, host planes in, record out
        dict(name="web_512x512", kind="encode", width=512, height=512, bit_depth=8, chroma_444=False, qindex=120, device=False,
             pruning="none"),
        # an odd, ragged size with 10-bit samples at a coarse quantizer
        dict(name="odd_811x613_10bit", kind="encode", width=811, height=613, bit_depth=10, chroma_444=False, qindex=200, device=False,
             pruning="none"),
        # full HD with 10-bit 4:4:4 samples at high quality: the heaviest format per pixel
        dict(name="hd_1920x1080_10bit_444", kind="encode", width=1920, height=1080, bit_depth=10, chroma_444=True, qindex=60,
             device=True, pruning="none"),
        # a photograph of 12 megapixels, planes on the device: the benchmark's workload
        dict(name="photo_4000x3000", kind="encode", width=4000, height=3000, bit_depth=8, chroma_444=False, qindex=120, device=True,
             pruning="none"),
        # a fast preset on one picture: two RD candidates and two tx types per block
        dict(name="pruned_1500x1001", kind="encode", width=1500, height=1001, bit_depth=8, chroma_444=False, qindex=160, device=True,
             pruning="options"),
        # a folder of pictures of uneven size and mixed format as one batch of host planes, the plain form
        dict(name="batch_12_mixed", kind="batch", images=12, max_mp=2.0, mix=True, device=False, pruning="none"),
        # the same with the learned shortlist, planes on the device: the throughput form
        dict(name="batch_16_learned", kind="batch", images=16, max_mp=3.0, mix=True, device=True, pruning="learned"),
        # the bitstream of one full-HD picture: one tile, the coder's serial chain
        dict(name="obu_1920x1080", kind="obu", images=1, width=1920, height=1080, bit_depth=8, chroma_444=False, qindex=120),
        # the bitstreams of a batch coded side by side
        dict(name="obu_batch_12", kind="obu", images=12, width=1024, height=768, bit_depth=8, chroma_444=False, qindex=90),
        # a picture from planes to file, with the post-filters
        dict(name="avif_1280x960", kind="avif", width=1280, height=960, bit_depth=8, chroma_444=False, qindex=140),
        # a training step of the shortlist network
        dict(name="train_4096", kind="train", rows=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    u = rng.random()
    if u < 0.5:
        bd, c444 = FORMATS[rng.choice((0, 0, 0, 1, 2, 3))]
        area, ar = math.exp(rng.uniform(math.log(1.2e4), math.log(6e6 if not c444 else 2e6))), math.exp(rng.uniform(-1.1, 1.1))
        return dict(kind="encode", width=max(16, int(math.sqrt(area * ar))), height=max(16, int(math.sqrt(area / ar))), bit_depth=bd,
                    chroma_444=c444, qindex=rng.randint(40, 220), device=rng.random() < 0.5,
                    pruning=rng.choice(("none", "none", "options", "learned")))
    if u < 0.7:
        return dict(kind="batch", images=_log_int(rng, 2, 24), max_mp=round(rng.uniform(0.4, 2.0), 3), mix=rng.random() < 0.7,
                    device=rng.random() < 0.5, pruning=rng.choice(("none", "options", "learned")))
    if u < 0.85:
        bd, c444 = FORMATS[rng.choice((0, 0, 1, 2, 3))]
        return dict(kind="obu", images=_log_int(rng, 1, 12), width=_log_int(rng, 100, 1400), height=_log_int(rng, 100, 1400),
                    bit_depth=bd, chroma_444=c444, qindex=rng.randint(40, 220))
    if u < 0.95:
        bd, c444 = FORMATS[rng.choice((0, 0, 1, 2, 3))]
        return dict(kind="avif", width=_log_int(rng, 100, 1600), height=_log_int(rng, 100, 1600), bit_depth=bd, chroma_444=c444,
                    qindex=rng.randint(40, 220))
    return dict(kind="train", rows=32 * _log_int(rng, 4, 256))


# ---- pictures: piecewise-constant cells, gradients, waves of period 4-64, oriented step edges and noise of sigma 3 (the
# recipe of av1gpu_b200.synth, made on the GPU) ----
def _plane(gen, w, h, centre, spread, cell):
    dev = gen.device
    f32 = torch.float32

    def uni(lo, hi, *shape):
        return torch.rand(shape, generator=gen, device=dev, dtype=f32) * (hi - lo) + lo

    yy = torch.arange(h, device=dev, dtype=f32)[:, None]
    xx = torch.arange(w, device=dev, dtype=f32)[None, :]
    gw, gh = (w + cell - 1) // cell + 2, (h + cell - 1) // cell + 2
    sx = (torch.arange(gw, device=dev, dtype=f32)[None, :] - 1 + uni(0, 1, gh, gw)) * cell
    sy = (torch.arange(gh, device=dev, dtype=f32)[:, None] - 1 + uni(0, 1, gh, gw)) * cell
    lv = uni(centre - spread, centre + spread, gh, gw)
    cy = (torch.arange(h, device=dev) // cell + 1)[:, None]
    cx = (torch.arange(w, device=dev) // cell + 1)[None, :]
    best = torch.full((h, w), float("inf"), device=dev)
    out = torch.zeros((h, w), device=dev)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            gy, gx = (cy + dy).clamp(0, gh - 1), (cx + dx).clamp(0, gw - 1)
            d = (xx - sx[gy, gx]) ** 2 + (yy - sy[gy, gx]) ** 2
            m = d < best
            best = torch.where(m, d, best)
            out = torch.where(m, lv[gy, gx], out)
    s = spread / 110.0
    par = torch.rand(5, 4, generator=gen, device=dev).tolist()
    diag = math.hypot(w, h)
    for a, b, _, _ in par[:2]:
        th = a * math.pi
        out += (10 + 30 * b) * s * ((xx - w / 2) * math.cos(th) + (yy - h / 2) * math.sin(th)) / (diag / 2)
    for a, b, c, d in par[2:]:
        th, per = a * math.pi, 4 + 60 * b
        out += (3 + 9 * c) * s * torch.sin(2 * math.pi * ((xx * math.cos(th) + yy * math.sin(th)) / per + d))
    ah, aw = (h + 255) // 256, (w + 255) // 256   # step edges over discs, one per 256 x 256 area and layer
    ay, ax = (torch.arange(h, device=dev) // 256)[:, None], (torch.arange(w, device=dev) // 256)[None, :]
    for _ in range(8):
        ex, ey, th, r = uni(0, 256, ah, aw), uni(0, 256, ah, aw), uni(0, 2 * math.pi, ah, aw), uni(24, 96, ah, aw)
        amp = uni(-40, 40, ah, aw) * s
        px, py = (xx % 256) - ex[ay, ax], (yy % 256) - ey[ay, ax]
        m = (px * px + py * py < r[ay, ax] ** 2) & (px * torch.cos(th)[ay, ax] + py * torch.sin(th)[ay, ax] > 0)
        out += amp[ay, ax] * m
    out += 3.0 * torch.randn((h, w), generator=gen, device=dev, dtype=f32)
    return out.round().clamp(0, 255)


def _planes(width, height, bit_depth, chroma_444, seed, device):
    """(Y, U, V): uint8 / int16 CUDA tensors (device) or uint8 / uint16 numpy arrays."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    cw, ch = (width, height) if chroma_444 else ((width + 1) // 2, (height + 1) // 2)
    out = []
    for p, (w, h) in enumerate(((width, height), (cw, ch), (cw, ch))):
        v = _plane(gen, w, h, 128.0 if p else 125.5, 48.0 if p else 109.5, 24 if p and not chroma_444 else 48)
        v = torch.round(v * (1023.0 / 255.0)).to(torch.int16) if bit_depth == 10 else v.to(torch.uint8)
        out.append(v if device else v.cpu().numpy().view(np.uint16 if bit_depth == 10 else np.uint8))
    return out


def _batch_images(case):
    """(width, height, bit depth, 4:4:4, qindex) of a batch's images: log-uniform areas of 0.18 MP up to max_mp, aspect
    1:3 to 3:1, one in five 10-bit 4:4:4 with mix, qindex 40 .. 220; the same for every seed of a case."""
    rng = np.random.default_rng([case["images"], int(case["max_mp"] * 1000), int(case["mix"])])
    out = []
    for i in range(case["images"]):
        area, ar = math.exp(rng.uniform(math.log(0.18e6), math.log(case["max_mp"] * 1e6))), math.exp(rng.uniform(-math.log(3), math.log(3)))
        ten = bool(case["mix"] and i % 5 == 3)
        out.append((int(math.sqrt(area * ar)) & ~1, int(math.sqrt(area / ar)) & ~1, 10 if ten else 8, ten, int(rng.integers(40, 221))))
    return out


def _set_pruning(enc, pruning):
    if pruning == "options":
        enc.set_search_options(rd_k=2, tx_keep=2)
    elif pruning == "learned":
        enc.set_shortlist(shortlist.load_params(WEIGHTS), **shortlist.LEARNED)
        enc.set_search_options(**shortlist.LEARNED_OTHER)


def _record_buffers(width, height, bit_depth, chroma_444):
    """Page-locked buffers a record of the size fits in, as a program that searches many pictures keeps them."""
    sbs = ((width + 63) // 64) * ((height + 63) // 64)
    per = 12288 if chroma_444 else 6144

    def pinned(nbytes, dt):
        return torch.zeros(nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(dt)

    cw, ch = (width, height) if chroma_444 else ((width + 1) // 2, (height + 1) // 2)
    dt = np.dtype(np.uint16 if bit_depth == 10 else np.uint8)
    return {"blocks": pinned(sbs * 256 * 16, isearch.BLOCK_DT), "block_txb": pinned((sbs * 256 + 1) * 4, np.uint32),
            "txb": pinned(sbs * 768 * 16, isearch.TXB_DT), "coeffs": pinned(sbs * per * 2, np.int16),
            "recon": [pinned(h * w * dt.itemsize, dt).reshape(h, w) for w, h in ((width, height), (cw, ch), (cw, ch))]}


def _room(dims):
    """Zeroed buffers that hold the records and streams of the images, where a pass leaves its results back to back."""
    sbs = sum(((w + 63) // 64) * ((h + 63) // 64) for w, h, _, _, _ in dims)
    px = sum(((w + 63) & ~63) * ((h + 63) & ~63) * (3 if c else 2) for w, h, _, c, _ in dims)
    recon = sum(2 * w * h * (3 if c else 2) for w, h, _, c, _ in dims)
    size = {"blocks": sbs * 4096, "block_txb": sbs * 256 + len(dims), "txb": sbs * 768 * 16, "coeffs": px, "recon": recon, "obu": px}
    kind = {"block_txb": np.uint32, "coeffs": np.int16}
    return {k: np.zeros(n, kind.get(k, np.uint8)) for k, n in size.items()}


def _leave(room, key, arrays):
    o, buf = 0, room[key]
    for a in arrays:
        a = a.ravel().view(buf.dtype)
        buf[o:o + a.size] = a
        o += a.size
    return buf


def _records(room, recs):
    return {"blocks": _leave(room, "blocks", [r.blocks for r in recs]), "block_txb": _leave(room, "block_txb", [r.block_txb for r in recs]),
            "txb": _leave(room, "txb", [r.txb for r in recs]), "coeffs": _leave(room, "coeffs", [r.coeffs for r in recs]),
            "recon": _leave(room, "recon", [p for r in recs for p in r.recon])}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "train":
        with_rows = Encoder(0)
        rows = []
        k = 0
        while sum(x.shape[0] for x, _ in rows) < case["rows"]:
            with_rows.encode_device_async(_planes(512, 384, 8, False, seed * 16 + k, True), 120)
            rows.append(shortlist.image_rows(with_rows))
            k += 1
        with_rows.close()
        X, y = torch.cat([x for x, _ in rows]), torch.cat([v for _, v in rows])
        perm = torch.randperm(X.shape[0], generator=torch.Generator().manual_seed(seed))[:case["rows"]].to(X.device)
        s["X"], s["y"] = X[perm].contiguous(), y[perm].contiguous()
        s["params"] = shortlist.init_params(seed)
        s["learner"] = shortlist.Learner(max_batch=case["rows"])
        s["learner"].set_params(s["params"])
        return s
    s["enc"] = enc = Encoder(0)
    if kind == "batch":
        _set_pruning(enc, case["pruning"])
        if case["device"]:
            enc.set_batch_options(front_streams=2)
        dims = _batch_images(case)
        s["images"] = [_planes(w, h, bd, c, seed * 64 + i, case["device"]) for i, (w, h, bd, c, _) in enumerate(dims)]
        s["q"], s["dims"], s["room"] = [d[4] for d in dims], dims, _room(dims)
        return s
    w, h, bd, c444, q = case["width"], case["height"], case["bit_depth"], case["chroma_444"], case["qindex"]
    if kind == "obu":
        ims = [_planes(w, h, bd, c444, seed * 64 + i, True) for i in range(case["images"])]
        enc.encode_batch_async(ims, [q] * len(ims), host=False)
        s["room"] = _room([(w, h, bd, c444, q)] * len(ims))
        return s
    s["planes"] = _planes(w, h, bd, c444, seed, kind == "encode" and case["device"])
    s["room"] = _room([(w, h, bd, c444, q)])
    if kind == "encode":
        _set_pruning(enc, case["pruning"])
        if case["device"]:
            s["out"] = _record_buffers(w, h, bd, c444)
    else:
        fp = isearch.postfilter_from_q(isearch.frame_params(w, h, q, bd, c444), q, bd)
        fp[36], fp[38] = 1, 1                       # enable_cdef, cdef_bits: two presets
        fp[39:41], fp[47:49] = (2, 6), (1, 2)       # luma primary and secondary strengths
        fp[55:57], fp[63:65] = (1, 4), (0, 2)       # chroma
        s["fp"] = fp
        sbs = ((w + 63) // 64) * ((h + 63) // 64)
        s["cdef"] = np.random.default_rng(seed).integers(0, 2, sbs).astype(np.int8)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        loss, correct = state["learner"].train_step(state["X"], state["y"], 2e-3)
        return {"loss": loss, "correct": correct, "params": state["learner"].get_params()}
    enc = state["enc"]
    if kind == "encode" and case["device"]:   # into the program's page-locked buffers
        enc.encode_device_async(state["planes"], case["qindex"])
        out = state["out"]
        enc.fetch(case["width"], case["height"], case["qindex"], out=out, bit_depth=case["bit_depth"], chroma_444=case["chroma_444"])
        return {"blocks": out["blocks"].view(np.uint8), "block_txb": out["block_txb"], "txb": out["txb"].view(np.uint8),
                "coeffs": out["coeffs"], "recon": out["recon"]}
    if kind == "encode":
        return _records(state["room"], [enc.encode(state["planes"], case["qindex"])])
    if kind == "batch":
        if not case["device"]:
            return _records(state["room"], enc.encode_batch(state["images"], state["q"]))
        enc.encode_batch_async(state["images"], state["q"], host=False)
        return _records(state["room"], [enc.batch_fetch(i, w, h, q, bd, c) for i, (w, h, bd, c, q) in enumerate(state["dims"])])
    if kind == "obu":
        streams = enc.obu(0, case["images"])
        return {"obu": _leave(state["room"], "obu", [np.frombuffer(b, np.uint8) for b in streams]),
                "sizes": np.array([len(b) for b in streams])}
    rec = enc.encode(state["planes"], case["qindex"])
    enc.postfilter(state["fp"], state["cdef"])
    return {"avif": _leave(state["room"], "obu", [np.frombuffer(enc.avif(0, 1)[0], np.uint8)]),
            "blocks": _leave(state["room"], "blocks", [rec.blocks])}


# Operations of the path are integer operations (the search and the coder use no floating point): those of the search per
# luma sample as the CPU restatement counts them at qindex 120, of the coder about 30 per symbol of 0.7 symbols per sample.
SEARCH_OPS, CODER_OPS = 16456.9 + 830.3, 20.0


def work(case):
    if case["kind"] == "train":
        n = case["rows"]
        macs = 256 * 8 * 9 + 64 * 16 * 72 + 16 * 16 * 144 + 160 * 288 + 80 * 160
        return {"bytes": n * (1056 * 2 + 12) + 6 * 4 * 62688, "flops": 6.0 * n * macs}
    if case["kind"] == "batch":
        dims = _batch_images(case)
    else:
        dims = [(case["width"], case["height"], case["bit_depth"], case["chroma_444"], case["qindex"])] * case.get("images", 1)
    by, ops = 0.0, 0.0
    for w, h, bd, c444, _ in dims:
        px, samples = w * h, w * h * (3.0 if c444 else 1.5)
        if case["kind"] == "obu":
            by += 2 * samples + 0.4 * px + 0.1 * samples
            ops += CODER_OPS * samples / 1.5
        else:
            by += samples * (bd + 7) // 8 * 2 + 2 * samples + 0.4 * px
            ops += SEARCH_OPS * px
    return {"bytes": by, "flops": ops}


def exact(case, seed):
    """The training step in float64: loss, rows whose best class is the label, and the parameters after one Adam step from
    the same start (no bf16 rounding anywhere).  The other kinds return whole numbers only."""
    if case["kind"] != "train":
        return None
    s = prepare(case, seed)
    X, y = s["X"].double(), s["y"].long()
    s["learner"].close()
    n = X.shape[0]
    p = torch.from_numpy(s["params"]).cuda().double().requires_grad_(True)
    parts, o = {}, 0
    for name, shp in shortlist.SHAPES:
        k = int(np.prod(shp))
        parts[name] = p[o:o + k].reshape(shp)
        o += k

    def conv(a, w, b, cin):   # weight columns: tap * cin + channel
        k = w.reshape(w.shape[0], 3, 3, cin).permute(0, 3, 1, 2)
        return torch.relu(torch.nn.functional.conv2d(a, k, b, stride=2, padding=1))

    a = conv(X[:, :1024].reshape(n, 1, 32, 32), parts["c1w"], parts["c1b"], 1)
    a = conv(a, parts["c2w"], parts["c2b"], 8)
    a = conv(a, parts["c3w"], parts["c3b"], 16)
    z = torch.cat([a.permute(0, 2, 3, 1).reshape(n, 256), X[:, 1024:]], 1)
    hid = torch.relu(z @ parts["f1w"].T + parts["f1b"])
    sc = hid @ parts["f2w"].T + parts["f2b"]
    loss = torch.nn.functional.cross_entropy(sc[:, :61], y[:, 0], reduction="none")
    valid = ((y[:, 2:3] >> torch.arange(16, device=y.device)) & 1).bool()
    has = y[:, 1] >= 0
    tx = torch.log_softmax(sc[:, 64:80].masked_fill(~valid, float("-inf"))[has], 1)
    loss = (loss.sum() - tx.gather(1, y[has][:, 1:2]).sum()) / n
    loss.backward()
    g = p.grad
    m, v = 0.1 * g / (1 - 0.9), 0.001 * g * g / (1 - 0.999)
    new = p.detach() - 2e-3 * m / (v.sqrt() + 1e-8)
    return {"loss": float(loss), "correct": None, "params": new.cpu().numpy()}
