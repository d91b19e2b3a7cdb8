"""Performance cases: the work this library does for its users, through the
entry points of cuda-orb_b200/orbx.py.

A process keeps one context per parameter set on one CUDA stream, as a user's
program does; a state is one set of that program's inputs and output buffers
(a frame, a pair, a descriptor set), so consecutive passes may come with other
images in other buffers.

Images follow the generator of cuda-orb_b200/synth.py (blobs, rectangles and
convex polygons, noise sigma 3; the partner warped by a random homography),
written in torch so that they are made on the GPU.
"""
import collections
import ctypes
import math
import os
import sys
import types

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-orb_b200"))
import orbx  # noqa: E402
import synth  # noqa: E402

MODES = {"popc": orbx.MATCH_POPC, "imma": orbx.MATCH_IMMA, "auto": orbx.MATCH_AUTO}
LEARNED_IMAGE = 1024  # side of the images whose descriptors fill a learned index


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # one VGA camera frame, detect + describe: the call of a tracking loop, where latency counts
        dict(name="frame 640x480", kind="frame", w=640, h=480, score="harris", wta=2, octaves=8, cap=5000),
        # a still image of odd size at the upper end of the range, with the other score and sampling
        dict(name="frame 3839x2157 fast wta4", kind="frame", w=3839, h=2157, score="fast", wta=4, octaves=5,
             cap=10000),
        # the keypoints of two such frames matched, counts on the device
        dict(name="match 1100x1300", kind="match", n1=1100, n2=1300, cap=10000, mode="popc"),
        # a small pair end to end on the device (the smallest resolution of the batched workload)
        dict(name="pair 320x240", kind="pair", w=320, h=240, score="harris", wta=2, octaves=8, cap=1000),
        # the 1080p pair of the benchmark, images and results on the device
        dict(name="pair 1920x1080", kind="pair", w=1920, h=1080, score="harris", wta=2, octaves=8, cap=10000),
        # the same from pinned host images to host keypoints, matches and descriptors
        dict(name="pair host 1920x1080", kind="pair_host", w=1920, h=1080, score="harris", wta=2, octaves=8,
             cap=10000),
        # offline matching of an image collection: pairs of mixed resolution and caps in one call
        dict(name="batch of 24 pairs", kind="batch", pairs=24, layout=1, form=0),
        # two full VGA keypoint sets (5000 each) in the popcount form
        dict(name="knn2 5000x4801 popc", kind="knn2", nq=5000, ndb=4801, mode="popc"),
        # the matching workload of the benchmark
        dict(name="knn2 65536x65536 imma", kind="knn2", nq=65536, ndb=65536, mode="imma"),
        # relocalisation: one frame's keypoints against a map
        dict(name="knn2 1500x262144 auto", kind="knn2", nq=1500, ndb=262144, mode="auto"),
        # OpenCV-compatible mode at 1080p with its default parameters
        dict(name="ocv 1920x1080", kind="ocv", w=1920, h=1080, score="harris", nfeatures=5000, nlevels=8),
        # the learned index: search of a trained index, one cluster per 256 rows
        dict(name="learned search 32768x131072", kind="learned_search", nq=32768, ndb=131072, clusters=512, spill=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng):
    h = _log(rng, 160, 2160)
    return min(3840, max(160, int(h * rng.uniform(1.0, 1.9)))), h


def draw(rng):
    kind = rng.choice(["frame", "frame", "match", "pair", "pair", "pair_host", "batch", "knn2", "knn2", "knn2", "ocv",
                       "ocv", "learned_search"])
    if kind in ("frame", "pair", "pair_host"):
        w, h = _size(rng)
        if kind == "pair_host":
            w, h = min(w, 1920), min(h, 1080)
        return dict(kind=kind, w=w, h=h, score=rng.choice(["harris", "harris", "fast"]), wta=rng.choice([2, 2, 3, 4]),
                    octaves=rng.choice([1, 5, 8, 8]), cap=_log(rng, 500, 10000))
    if kind == "match":
        n1 = _log(rng, 100, 10000)
        n2 = _log(rng, 100, 10000)
        return dict(kind=kind, n1=n1, n2=n2, cap=rng.choice([max(n1, n2), 10000]),
                    mode=rng.choice(["popc", "popc", "auto", "imma"]))
    if kind == "batch":
        return dict(kind=kind, pairs=rng.randint(2, 24), layout=rng.randrange(2, 1 << 20), form=rng.choice([0, 1]))
    if kind == "knn2":
        mode = rng.choice(["popc", "imma", "auto"])
        if mode == "popc":
            return dict(kind=kind, nq=_log(rng, 64, 16384), ndb=_log(rng, 256, 32768), mode=mode)
        return dict(kind=kind, nq=_log(rng, 64, 16384), ndb=_log(rng, 1024, 262144), mode=mode)
    if kind == "ocv":
        w, h = _size(rng)
        return dict(kind=kind, w=min(w, 1920), h=min(h, 1080), score=rng.choice(["harris", "fast"]),
                    nfeatures=_log(rng, 500, 8000), nlevels=rng.randint(4, 8))
    return dict(kind=kind, nq=_log(rng, 1024, 32768), ndb=128 * _log(rng, 256, 1024), clusters=256 * rng.randint(1, 2),
                spill=rng.choice([1, 2, 4, 8]))


# ---- what a program keeps ----------------------------------------------------
_contexts = collections.OrderedDict()
_stream = None


def _the_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _context(score="harris", wta=2, octaves=8, cap=10000, form=0):
    """The process's context for these parameters (the last few are kept)."""
    key = (score, wta, octaves, cap, form)
    if key not in _contexts:
        p = orbx.make_params(noctaves=octaves, wta_k=wta, max_pts=cap,
                             score_type=orbx.HARRIS_SCORE if score == "harris" else orbx.FAST_SCORE)
        ctx = orbx.Context(0, p, stream=_the_stream())
        if form:
            t = ctx.get_tuning()
            t.batch_form = form
            ctx.set_tuning(t)
        _contexts[key] = ctx
        while len(_contexts) > 4:
            _contexts.popitem(last=False)
    _contexts.move_to_end(key)
    return _contexts[key]


# ---- inputs ------------------------------------------------------------------
def _clean(rng, w, h):
    """Blobs overdrawn with rectangles and convex polygons, float32 (h, w)."""
    n = 200
    cx, cy = rng.uniform(0, w, n), rng.uniform(0, h, n)
    sig = rng.uniform(2.0, 20.0, n)
    amp = rng.uniform(30.0, 200.0, n) * rng.choice([-1.0, 1.0], n)
    c = torch.tensor(np.stack([cx, cy, sig, amp]), dtype=torch.float32, device="cuda")[:, :, None]
    xs = torch.arange(w, device="cuda", dtype=torch.float32)
    ys = torch.arange(h, device="cuda", dtype=torch.float32)
    gx = torch.exp(-(xs - c[0]) ** 2 / (2 * c[2] ** 2))
    gy = torch.exp(-(ys - c[1]) ** 2 / (2 * c[2] ** 2)) * c[3]
    img = gy.t() @ gx
    m = min(w, h)
    for _ in range(100):
        val = rng.uniform(0.0, 255.0)
        if rng.uniform() < 0.5:
            rw, rh = rng.uniform(0.02, 0.25) * w, rng.uniform(0.02, 0.25) * h
            x0, y0 = rng.uniform(-0.1 * w, w), rng.uniform(-0.1 * h, h)
            xa, xb = int(max(0, x0)), int(min(w, x0 + rw))
            ya, yb = int(max(0, y0)), int(min(h, y0 + rh))
            if xa < xb and ya < yb:
                img[ya:yb, xa:xb] = val
            continue
        k = int(rng.integers(3, 9))
        px, py = rng.uniform(0, w), rng.uniform(0, h)
        rad = rng.uniform(0.02, 0.15) * m
        ang = np.sort(rng.uniform(0, 2 * np.pi, k))
        vx, vy = px + rad * np.cos(ang), py + rad * np.sin(ang)
        x0, x1 = max(0, int(vx.min())), min(w, int(vx.max()) + 1)
        y0, y1 = max(0, int(vy.min())), min(h, int(vy.max()) + 1)
        if x0 >= x1 or y0 >= y1:
            continue
        ex, ey = np.roll(vx, -1) - vx, np.roll(vy, -1) - vy
        # left of every edge: ex * y - ey * x >= ex * vy - ey * vx
        e = torch.tensor(np.stack([ex, ey, ex * vy - ey * vx]), dtype=torch.float32, device="cuda")[:, :, None, None]
        inside = (e[0] * (ys[y0:y1, None] + 0.5) - e[1] * (xs[x0:x1] + 0.5) >= e[2]).all(0)
        img[y0:y1, x0:x1].masked_fill_(inside, val)
    return img


def _finish(img, gen):
    """Noise, rounding to bytes and rows padded with zeros to a multiple of 128."""
    h, w = img.shape
    out = torch.zeros((h, (w + 127) // 128 * 128), dtype=torch.uint8, device="cuda")
    noise = torch.randn((h, w), generator=gen, device="cuda") * 3.0
    out[:, :w] = (img + noise).round().clamp(0, 255).to(torch.uint8)
    return out


def _warp(rng, img):
    """img seen through a random homography (zeros outside)."""
    h, w = img.shape
    th, s = np.deg2rad(rng.uniform(-30.0, 30.0)), rng.uniform(0.8, 1.2)
    tx, ty = rng.uniform(-40.0, 40.0, 2)
    p1, p2 = rng.uniform(-1e-4, 1e-4, 2)
    to_c = np.array([[1, 0, -w / 2], [0, 1, -h / 2], [0, 0, 1]])
    from_c = np.array([[1, 0, w / 2 + tx], [0, 1, h / 2 + ty], [0, 0, 1]])
    m = np.array([[s * np.cos(th), -s * np.sin(th), 0], [s * np.sin(th), s * np.cos(th), 0], [p1, p2, 1]])
    inv = np.linalg.inv(from_c @ m @ to_c)
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    den = inv[2, 0] * x + inv[2, 1] * y + inv[2, 2]
    sx = (inv[0, 0] * x + inv[0, 1] * y + inv[0, 2]) / den * (2.0 / (w - 1)) - 1.0
    sy = (inv[1, 0] * x + inv[1, 1] * y + inv[1, 2]) / den * (2.0 / (h - 1)) - 1.0
    return torch.nn.functional.grid_sample(img[None, None], torch.stack([sx, sy], -1)[None], mode="bilinear",
                                           padding_mode="zeros", align_corners=True)[0, 0]


def _images(rng, w, h, warped):
    """An image, or an image and its warped partner, uint8 (h, align_up(w, 128)) on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 62)))
    clean = _clean(rng, w, h)
    a = _finish(clean, gen)
    return (a, _finish(_warp(rng, clean), gen)) if warped else (a,)


def _descriptor_sets(rng, nq, ndb):
    """Uniform database rows; the first half of the queries are copies of random
    database rows with each bit flipped with probability 0.05, the rest uniform."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 62)))
    db = torch.randint(0, 256, (ndb, 32), generator=gen, device="cuda", dtype=torch.uint8)
    q = torch.randint(0, 256, (nq, 32), generator=gen, device="cuda", dtype=torch.uint8)
    half = nq // 2
    src = torch.randint(0, ndb, (half,), generator=gen, device="cuda")
    flips = torch.rand((half, 32, 8), generator=gen, device="cuda") < 0.05
    bits = (flips * (2 ** torch.arange(8, device="cuda"))).sum(-1).to(torch.uint8)
    q[:half] = db[src] ^ bits
    return q, db


def _pipeline_descriptors(rng, ndb, nq):
    """ndb descriptors of generated images and nq of warped views of the first of them."""
    ctx = _context()
    bufs = orbx.FrameBuffers(10000)
    rows, views, nr, nv = [], [], 0, 0
    while nr < ndb or nv < nq:
        for img, got in zip(_images(rng, LEARNED_IMAGE, LEARNED_IMAGE, nv < nq), (rows, views)):
            orbx.detect_and_compute(ctx, img, LEARNED_IMAGE, LEARNED_IMAGE, bufs=bufs)
            got.append(bufs.desc[:int(bufs.count.item())].clone())
        nr = sum(len(r) for r in rows)
        nv = sum(len(v) for v in views)
    return torch.cat(rows)[:ndb].contiguous(), torch.cat(views)[:nq].contiguous()


# ---- preparing and running ---------------------------------------------------
def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(0x0E0000 + int(seed)))
    s = types.SimpleNamespace(kind=case["kind"])
    stream = _the_stream()
    with torch.cuda.stream(stream):
        globals()["_prepare_" + case["kind"]](s, case, rng)
    stream.synchronize()
    return s


def run(s):
    return globals()["_run_" + s.kind](s)


def _prepare_frame(s, c, rng):
    s.ctx = _context(c["score"], c["wta"], c["octaves"], c["cap"])
    s.w, s.h = c["w"], c["h"]
    s.img, = _images(rng, s.w, s.h, False)
    s.out = orbx.FrameBuffers(c["cap"])


def _run_frame(s):
    o = orbx.detect_and_compute(s.ctx, s.img, s.w, s.h, bufs=s.out)
    return {"points": o.points, "desc": o.desc, "count": o.count}


def _prepare_match(s, c, rng):
    s.ctx = _context(cap=c["cap"])
    s.cap, s.mode = c["cap"], MODES[c["mode"]]
    s.A, s.B = orbx.FrameBuffers(s.cap), orbx.FrameBuffers(s.cap)
    s.A.desc[:c["n1"]], s.B.desc[:c["n2"]] = _descriptor_sets(rng, c["n1"], c["n2"])
    s.A.count.fill_(c["n1"])
    s.B.count.fill_(c["n2"])


def _run_match(s):
    s.ctx.match_ptr(s.A.points, s.A.count, s.A.desc, s.B.count, s.B.desc, s.cap, s.cap, s.mode)
    return {"points": s.A.points}


def _prepare_pair(s, c, rng):
    s.ctx = _context(c["score"], c["wta"], c["octaves"], c["cap"])
    s.w, s.h = c["w"], c["h"]
    s.a, s.b = _images(rng, s.w, s.h, True)
    s.A, s.B = orbx.FrameBuffers(c["cap"]), orbx.FrameBuffers(c["cap"])


def _run_pair(s):
    A, B = s.A, s.B
    s.ctx.pair_ptr(s.a, s.b, s.w, s.h, s.a.shape[1], A.points, A.desc, A.count, B.points, B.desc, B.count)
    return {"points_a": A.points, "desc_a": A.desc, "count_a": A.count, "points_b": B.points, "desc_b": B.desc,
            "count_b": B.count}


def _prepare_pair_host(s, c, rng):
    s.ctx = _context(c["score"], c["wta"], c["octaves"], c["cap"])
    s.w, s.h = c["w"], c["h"]
    s.a, s.b = (t.cpu().pin_memory() for t in _images(rng, s.w, s.h, True))
    s.pts = [np.zeros((c["cap"], 7), np.int32) for _ in range(2)]
    s.desc = [np.zeros((c["cap"], 32), np.uint8) for _ in range(2)]
    s.n = [np.zeros(1, np.int32) for _ in range(2)]


def _run_pair_host(s):
    s.ctx.pair_host(s.a, s.b, s.w, s.h, s.a.shape[1], s.pts[0], s.n[0], s.pts[1], s.n[1], s.desc[0], s.desc[1])
    return {"points_a": s.pts[0], "desc_a": s.desc[0], "count_a": s.n[0], "points_b": s.pts[1], "desc_b": s.desc[1],
            "count_b": s.n[1]}


def _prepare_batch(s, c, rng):
    s.ctx = _context(form=c["form"])
    lay = synth.batch_layout(c["pairs"], c["layout"])
    total = 2 * sum(cap for _, _, cap in lay)
    s.points = torch.zeros((total, 7), dtype=torch.int32, device="cuda")
    s.desc = torch.zeros((total, 32), dtype=torch.uint8, device="cuda")
    s.counts = torch.zeros(2 * len(lay), dtype=torch.int32, device="cuda")
    s.imgs = []
    b = s.batch = types.SimpleNamespace(n=len(lay))
    for f in ("ia", "ib"):
        setattr(b, f, (orbx.Image * b.n)())
    for f in ("oa", "ob"):
        setattr(b, f, (orbx.FrameOut * b.n)())
    at = 0
    for i, (w, h, cap) in enumerate(lay):
        for j, (img, im, out) in enumerate(zip(_images(rng, w, h, True), (b.ia, b.ib), (b.oa, b.ob))):
            s.imgs.append(img)
            im[i] = orbx.Image(img.data_ptr(), w, h, img.shape[1])
            out[i] = orbx.FrameOut(s.points[at:].data_ptr(), s.desc[at:].data_ptr(), s.counts[2 * i + j:].data_ptr(),
                                   cap)
            at += cap


def _run_batch(s):
    s.ctx.batch_pairs(s.batch)
    return {"points": s.points, "desc": s.desc, "counts": s.counts}


def _prepare_knn2(s, c, rng):
    s.ctx, s.mode = _context(), MODES[c["mode"]]
    s.q, s.db = _descriptor_sets(rng, c["nq"], c["ndb"])
    s.dist = torch.zeros((c["nq"], 2), dtype=torch.int32, device="cuda")
    s.idx = torch.zeros((c["nq"], 2), dtype=torch.int32, device="cuda")


def _run_knn2(s):
    s.ctx.knn2_ptr(s.q, s.q.shape[0], s.db, s.db.shape[0], s.dist, s.idx, s.mode)
    return {"dist": s.dist, "idx": s.idx}


def _prepare_ocv(s, c, rng):
    s.ctx = _context()
    s.w, s.h = c["w"], c["h"]
    s.params = orbx.ocv_params(nfeatures=c["nfeatures"], nlevels=c["nlevels"],
                               score_type=orbx.HARRIS_SCORE if c["score"] == "harris" else orbx.FAST_SCORE)
    s.img, = _images(rng, s.w, s.h, False)
    s.cap = c["nfeatures"]
    s.points = torch.zeros((s.cap, 6), dtype=torch.int32, device="cuda")
    s.desc = torch.zeros((s.cap, 32), dtype=torch.uint8, device="cuda")
    s.count = torch.zeros(1, dtype=torch.int32, device="cuda")


def _run_ocv(s):
    status = orbx.lib().orbx_ocv_detect_and_compute(s.ctx.h, ctypes.byref(s.params), s.img.data_ptr(), s.w, s.h,
                                                    s.img.shape[1], s.points.data_ptr(), s.desc.data_ptr(),
                                                    s.count.data_ptr(), s.cap)
    if status != orbx.ORBX_OK:
        raise orbx.OrbxError(status, "orbx_ocv_detect_and_compute")
    return {"points": s.points, "desc": s.desc, "count": s.count}


def _prepare_learned_search(s, c, rng):
    s.ctx = _context()
    db, s.q = _pipeline_descriptors(rng, c["ndb"], c["nq"])
    p = orbx.learned_params(n_clusters=c["clusters"], spill=c["spill"], epochs=2, kmeans_iters=8)
    s.index = orbx.LearnedIndex(s.ctx, db, db[:c["ndb"] // 4096 * 1024], p)
    s.index.set_margin(0.05)  # the closest calls go to exact search


def _run_learned_search(s):
    with torch.cuda.stream(_the_stream()):
        dist, idx, margin, fallback = s.index.search(s.q)
    return {"dist": dist, "idx": idx, "margin": margin, "fallback": fallback}


# ---- what a pass cannot do without -------------------------------------------
def _frame_bytes(w, h, cap):
    # the image in; keypoints and descriptors out (about one keypoint per 1000 pixels, at most the cap)
    return w * h + min(cap, w * h // 1000) * (28 + 32)


def work(case):
    k = case["kind"]
    if k in ("frame", "ocv"):
        return {"bytes": _frame_bytes(case["w"], case["h"], case.get("cap", case.get("nfeatures"))), "flops": 0}
    if k in ("pair", "pair_host"):
        return {"bytes": 2 * _frame_bytes(case["w"], case["h"], case["cap"]), "flops": 0}
    if k == "batch":
        return {"bytes": sum(2 * _frame_bytes(w, h, cap) for w, h, cap in synth.batch_layout(case["pairs"],
                                                                                            case["layout"])),
                "flops": 0}
    if k == "match":
        # 256 bit comparisons and their sum, as a dot product of 256 terms
        return {"bytes": 32 * (case["n1"] + case["n2"]) + 8 * case["n1"], "flops": 512 * case["n1"] * case["n2"]}
    if k == "knn2":
        return {"bytes": 32 * (case["nq"] + case["ndb"]) + 16 * case["nq"], "flops": 512 * case["nq"] * case["ndb"]}
    # learned search: the proposal network, then 8 probed clusters of spill * ndb / clusters rows each
    nq, rows = case["nq"], 8 * case["spill"] * case["ndb"] / case["clusters"]
    return {"bytes": 32 * (nq + case["ndb"]) + 20 * nq,
            "flops": nq * (2 * 512 * (256 + case["clusters"]) + 512 * rows)}


# ---- the same in 64 bits -----------------------------------------------------
def _signs(d):
    bits = (d[:, :, None] >> torch.arange(8, device=d.device, dtype=torch.uint8)) & 1
    return bits.reshape(d.shape[0], 256).to(torch.float64) * 2 - 1


def _nearest2(q, db):
    """(distance, index) of the two nearest rows, ordered by distance and index, by 64-bit arithmetic."""
    t = _signs(db).t()
    col = torch.arange(db.shape[0], device=db.device, dtype=torch.float64)
    dist, idx = [], []
    step = max(1, (1 << 28) // max(1, db.shape[0]))
    for i in range(0, q.shape[0], step):
        key = (256 - _signs(q[i:i + step]) @ t) / 2 * (1 << 22) + col  # exact: below 2^53
        best = torch.topk(key, min(2, db.shape[0]), dim=1, largest=False, sorted=True).values.to(torch.int64)
        dist.append(best >> 22)
        idx.append(best & ((1 << 22) - 1))
    return torch.cat(dist), torch.cat(idx)


def exact(case, seed):
    """Distances and indices of the exact searches.  The other results are whole
    numbers (keypoints and descriptors, byte for byte) or depend on trained weights."""
    if case["kind"] == "knn2":
        s = prepare(case, seed)
        d, i = _nearest2(s.q, s.db)
        return {"dist": d.to(torch.int32), "idx": i.to(torch.int32)}
    if case["kind"] == "match":
        s = prepare(case, seed)
        d, i = _nearest2(s.A.desc[:case["n1"]], s.B.desc[:case["n2"]])
        unique = (d[:, 0] < d[:, 1]) & (d[:, 0] < 64)
        points = torch.zeros((case["cap"], 7), dtype=torch.int32, device=d.device)
        points[:case["n1"], 5] = torch.where(unique, i[:, 0], -1).to(torch.int32)
        points[:case["n1"], 6] = torch.where(unique, d[:, 0], -1).to(torch.int32)
        return {"points": points}
    return None
