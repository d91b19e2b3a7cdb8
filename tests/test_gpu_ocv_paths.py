"""The OpenCV-compatible mode where its kernels branch: images whose rows do or do
not start on 16 bytes (in place or copied), one level or several, and the two
retains, whose results must be the best keys of the unlimited detection with
equal scores resolved in raster order."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402
import synth  # noqa: E402


@pytest.fixture(scope="module")
def ctx():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = orbx.Context(0)
    yield c
    c.close()


def _run(ctx, img, w, h, pitch, shift, **kw):
    p = orbx.ocv_params(**kw)
    buf = torch.zeros(shift + h * pitch + 16, dtype=torch.uint8, device="cuda")
    view = buf[shift:shift + h * pitch].view(h, pitch)
    view[:, :w] = torch.from_numpy(img[:, :w]).cuda()
    cap = p.nfeatures
    pts = torch.zeros((cap, 6), dtype=torch.int32, device="cuda")
    desc = torch.zeros((cap, 32), dtype=torch.uint8, device="cuda")
    n = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = orbx.lib().orbx_ocv_detect_and_compute(ctx.h, ctypes.byref(p), view.data_ptr(), w, h, pitch, pts.data_ptr(),
                                                desc.data_ptr(), n.data_ptr(), cap)
    assert st == orbx.ORBX_OK
    ctx.sync()
    k = int(n.item())
    return pts[:k].cpu().numpy().copy().view(orbx.OCV_KEYPOINT_DTYPE).reshape(k), desc[:k].cpu().numpy()


@pytest.mark.parametrize("w,h,nlevels", [(333, 257, 8), (64, 64, 1), (65, 90, 2), (130, 131, 3), (640, 480, 1)])
def test_row_alignment(ctx, w, h, nlevels):
    img = synth.make_image(w, h, seed=61)
    p0 = (w + 15) // 16 * 16
    want = _run(ctx, img, w, h, p0, 0, nfeatures=400, nlevels=nlevels)
    for pitch, shift in ((w + 3, 0), (p0, 5), (p0 + 16, 0)):
        got = _run(ctx, img, w, h, pitch, shift, nfeatures=400, nlevels=nlevels)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("budget", [1, 7, 64, 300, 900])
def test_retain_keeps_the_best(ctx, budget):
    w, h = 640, 480
    img = synth.make_image(w, h, seed=62)
    every, edesc = _run(ctx, img, w, h, w, 0, nfeatures=8000, nlevels=1, score_type=orbx.FAST_SCORE, fast_threshold=8)
    assert 1000 < len(every) < 8000
    raster = every["y"].astype(np.int64) * w + every["x"].astype(np.int64)
    order = np.lexsort((raster, -every["response"]))
    assert np.array_equal(order, np.arange(len(every)))  # decreasing score, then raster order
    best, bdesc = _run(ctx, img, w, h, w, 0, nfeatures=budget, nlevels=1, score_type=orbx.FAST_SCORE, fast_threshold=8)
    assert np.array_equal(best, every[:budget]) and np.array_equal(bdesc, edesc[:budget])
    # Harris: the best `budget` by Harris score of the best 2 * budget by FAST score
    harris, _ = _run(ctx, img, w, h, w, 0, nfeatures=4000, nlevels=1, fast_threshold=8)
    score = {(x, y): r for x, y, r in zip(harris["x"], harris["y"], harris["response"])}
    pool = every[:2 * budget]
    r = np.array([score[(x, y)] for x, y in zip(pool["x"], pool["y"])], np.float32)
    order = np.lexsort((raster[:2 * budget], -r))[:budget]
    got, _ = _run(ctx, img, w, h, w, 0, nfeatures=budget, nlevels=1, fast_threshold=8)
    assert np.array_equal(got["x"], pool["x"][order]) and np.array_equal(got["y"], pool["y"][order])
    assert np.array_equal(got["response"], r[order])
