"""Score map (FAST-9 corners, Harris or FAST score, octave merge) against the
oracle, bit for bit, where the packed pre-test and the staged halos of k_detect
can go wrong: every kind of threshold on images with extreme contrasts, and
sizes that end inside a detect tile, one pixel past it and on it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402
from oracle import oracle as O  # noqa: E402


def _image(rng, w, h, kind):
    if kind == "noise":
        return rng.integers(0, 256, (h, w), dtype=np.uint8)
    if kind == "extreme":
        return rng.choice(np.array([0, 1, 127, 128, 254, 255], np.uint8), (h, w))
    y, x = np.mgrid[0:h, 0:w]  # blocks of 5 x 7 pixels: corners at every octave
    return (((x // 5 + y // 7) % 2) * 200 + rng.integers(0, 30, (h, w))).astype(np.uint8)


@pytest.mark.parametrize("score", [orbx.HARRIS_SCORE, orbx.FAST_SCORE])
@pytest.mark.parametrize("thr", [0, 1, 20, 127, 128, 254, 255])
def test_score_map(score, thr):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = orbx.Context(0, orbx.make_params(noctaves=5, max_pts=64, score_type=score, fast_threshold=thr))
    rng = np.random.default_rng(thr)
    for w, h, kind in ((128, 96, "noise"), (129, 97, "extreme"), (191, 161, "blocks"), (333, 330, "extreme"),
                       (640, 650, "noise"), (1290, 1281, "blocks")):
        n, oszp = O.layout(w, h, 5)
        img = np.zeros((h, int(oszp[3 * n])), np.uint8)
        img[:, :w] = _image(rng, w, h, kind)
        orbx.detect_and_compute(ctx, torch.from_numpy(img).cuda(), w, h)
        ctx.sync()
        got = ctx.debug_buffers(w, h)
        store, _ = O.pyramid(img, w, h, n, oszp)
        vmap, layer = O.score_map(store, n, oszp, thr, score == orbx.HARRIS_SCORE)
        assert np.array_equal(got["vmap"].view(np.uint32), np.asarray(vmap, np.float32).reshape(-1).view(np.uint32)), (w, h)
        on = got["vmap"] > 0
        assert np.array_equal(got["layer"][on], np.asarray(layer).reshape(-1)[on]), (w, h)
    ctx.close()
