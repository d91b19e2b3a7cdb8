"""Raw and blurred pyramid against the oracle, byte for byte, at the sizes where
the tiles and words of k_pyramid_blur end: widths around the 128-column tile, its
64-column halves and 8-column threads, heights around the 26, 42 and 58 row tiles,
images whose base or row pitch leaves word loads unaligned, and the padding that
octave 0 carries when the pitch is the reference's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402
from oracle import oracle as O  # noqa: E402


def _oracle(img, w, h):
    n, oszp = O.layout(w, h, 5)
    store, raw = O.pyramid(img, w, h, n, oszp)
    _, blur = O.blur(store, n, oszp)
    lay = O.split(oszp, n)
    # the oracle filters the columns of each octave; the padding of a blurred row is that of the raw row
    inside = np.concatenate([np.tile(np.arange(p) < ow, oh) for ow, oh, p in
                             zip(lay["widths"], lay["heights"], lay["pitchs"])])
    return raw, np.where(inside, blur, raw)


@pytest.mark.parametrize("shape", [0, 1, 2, 3])
def test_tile_and_word_edges(shape):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = orbx.Context(0, orbx.make_params(noctaves=5, max_pts=64))
    t = ctx.get_tuning()
    t.pyr_tile = shape
    ctx.set_tuning(t)
    rng = np.random.default_rng(shape)
    sizes = [(128 + d, 85 + d) for d in range(-4, 14)]  # one octave
    sizes += [(192, 84), (200, 104), (255, 116), (256, 117), (257, 168), (320, 240), (333, 257), (648, 330), (1281, 1283)]
    for w, h in sizes:
        p0 = (w + 127) // 128 * 128
        for pitch, shift in ((p0, 0), (p0 + 128, 0), (w, 0), (p0, 1), (p0 + 4, 4)):
            buf = torch.from_numpy(rng.integers(0, 256, (h + 1) * pitch + 16, dtype=np.uint8)).cuda()
            out = orbx.FrameBuffers(64)
            ctx.detect_and_compute_ptr(buf.data_ptr() + shift, w, h, pitch, out.points, out.desc, out.count)
            ctx.sync()
            got = ctx.debug_buffers(w, h)
            rows = buf.cpu().numpy()[shift:shift + h * pitch].reshape(h, pitch)
            img = np.zeros((h, p0), np.uint8)
            img[:, :w] = rows[:, :w]
            if pitch == p0:
                img[:, w:] = rows[:, w:]
            raw, blur = _oracle(img, w, h)
            assert np.array_equal(got["pyr"], raw), (w, h, pitch, shift)
            assert np.array_equal(got["blur"], blur), (w, h, pitch, shift)
    ctx.close()
