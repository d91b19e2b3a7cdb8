"""The OpenCV-compatible mode on images that a program cuts out of others: views whose
last pixel ends their allocation, read in place or copied, give the same results."""
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


def _run(ctx, ptr, w, h, pitch, **kw):
    p = orbx.ocv_params(**kw)
    cap = p.nfeatures
    pts = torch.zeros((cap, 6), dtype=torch.int32, device="cuda")
    desc = torch.zeros((cap, 32), dtype=torch.uint8, device="cuda")
    n = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = orbx.lib().orbx_ocv_detect_and_compute(ctx.h, ctypes.byref(p), ptr, w, h, pitch, pts.data_ptr(),
                                                desc.data_ptr(), n.data_ptr(), cap)
    assert st == orbx.ORBX_OK
    ctx.sync()
    k = int(n.item())
    return pts[:k].cpu().numpy().copy().view(orbx.OCV_KEYPOINT_DTYPE).reshape(k), desc[:k].cpu().numpy()


@pytest.mark.parametrize("w,h,x0,nlevels", [(320, 240, 320, 4), (311, 201, 16, 3), (273, 131, 368, 1), (129, 131, 496, 2)])
def test_view_at_the_end_of_its_allocation(ctx, w, h, x0, nlevels):
    pitch = 640
    img = synth.make_image(w, h, seed=63)[:, :w]
    size = (h - 1) * pitch + x0 + w  # ends with the view's last pixel
    parent = torch.randint(0, 256, (size,), dtype=torch.uint8, device="cuda")
    assert parent.data_ptr() % 16 == 0
    rows = torch.as_strided(parent, (h, w), (pitch, 1), x0)
    rows.copy_(torch.from_numpy(np.ascontiguousarray(img)))
    got = _run(ctx, parent.data_ptr() + x0, w, h, pitch, nfeatures=400, nlevels=nlevels)
    copied = torch.zeros(h * (w + 3) + 16, dtype=torch.uint8, device="cuda")  # rows off 16 bytes: copied
    torch.as_strided(copied, (h, w), (w + 3, 1), 1).copy_(rows)
    want = _run(ctx, copied.data_ptr() + 1, w, h, w + 3, nfeatures=400, nlevels=nlevels)
    assert len(want[0]) > 0
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_more_rows_than_a_grid_dimension(ctx):
    """An image of more than 4 * 65535 rows, in place and copied: the keypoints of its
    last rows are those of the same rows alone.  Level 1 is half of level 0, so an even
    offset keeps its pixels."""
    w, h, off = 160, 400, 262200
    tail = torch.zeros((h, w), dtype=torch.uint8, device="cuda")
    tail[100:] = torch.from_numpy(np.ascontiguousarray(synth.make_image(w, 300, seed=64)[:, :w]))
    kw = dict(nfeatures=2000, nlevels=2, scale_factor=2.0)
    want = _run(ctx, tail.data_ptr(), w, h, w, **kw)
    assert len(want[0]) > 20 and want[0]["octave"].max() == 1
    for pitch, shift in ((w, 0), (w + 1, 1)):
        tall = torch.zeros((off + h) * pitch + 1, dtype=torch.uint8, device="cuda")
        torch.as_strided(tall, (h, w), (pitch, 1), shift + off * pitch).copy_(tail)
        pts, desc = _run(ctx, tall.data_ptr() + shift, w, off + h, pitch, **kw)
        pts["y"] -= off
        assert np.array_equal(pts, want[0]) and np.array_equal(desc, want[1])
