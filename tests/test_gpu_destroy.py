"""A destroyed context gives its device memory back, whichever forms it ran."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402
import synth  # noqa: E402


@pytest.mark.parametrize("pair_form,bands,overlap", [(0, 0, 0), (1, 0, 0), (0, 4, 0), (0, 0, 1)])
def test_memory_is_given_back(pair_form, bands, overlap):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    w, h, cap = 320, 240, 40000  # 20 MB of matcher scratch
    a, b, _ = synth.make_pair(w, h, seed=51)

    def once():
        ctx = orbx.Context(0, orbx.make_params(max_pts=cap))
        t = ctx.get_tuning()
        t.pair_form, t.upload_bands, t.host_overlap = pair_form, bands, overlap
        ctx.set_tuning(t)
        pa, pb = np.zeros((cap, 7), np.int32), np.zeros((cap, 7), np.int32)
        na, nb = np.zeros(1, np.int32), np.zeros(1, np.int32)
        for _ in range(3):
            ctx.pair_host(a, b, w, h, a.shape[1], pa, na, pb, nb)
        ctx.close()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    first = once()
    for _ in range(4):
        last = once()
    assert first - last < 8 << 20
