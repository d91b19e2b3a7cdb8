"""The banded form of orbx_pair_host as the first library call of a process, when none of
its kernels is loaded yet: the launch that waits for the bands must not keep the kernel
behind it from loading."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/cuda-orb_b200"]
import numpy as np
import torch
import orbx, synth
w, h, cap = 640, 480, 5000
a, b, _ = synth.make_pair(w, h, seed=47)
if sys.argv[3] == "pinned":
    a, b = (torch.from_numpy(x).pin_memory().numpy() for x in (a, b))
ctx = orbx.Context(0, orbx.make_params(max_pts=cap))

def run(bands):
    t = ctx.get_tuning()
    t.upload_bands, t.host_overlap = bands, 0
    ctx.set_tuning(t)
    pa, pb = np.zeros((cap, 7), np.int32), np.zeros((cap, 7), np.int32)
    na, nb = np.zeros(1, np.int32), np.zeros(1, np.int32)
    da, db = np.zeros((cap, 32), np.uint8), np.zeros((cap, 32), np.uint8)
    ctx.pair_host(a, b, w, h, a.shape[1], pa, na, pb, nb, da, db)
    return pa, na, pb, nb, da, db

bands = int(sys.argv[2])
got = [run(bands) for _ in range(3)]
want = run(0)
assert want[1][0] > 100
for g in got:
    assert all(np.array_equal(x, y) for x, y in zip(g, want))
print("same")
"""


@pytest.mark.parametrize("bands,memory", [(4, "pinned"), (1, "pinned"), (4, "pageable")])
def test_bands_first(bands, memory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    env = dict(os.environ, CUDA_MODULE_LOADING="LAZY")
    out = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(bands), memory], capture_output=True, text=True, env=env,
                         timeout=300)
    assert out.returncode == 0 and out.stdout.strip().endswith("same"), out.stderr[-2000:]
