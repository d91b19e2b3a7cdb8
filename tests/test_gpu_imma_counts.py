"""The tensor-core matcher with counts on the device far below the capacities, in a
context that has served larger ones: its merge scratch is shared out by the counts."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402


@pytest.mark.parametrize("caps", [(300,), (10000, 1000), (2500, 20000, 2500)])
def test_counts_below_the_capacity(caps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(sum(caps))
    ctx = orbx.Context(0)
    for cap in caps:
        A, B = orbx.FrameBuffers(cap), orbx.FrameBuffers(cap)
        base = torch.randint(0, 256, (50, 32), generator=gen, device="cuda", dtype=torch.uint8)
        for n1 in (1, 128, 129, 256, 257, 600, 2100, cap):
            for n2 in (0, 240, 9000):
                if n1 > cap or n2 > cap:
                    continue
                for f, n in ((A, n1), (B, n2)):
                    f.desc[:n] = base[torch.randint(0, 50, (n,), generator=gen, device="cuda")]
                    f.desc[:n, 3] ^= torch.randint(0, 8, (n,), generator=gen, device="cuda").to(torch.uint8)
                    f.count.fill_(n)
                got = []
                for mode in (orbx.MATCH_POPC, orbx.MATCH_IMMA):
                    A.points.fill_(-7)
                    torch.cuda.synchronize()
                    ctx.match_ptr(A.points, A.count, A.desc, B.count, B.desc, cap, cap, mode)
                    ctx.sync()
                    got.append(A.points.clone())
                assert torch.equal(*got), (cap, n1, n2)
    ctx.close()
