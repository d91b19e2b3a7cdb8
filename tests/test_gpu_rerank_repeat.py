"""The tensor-core rerank over many searches in a row: a packed database tile that
is given back before all of its words are read corrupts about one tile in 50000,
so one search says nothing; every one of 300 has to equal the XOR-popc form."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402


@pytest.mark.parametrize("spill", [1, 4])
def test_many_searches_equal_the_popcount_form(spill):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(spill)

    def noisy(rows, p):
        flips = torch.rand((len(rows), 32, 8), generator=gen, device="cuda") < p
        return rows ^ (flips * (2 ** torch.arange(8, device="cuda"))).sum(-1).to(torch.uint8)

    centers = torch.randint(0, 256, (2048, 32), generator=gen, device="cuda", dtype=torch.uint8)
    db = noisy(centers[torch.randint(0, 2048, (131072,), generator=gen, device="cuda")], 0.12)
    q = noisy(db[torch.randint(0, 131072, (32768,), generator=gen, device="cuda")], 0.08)
    torch.cuda.synchronize()
    ctx = orbx.Context(0)
    idx = orbx.LearnedIndex(ctx, db, db[:32768].contiguous(),
                            orbx.learned_params(n_clusters=512, spill=spill, epochs=1, kmeans_iters=4))
    try:
        idx.set_rerank(orbx.RERANK_POPC)
        want = idx.search(q)
        ctx.sync()
        idx.set_rerank(orbx.RERANK_TENSOR)
        for _ in range(50):
            got = [idx.search(q) for _ in range(6)]
            ctx.sync()
            for g in got:
                assert torch.equal(g[0], want[0]) and torch.equal(g[1], want[1])
    finally:
        idx.close()
        ctx.close()
