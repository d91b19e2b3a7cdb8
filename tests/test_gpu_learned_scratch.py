"""The learned search's scratch, laid out anew when the query count grows: searches of
any counts in any order give what the whole set gives, for both proposals."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402


@pytest.mark.parametrize("kw", [dict(n_clusters=256, hidden=512, epochs=1, batch=512, kmeans_iters=3, spill=2),
                                dict(proposal=orbx.PROPOSAL_LSH, lsh_bits=8, n_clusters=256)])
def test_growing_query_counts(kw):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(49)
    db = torch.randint(0, 256, (9000, 32), generator=gen, device="cuda", dtype=torch.uint8)
    q = db[torch.randint(0, 9000, (4000,), generator=gen, device="cuda")]
    q[:, 7] ^= torch.randint(0, 256, (4000,), generator=gen, device="cuda").to(torch.uint8)
    torch.cuda.synchronize()
    ctx = orbx.Context(0)
    idx = orbx.LearnedIndex(ctx, db, db[:1024].contiguous(), orbx.learned_params(**kw))
    try:
        idx.set_margin(0.5)  # part of the queries go to exact search
        got = []
        for n in (1, 129, 2500, 300, 4000, 4000):
            d, i, _, _ = idx.search(q[:n].contiguous())
            ctx.sync()
            got.append((n, d.clone(), i.clone()))
        for n, d, i in got:
            assert torch.equal(d, got[-1][1][:n]) and torch.equal(i, got[-1][2][:n]), n
    finally:
        idx.close()
        ctx.close()
