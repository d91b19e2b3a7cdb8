"""The popcount matcher where its blocks end: queries around its 128-query tile,
train rows around its four-row steps, row groups, 512-row chunks and splits, on
descriptors with few distinct values, so that most distances tie and the order by
index decides.  Both the k = 2 lists and the keypoint fields, counts known to the
host and counts on the device, against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402
from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("nq", [1, 31, 127, 128, 129, 257])
def test_tile_chunk_and_tie_edges(nq):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(nq)
    ctx = orbx.Context(0, orbx.make_params(max_pts=4096))
    base = rng.integers(0, 256, (6, 32), dtype=np.uint8)
    for ndb in (0, 1, 2, 3, 4, 5, 15, 16, 17, 63, 64, 65, 130, 511, 512, 513, 1030, 2049, 4096):
        def draw(n):
            d = base[rng.integers(0, 6, n)]
            d[:, 0] ^= rng.integers(0, 4, n).astype(np.uint8)
            return d
        q, db = draw(nq), draw(ndb)
        tq, tdb = torch.from_numpy(q).cuda(), torch.from_numpy(db.reshape(ndb, 32)).cuda()
        dist, idx = orbx.knn2(ctx, tq, tdb, orbx.MATCH_POPC)
        A = orbx.FrameBuffers(4096)
        B = orbx.FrameBuffers(4096)
        A.desc[:nq] = tq
        B.desc[:ndb] = tdb
        A.count.fill_(nq)
        B.count.fill_(ndb)
        torch.cuda.synchronize()
        ctx.match_ptr(A.points, A.count, A.desc, B.count, B.desc, 4096, 4096, orbx.MATCH_POPC)
        ctx.sync()
        od, oi = O.knn2(q, db)
        assert np.array_equal(dist.cpu().numpy().view(np.uint32), np.asarray(od, np.uint32).reshape(nq, 2)), ndb
        assert np.array_equal(idx.cpu().numpy(), np.asarray(oi, np.int32).reshape(nq, 2)), ndb
        m, d = O.match(q, db)
        got = A.points[:nq].cpu().numpy()
        assert np.array_equal(got[:, 5], m) and np.array_equal(got[:, 6], d), ndb
    ctx.close()


@pytest.mark.parametrize("nq", [1, 127, 128, 129, 255, 256, 257, 600])
def test_tensor_core_form_equals_popcount_form(nq):
    """One or two query tiles per block, database rows around the 256-row tiles, few
    or many splits (which share their bounds), and distances that mostly tie."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(1000 + nq)
    ctx = orbx.Context(0, orbx.make_params(max_pts=1024))
    base = rng.integers(0, 256, (40, 32), dtype=np.uint8)
    base[0], base[1] = 0, 255
    for ndb in (1, 2, 31, 255, 256, 257, 511, 513, 2048, 9000, 70001):
        def draw(n):
            d = base[rng.integers(0, 40, n)]
            d[:, 5] ^= rng.integers(0, 8, n).astype(np.uint8)
            return torch.from_numpy(d).cuda()
        q, db = draw(nq), draw(ndb)
        torch.cuda.synchronize()
        want = orbx.knn2(ctx, q, db, orbx.MATCH_POPC)
        got = orbx.knn2(ctx, q, db, orbx.MATCH_IMMA)
        ctx.sync()
        for w, g in zip(want, got):
            assert torch.equal(w, g), ndb
    ctx.close()


@pytest.mark.parametrize("nq", [2100, 2305])
def test_panels_of_a_large_database(nq):
    """A database that goes by panels, all queries against one before the next: the
    last block of queries has one query tile, between blocks with two."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(nq)
    ndb = 3072 * 240 + 77
    db = torch.randint(0, 256, (ndb, 32), generator=gen, device="cuda", dtype=torch.uint8)
    q = torch.randint(0, 256, (nq, 32), generator=gen, device="cuda", dtype=torch.uint8)
    db[ndb - 1000:] = db[:1000]  # equal distances far apart
    q[:500] = db[:500]
    torch.cuda.synchronize()
    ctx = orbx.Context(0, orbx.make_params(max_pts=1024))
    want = orbx.knn2(ctx, q, db, orbx.MATCH_POPC)
    got = orbx.knn2(ctx, q, db, orbx.MATCH_IMMA)
    ctx.sync()
    for w, g in zip(want, got):
        assert torch.equal(w, g)
    ctx.close()
