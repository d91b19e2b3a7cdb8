"""The tensor-core matcher and rerank where their tiles end: 240 database rows per tile,
in two column parts of 120, examined 60 at a time in groups of 15.  Few distinct
descriptors, so that most distances tie and the order by index decides."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402

EDGES = [n + d for n in (15, 60, 120, 180, 240, 300, 360, 480, 720) for d in (-1, 0, 1)]


@pytest.mark.parametrize("nq", [1, 128, 129, 256, 300])
def test_matcher_rows_around_tiles_parts_and_chunks(nq):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2000 + nq)
    ctx = orbx.Context(0)
    base = torch.randint(0, 256, (30, 32), generator=gen, device="cuda", dtype=torch.uint8)
    for ndb in EDGES:
        def draw(n):
            d = base[torch.randint(0, 30, (n,), generator=gen, device="cuda")]
            d[:, 9] ^= torch.randint(0, 4, (n,), generator=gen, device="cuda").to(torch.uint8)
            return d
        q, db = draw(nq), draw(ndb)
        db[-1] = q[-1]  # the last row is some query's nearest
        torch.cuda.synchronize()
        want = orbx.knn2(ctx, q, db, orbx.MATCH_POPC)
        got = orbx.knn2(ctx, q, db, orbx.MATCH_IMMA)
        ctx.sync()
        for w, g in zip(want, got):
            assert torch.equal(w, g), ndb
    ctx.close()


@pytest.mark.parametrize("per_cluster", [3, 130])
def test_rerank_lists_around_tiles_parts_and_chunks(per_cluster):
    """Lists of exactly those lengths: an index whose centroids are far apart, loaded
    over a database with so many near copies of each."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from test_gpu_learned import CKPT_HEAD
    rng = np.random.default_rng(per_cluster)
    ctx = orbx.Context(0)
    rows = rng.integers(0, 256, (2000, 32), dtype=np.uint8)
    t = torch.from_numpy(rows).cuda()
    p = orbx.learned_params(n_clusters=256, hidden=512, epochs=0, batch=512, kmeans_iters=1, spill=1)
    built = orbx.LearnedIndex(ctx, t, t[:512].contiguous(), p)
    blob = built.save()
    built.close()
    cent = np.frombuffer(blob, dtype=np.uint8, count=256 * 32, offset=CKPT_HEAD).reshape(256, 32)
    sizes = [1, 2] + EDGES
    sizes += [8] * (256 - len(sizes))
    db = np.repeat(cent, sizes, axis=0)
    db[np.arange(len(db)), rng.integers(0, 32, len(db))] ^= (1 << rng.integers(0, 3, len(db))).astype(np.uint8)
    of = np.repeat(np.arange(256), sizes)
    perm = rng.permutation(len(db))
    db, of = db[perm], of[perm]
    # queries around every centroid: 130 make a second work item of a cluster
    q = np.repeat(cent, per_cluster, axis=0)
    q[np.arange(len(q)), rng.integers(0, 32, len(q))] ^= (1 << rng.integers(0, 8, len(q))).astype(np.uint8)
    tdb, tq = torch.from_numpy(db).cuda(), torch.from_numpy(q).cuda()
    idx = orbx.LearnedIndex.load(ctx, blob, tdb)
    try:
        assert np.array_equal(np.diff(idx.export(weights=False)["offsets"]), np.bincount(of, minlength=256))
        out = []
        for form in (orbx.RERANK_TENSOR, orbx.RERANK_POPC):
            idx.set_rerank(form)
            out.append(idx.search(tq))
            ctx.sync()
        for a, b in zip(*out):
            assert torch.equal(a, b)
        assert float((out[0][0][:, 0] <= 3).float().mean()) > 0.5  # the right lists were probed
    finally:
        idx.close()
        ctx.close()
