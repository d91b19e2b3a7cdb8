"""Batches with changing buffers.  Calls of one layout replay a graph, whichever buffers
they come with; inside a caller's stream capture a call is recorded only when its tables
are on the device already, and a captured call is not affected by later ones.  Both
forms, against orbx_pair on each pair."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import orbx  # noqa: E402
import synth  # noqa: E402

SIZES = [(320, 240, 500), (333, 257, 200), (640, 480, 1000)]


def _make(seed):
    return orbx.PairBatch([(*synth.make_pair(w, h, seed=seed + k)[:2], w, h, cap) for k, (w, h, cap) in enumerate(SIZES)])


@pytest.fixture(scope="module")
def stream():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.cuda.Stream()


@pytest.fixture(scope="module")
def sets(stream):
    """Two batches of one layout and what each pair gives alone."""
    out = []
    single = orbx.Context(0, orbx.make_params(max_pts=1000))
    for seed in (300, 400):
        pb, want = _make(seed), []
        for i, (w, h, cap) in enumerate(SIZES):
            single.init(orbx.make_params(max_pts=cap))
            (a, b), A, B = pb.imgs[i], orbx.FrameBuffers(cap), orbx.FrameBuffers(cap)
            single.pair_ptr(a, b, w, h, a.shape[1], A.points, A.desc, A.count, B.points, B.desc, B.count)
            single.sync()
            want.append(A.to_host() + B.to_host())
        out.append((pb, want))
    single.close()
    return out


def _clear(pb):
    for A, B in pb.outs:
        for f in (A, B):
            f.points.fill_(-7)
            f.desc.fill_(7)
            f.count.fill_(0)
    torch.cuda.synchronize()


def _check(pb, want):
    for i in range(len(SIZES)):
        assert all(np.array_equal(g, w) for g, w in zip(pb.results(i), want[i])), i


def _context(stream, form):
    ctx = orbx.Context(0, orbx.make_params(max_pts=1000), stream=stream)
    t = ctx.get_tuning()
    t.batch_form = form
    t.pair_form = form
    ctx.set_tuning(t)
    return ctx


def _capture(stream, call, mode="relaxed"):
    """The graph of `call`, or None when the call was refused."""
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    ok = True
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode=mode)
        try:
            call()
        except orbx.OrbxError:
            ok = False
        finally:
            g.capture_end()
    return g if ok else None


@pytest.mark.parametrize("form", [0, 1])
def test_graph_replays_with_other_buffers(stream, sets, form):
    ctx = _context(stream, form)
    for k in (0, 0, 0, 1, 0, 1, 1):  # plain, captured, replayed, then with changing buffers
        pb, want = sets[k]
        _clear(pb)
        ctx.batch_pairs(pb)
        ctx.sync()
        _check(pb, want)
    ctx.close()


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
@pytest.mark.parametrize("form", [0, 1])
def test_capture_with_other_buffers_is_refused(stream, sets, form, mode):
    (a, want_a), (b, want_b) = sets
    ctx = _context(stream, form)
    assert _capture(stream, lambda: ctx.batch_pairs(a), mode) is None  # never run
    for pb, want in ((a, want_a), (b, want_b), (a, want_a)):
        _clear(a)
        _clear(b)
        ctx.batch_pairs(pb)
        ctx.sync()
        _check(pb, want)
        other, other_want = (b, want_b) if pb is a else (a, want_a)
        assert _capture(stream, lambda: ctx.batch_pairs(other), mode) is None
        # the refused call has left nothing behind: both run as before
        _clear(other)
        ctx.batch_pairs(other)
        ctx.sync()
        _check(other, other_want)
        _check(pb, want)
    ctx.close()


@pytest.mark.parametrize("form", [0, 1])
def test_captured_batch_keeps_its_buffers(stream, sets, form):
    (a, want_a), (b, want_b) = sets
    ctx = _context(stream, form)
    ctx.batch_pairs(a)
    ctx.sync()
    graph_a = _capture(stream, lambda: ctx.batch_pairs(a))
    ctx.batch_pairs(b)
    ctx.sync()
    graph_b = _capture(stream, lambda: ctx.batch_pairs(b))
    assert graph_a is not None and graph_b is not None
    for _ in range(2):
        for graph, pb, want, other in ((graph_a, a, want_a, b), (graph_b, b, want_b, a)):
            ctx.batch_pairs(other)
            ctx.sync()
            _clear(a)
            _clear(b)
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            _check(pb, want)
            assert all(int(f.count.item()) == 0 for AB in other.outs for f in AB)  # not written
    ctx.close()


@pytest.mark.parametrize("form", [0, 1])
def test_captured_pair(stream, sets, form):
    (pb, want), _ = sets
    w, h, cap = SIZES[2]
    ctx = _context(stream, form)
    (da, db), (A, B) = pb.imgs[2], pb.outs[2]

    def call():
        ctx.pair_ptr(da, db, w, h, da.shape[1], A.points, A.desc, A.count, B.points, B.desc, B.count)

    def check():
        assert all(np.array_equal(g, e) for g, e in zip(pb.results(2), want[2]))

    assert _capture(stream, call) is None  # workspaces not there yet
    for _ in range(3):
        _clear(pb)
        call()
        ctx.sync()
        check()
    graph = _capture(stream, call)
    assert graph is not None
    _clear(pb)
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    check()
    ctx.close()
