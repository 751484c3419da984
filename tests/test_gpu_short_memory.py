"""Device memory that runs short at any point of a call: what is not needed is
done without, with the same results, and a call that cannot go on says
DYG_ENOMEM and leaves handles that work."""
import contextlib
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import dyg, same_graph  # noqa: F401

pytestmark = pytest.mark.gpu
EINVAL, ENOMEM = 1, 2


@contextlib.contextmanager
def failing(dyg, skip, fail):  # noqa: F811
    """Allocations skip + 1 to skip + fail of this thread fail."""
    f = dyg.lib().dyg_testing_fail_allocations
    f.argtypes, f.restype = [C.c_uint32, C.c_uint32], None
    f(skip, fail)
    try:
        yield
    finally:
        f(0, 0)


def some_graph(n, rng):
    """A path, a row of 700 slots, one of 5,000, repeated edges and self-loops."""
    s = np.concatenate([np.arange(n - 1), np.zeros(700, np.int64), np.full(5000, 9), [3, 3, 5]])
    d = np.concatenate([np.arange(1, n), 2 + np.arange(700), 20 + np.arange(5000), [3, 3, 6]])
    o = rng.permutation(len(s))
    return s[o].astype(np.uint32), d[o].astype(np.uint32), rng.uniform(0.5, 2.0, len(s)).astype(np.float32)


@pytest.mark.parametrize("fail", [1, 2, 100])
def test_build(dyg, oracle, fail):  # noqa: F811
    n = 6000
    s, d, w = some_graph(n, np.random.default_rng(1))
    go = oracle.OGraph(n, s, d, w)
    done = 0
    for skip in range(14):
        try:
            with failing(dyg, skip, fail):
                g = dyg.Graph.from_edges(n, s, d, w)
                assert dyg.lib().dyg_last_error_string() == b""
        except dyg.DygError as e:
            assert e.status == ENOMEM and fail > 1
            continue
        done += 1
        same_graph(g, go)
        assert g.info()["n_slots"] == 2 * len(s)
    # one failure is made up for by the second try; of more, those of the
    # list's copies are by the host
    assert done == {1: 14, 2: 9, 100: 3}[fail]


def test_build_by_the_host_checks_its_input(dyg):  # noqa: F811
    m = 70_000
    s, d, w = np.arange(m, dtype=np.uint32), np.arange(1, m + 1, dtype=np.uint32), np.ones(m, np.float32)
    d[66_000] = m + 1
    with failing(dyg, 5, 2), pytest.raises(dyg.DygError) as e:
        dyg.Graph.from_edges(m + 1, s, d, w)
    assert e.value.status == EINVAL and "dst[66000]" in str(e.value)


@pytest.mark.parametrize("fail", [1, 2, 100])
@pytest.mark.parametrize("cap", [None, 50])
def test_export(dyg, fail, cap):  # noqa: F811
    n = 6000
    g = dyg.Graph.from_edges(n, *some_graph(n, np.random.default_rng(2)))
    rp0, col0, w0 = g.export()
    k = len(col0) if cap is None else cap
    for skip in range(5):
        rp, col, w = np.zeros(n + 1, np.uint64), np.zeros(len(col0), np.uint32), np.zeros(len(col0), np.float32)
        with failing(dyg, skip, fail):
            rc = dyg.lib().dyg_graph_export(g.handle, rp.ctypes.data, col.ctypes.data, w.ctypes.data, k)
        assert rc == (0 if cap is None else 4)
        assert np.array_equal(rp, rp0) and np.array_equal(col[:k], col0[:k]) and np.array_equal(w[:k], w0[:k])
        assert not col[k:].any() and not w[k:].any()


def cycles(k, rng):
    """k cycles of 3..200 vertices, whose deleted edges have winners of up to 199
    moves: more records than a call starts with room for."""
    sizes = np.where(np.arange(k) % 4 == 0, 200, rng.integers(3, 40, k))
    off = np.concatenate([[0], np.cumsum(sizes)])
    base, L = np.repeat(off[:-1], sizes), np.repeat(sizes, sizes)
    i = np.arange(off[-1]) - base
    # and a row of 400 slots: weighted walks have an index
    leaf = np.arange(400)
    s = np.concatenate([base + i, np.full(400, off[-1])]).astype(np.uint32)
    d = np.concatenate([base + (i + 1) % L, off[-1] + 1 + leaf]).astype(np.uint32)
    return int(off[-1]) + 401, off[:-1], s, d, rng.uniform(0.5, 2.0, len(s)).astype(np.float32)


@pytest.mark.parametrize("fail", [1, 2, 3, 100])
@pytest.mark.parametrize("transition", [0, 1])
@pytest.mark.parametrize("call", ["delete", "insert", "file_delete", "file_insert"])
def test_updates(dyg, oracle, call, transition, fail):  # noqa: F811
    """Every allocation of a call on fresh handles fails in turn.  With one
    failure the call goes on (a second try, or without the scratch); with more it
    goes on or says DYG_ENOMEM; and the handles work afterwards."""
    rng = np.random.default_rng(3)
    k = 300
    n, first, gs, gd, gw = cycles(k, rng)
    kw = dict(slack_per_row=0, arena_headroom=0.0)   # insertions and recoveries grow the arenas
    G0 = dyg.Graph.from_edges(n, gs, gd, gw, **kw)
    H0 = dyg.Graph.from_edges(n, *(a[np.r_[first, -400:0]] for a in (gs, gd, gw)), **kw)
    es = rng.integers(0, n, 3000).astype(np.uint32)
    ed = ((es + 1 + rng.integers(0, n - 1, 3000)) % n).astype(np.uint32)
    ew = rng.uniform(0.01, 0.5, 3000).astype(np.float32)
    p = dyg.WalkParams.make(threshold=10.0, walkers=64, max_steps=220, transition=transition, heuristic_walkers=2)
    dele = first
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, *(a[np.r_[first, -400:0]] for a in (gs, gd, gw)))
    if call == "delete":
        want = oracle.decremental(Go, Ho, gs[dele], gd[dele], p, batch_size=200)[:5]
    elif call == "insert":
        want = oracle.incremental(Ho, es, ed, ew, p, batch_size=1500, G=Go)[:3]
    elif call == "file_delete":
        want = oracle.stream_file(Go, Ho, 1, gs[dele], gd[dele], None, p, chunk=200)[:5]
    else:
        want = oracle.stream_file(Go, Ho, 0, es, ed, ew, p, chunk=1500)[:2]

    def go(G, H):
        if call == "delete":
            r = dyg.decremental_stream(G, H, gs[dele], gd[dele], p, batch_size=200)
        elif call == "insert":
            r = dyg.incremental_stream(H, es, ed, ew, p, 1500, G=G)
            return r.found_at, r.conductance, r.accepted
        elif call == "file_delete":
            r = dyg.stream_file(G, H, 1, gs[dele], gd[dele], None, p, chunk=200)
        else:
            r = dyg.stream_file(G, H, 0, es, ed, ew, p, chunk=1500)
            return r.status, r.conductance
        return r.status, r.conductance, r.rec_src, r.rec_dst, r.rec_kind

    def right(got, G, H):
        for a, b in zip(got, want):
            assert np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).astype(a.dtype).view(np.uint8))
        same_graph(G, Go)
        same_graph(H, Ho)

    for skip in list(range(0, 60, 1 if fail in (1, 2) else 3)):
        G, H = G0.clone(), H0.clone()
        try:
            with failing(dyg, skip, fail):
                got = go(G, H)
                assert dyg.lib().dyg_last_error_string() == b""
        except dyg.DygError as e:
            assert e.status == ENOMEM and fail > 1, (skip, str(e))
            G.copy_from(G0)
            H.copy_from(H0)
            got = go(G, H)
        right(got, G, H)
        G.close()
        H.close()


def test_large_scratch_is_kept_for_the_handles(dyg):  # noqa: F811
    """A row index of 0.6 GB stays with the device while it has handles, is lent
    to one after the other, and goes when the last is closed."""
    import gc
    import torch
    rng = np.random.default_rng(4)
    n, m = 1 << 20, 8_000_000
    s, d = rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)
    s[:400], d[:400] = 7, 100 + np.arange(400)
    w = np.ones(m, np.float32)
    p = dyg.WalkParams.make(threshold=10.0, walkers=32, max_steps=8, transition=1)

    def free():
        torch.cuda.synchronize()   # the pool gives back what is above its share then
        return torch.cuda.mem_get_info()[0]

    gc.collect()
    before = free()
    H = dyg.Graph.from_edges(n, s, d, w)
    H2 = H.clone()
    dyg.incremental_batch(H, s[:8], d[1:9], w[:8], p)
    held = free()
    for X in (H2, H, H2):
        dyg.incremental_batch(X, s[:8], d[1:9], w[:8], p)
        assert abs(free() - held) < 64 << 20
    H.close()
    H2.close()
    # the pool and the scratch keep 256 MB each
    assert before - free() < 560 << 20


def test_scratch_lent_to_threads(dyg, oracle):  # noqa: F811
    """Calls on four threads, each with handles and a stream of its own, borrow
    scratch side by side: every result is the oracle's."""
    import threading
    import torch
    rng = np.random.default_rng(6)
    n, first, gs, gd, gw = cycles(200, rng)
    hub = np.r_[first, -400:0]
    es = rng.integers(0, n, 800).astype(np.uint32)
    ed = ((es + 1 + rng.integers(0, n - 1, 800)) % n).astype(np.uint32)
    ew = rng.uniform(0.01, 0.5, 800).astype(np.float32)
    want = {}
    for tr in (0, 1):
        p = dyg.WalkParams.make(threshold=10.0, walkers=64, max_steps=220, transition=tr, heuristic_walkers=2)
        Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, gs[hub], gd[hub], gw[hub])
        fo, co, _, _ = oracle.incremental(Ho, es, ed, ew, p, batch_size=400, G=Go)
        st, cd, rx, ry, _, _ = oracle.decremental(Go, Ho, gs[first], gd[first], p, batch_size=100)
        want[tr] = (fo, co, st, cd, rx, ry)
    G0, H0 = dyg.Graph.from_edges(n, gs, gd, gw), dyg.Graph.from_edges(n, gs[hub], gd[hub], gw[hub])
    wrong = []

    def work(tr):
        try:
            p = dyg.WalkParams.make(threshold=10.0, walkers=64, max_steps=220, transition=tr, heuristic_walkers=2)
            s = torch.cuda.Stream()
            G, H = G0.clone(), H0.clone()
            for _ in range(8):
                G.copy_from(G0, stream=s.cuda_stream)
                H.copy_from(H0, stream=s.cuda_stream)
                a = dyg.incremental_stream(H, es, ed, ew, p, 400, G=G, stream=s.cuda_stream)
                b = dyg.decremental_stream(G, H, gs[first], gd[first], p, batch_size=100, stream=s.cuda_stream)
                got = (a.found_at, a.conductance, b.status, b.conductance, b.rec_src, b.rec_dst)
                for x, y in zip(got, want[tr]):
                    assert np.array_equal(np.asarray(x).view(np.uint8), np.asarray(y).astype(x.dtype).view(np.uint8))
            G.close()
            H.close()
        except BaseException as e:   # reported by the test's thread
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(k % 2,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
