"""Row operations at the sizes where a row's work changes hands (one lane, a
warp, the block; chains followed or scanned for; deletion groups of a hub
row; lists over one block and over several), against the CPU oracle."""
import numpy as np
import pytest

from test_gpu_parity import dyg, run_incr_both, same_graph  # noqa: F401

pytestmark = pytest.mark.gpu


def star(n, leaves, rng):
    """A path over all vertices and `leaves` edges from vertex 0, shuffled."""
    s = np.concatenate([np.arange(n - 1), np.zeros(leaves, np.int64)]).astype(np.uint32)
    d = np.concatenate([np.arange(1, n), 2 + np.arange(leaves)]).astype(np.uint32)
    flip = rng.random(len(s)) < 0.5
    s, d = np.where(flip, d, s), np.where(flip, s, d)
    o = rng.permutation(len(s))
    return s[o], d[o], rng.uniform(0.5, 2.0, len(s)).astype(np.float32)


# entries one row gets in a batch: lane chains end at 4, warp chains at 32;
# spread = further edges, one per row, so that the list needs several blocks
@pytest.mark.parametrize("k,leaves,spread", [(1, 0, 0), (4, 40, 0), (5, 3, 0), (32, 300, 600), (33, 0, 0),
                                             (33, 30, 3000), (257, 300, 0), (900, 20, 5000)])
def test_append_chains(dyg, oracle, k, leaves, spread):  # noqa: F811
    rng = np.random.default_rng(k + leaves + spread)
    n = 1000 + 2 * spread
    hs, hd, hw = star(n, leaves, rng)
    e = np.concatenate([np.stack([np.zeros(k, np.int64), 2 + rng.integers(0, n - 2, k)], 1),
                        np.stack([1000 + np.arange(spread), 1000 + spread + np.arange(spread)], 1)])
    e = e[rng.permutation(len(e))]
    flip = rng.random(len(e)) < 0.5
    es = np.where(flip, e[:, 1], e[:, 0]).astype(np.uint32)
    ed = np.where(flip, e[:, 0], e[:, 1]).astype(np.uint32)
    ew = rng.uniform(0.5, 2.0, len(e)).astype(np.float32)
    p = dyg.WalkParams.make(threshold=3.0, walkers=32, max_steps=8)
    run_incr_both(dyg, oracle, n, hs, hd, hw, es, ed, ew, p, batch_size=len(e), with_g=(hs, hd, hw))


# deletions of one row: lane rows end at 32 slots, warps look at 4096 slots in
# all, hub rows take deletions in groups of 128 (repeats force single searches)
@pytest.mark.parametrize("k,leaves,repeat,spread", [(1, 28, 0, 0), (4, 40, 1, 0), (5, 20, 0, 0), (32, 127, 0, 0),
                                                    (32, 140, 2, 0), (33, 60, 0, 900), (128, 300, 0, 0),
                                                    (129, 300, 3, 0), (500, 9000, 0, 2000)])
def test_delete_chains(dyg, oracle, k, leaves, repeat, spread):  # noqa: F811
    rng = np.random.default_rng(k + leaves + spread)
    n = max(1000, leaves + 10) + 2 * spread
    gs, gd, gw = star(n, leaves, rng)
    hub = np.flatnonzero((gs == 0) | (gd == 0))
    dele = rng.choice(hub, min(k, len(hub)), replace=False)
    rest = rng.choice(np.setdiff1d(np.arange(len(gs)), hub), spread, replace=False)
    dele = rng.permutation(np.concatenate([dele, dele[:repeat], rest]))
    in_h = rng.random(len(gs)) < 0.7
    hs, hd, hw = gs[in_h], gd[in_h], gw[in_h]
    G, H = dyg.Graph.from_edges(n, gs, gd, gw), dyg.Graph.from_edges(n, hs, hd, hw)
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, hs, hd, hw)
    p = dyg.WalkParams.make(walkers=32, max_steps=12, heuristic_walkers=3)
    r = dyg.decremental_batch(G, H, gs[dele], gd[dele], p)
    st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, gs[dele], gd[dele], p, batch_size=len(dele))
    assert np.array_equal(r.status, st)
    assert np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
    assert np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry)
    assert np.array_equal(r.rec_kind, rk)
    same_graph(G, Go)
    same_graph(H, Ho)


def test_one_handle_for_both_graphs_is_refused(dyg):  # noqa: F811
    """The append keeps one set of chains per handle."""
    g = dyg.Graph.from_edges(4, np.array([0, 1], np.uint32), np.array([1, 2], np.uint32),
                             np.ones(2, np.float32))
    one = (np.array([0], np.uint32), np.array([3], np.uint32))
    p = dyg.WalkParams.make(walkers=32)
    for call in (lambda: dyg.incremental_batch(g, *one, np.ones(1, np.float32), p, G=g),
                 lambda: dyg.decremental_batch(g, g, *one, p),
                 lambda: dyg.stream_file(g, g, 1, *one, None, p)):
        with pytest.raises(dyg.DygError):
            call()


# weighted walks on graphs with hub rows: rows indexed by a warp (33..1024
# slots) and by a block, a tile of a block's prefix pass (4096 slots), and
# rows that must not be indexed (a repeated column, sums past 2^64)
@pytest.mark.parametrize("leaves,repeat,huge", [(256, 0, 0), (1021, 0, 0), (1022, 0, 0), (1023, 2, 0), (4094, 0, 0),
                                                (4095, 0, 0), (9000, 0, 0), (5000, 3, 0), (700, 0, 4), (5000, 0, 4)])
def test_weighted_hub_rows(dyg, oracle, leaves, repeat, huge):  # noqa: F811
    rng = np.random.default_rng(leaves + repeat + huge)
    n = leaves + 40
    hs, hd, hw = star(n, leaves, rng)
    # a second row between the lane's and the block's lengths
    far = 20 + rng.choice(n - 30, 33, replace=False)
    far = far[far != 10]
    more = rng.choice(np.flatnonzero((hs == 0) | (hd == 0)), repeat, replace=False)
    hs = np.concatenate([hs, np.full(len(far), 10, np.uint32), hs[more]]).astype(np.uint32)
    hd = np.concatenate([hd, far, hd[more]]).astype(np.uint32)
    hw = np.concatenate([hw, rng.uniform(0.5, 2.0, len(far) + repeat)]).astype(np.float32)
    hw[rng.choice(np.flatnonzero((hs == 0) | (hd == 0)), huge, replace=False)] = 3e9
    es = rng.integers(0, n, 24).astype(np.uint32)
    ed = ((es + 1 + rng.integers(0, n - 1, 24)) % n).astype(np.uint32)
    ew = rng.uniform(0.01, 0.05, 24).astype(np.float32)
    p = dyg.WalkParams.make(threshold=100.0, walkers=64, max_steps=30, transition=1)
    run_incr_both(dyg, oracle, n, hs, hd, hw, es, ed, ew, p, batch_size=12)
    G, H = dyg.Graph.from_edges(n, hs, hd, hw), dyg.Graph.from_edges(n, hs, hd, hw)
    Go, Ho = oracle.OGraph(n, hs, hd, hw), oracle.OGraph(n, hs, hd, hw)
    dele = rng.choice(len(hs), 40, replace=False)
    r = dyg.decremental_batch(G, H, hs[dele], hd[dele], p)
    st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, hs[dele], hd[dele], p, batch_size=40)
    assert np.array_equal(r.status, st)
    assert np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
    assert np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry)
    same_graph(G, Go)
    same_graph(H, Ho)


@pytest.mark.parametrize("k", [1, 3, 40])
@pytest.mark.parametrize("room", [10_000, 100])
def test_records_beyond_those_fetched_ahead(dyg, oracle, k, room):  # noqa: F811
    """k deletions that recover 89 edges each, into host buffers with and
    without room for them."""
    L = 90
    base = np.repeat(np.arange(k) * L, L)
    i = np.tile(np.arange(L), k)
    gs, gd = (base + i).astype(np.uint32), (base + (i + 1) % L).astype(np.uint32)
    gw = np.linspace(0.5, 2.0, k * L).astype(np.float32)
    first = np.arange(k) * L
    G = dyg.Graph.from_edges(k * L, gs, gd, gw)
    H = dyg.Graph.from_edges(k * L, gs[first], gd[first], gw[first])
    Go, Ho = oracle.OGraph(k * L, gs, gd, gw), oracle.OGraph(k * L, gs[first], gd[first], gw[first])
    p = dyg.WalkParams.make(walkers=32)
    st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, gs[first], gd[first], p, batch_size=k)
    assert len(rx) == 89 * k
    out = (np.empty(k, np.int32), np.empty(k, np.float32), np.zeros(room, np.uint32), np.zeros(room, np.uint32),
           np.zeros(room, np.uint8))
    if len(rx) > room:
        with pytest.raises(dyg.DygError):
            dyg.decremental_stream_into(G, H, gs[first], gd[first], p, *out, room, batch_size=k)
    else:
        assert dyg.decremental_stream_into(G, H, gs[first], gd[first], p, *out, room, batch_size=k) == len(rx)
    m = min(room, len(rx))
    assert np.array_equal(out[0], st) and np.array_equal(out[1].view(np.uint32), cd.view(np.uint32))
    assert np.array_equal(out[2][:m], rx[:m]) and np.array_equal(out[3][:m], ry[:m]) and np.array_equal(out[4][:m], rk[:m])
    same_graph(G, Go)
    same_graph(H, Ho)


# the walk's remainder changes from the table to the general division at 256
@pytest.mark.parametrize("leaves", [1, 2, 253, 254, 255, 256, 257, 2000])
@pytest.mark.parametrize("steps", [1, 2, 4, 5, 40])
def test_uniform_degrees_and_lengths(dyg, oracle, leaves, steps):  # noqa: F811
    rng = np.random.default_rng(leaves + steps)
    n = leaves + 30
    hs, hd, hw = star(n, leaves, rng)
    es = np.concatenate([np.zeros(8, np.int64), rng.integers(1, n, 24)]).astype(np.uint32)
    ed = ((es + 1 + rng.integers(0, n - 1, 32)) % n).astype(np.uint32)
    ew = rng.uniform(0.01, 0.05, 32).astype(np.float32)
    p = dyg.WalkParams.make(threshold=10.0, walkers=96, max_steps=steps)
    run_incr_both(dyg, oracle, n, hs, hd, hw, es, ed, ew, p, batch_size=20)


# rows built by a lane (8), a warp (256), in one shared-memory tile of a block
# (4096) and in several; every row in edge-list order, as a stable sort gives it
@pytest.mark.parametrize("leaves", [0, 7, 8, 31, 32, 33, 255, 256, 257, 4095, 4096, 9000])
def test_build_and_export_rows(dyg, leaves):  # noqa: F811
    rng = np.random.default_rng(leaves)
    n = leaves + 50
    s, d, w = star(n, leaves, rng)
    # repeated edges, self-loops and an isolated last vertex
    s = np.concatenate([s, s[:9], [3, 3]]).astype(np.uint32)
    d = np.concatenate([d, d[:9], [3, 3]]).astype(np.uint32)
    w = np.concatenate([w, w[:9] + 1, [5, 6]]).astype(np.float32)
    g = dyg.Graph.from_edges(n + 1, s, d, w)
    rows, cols = np.stack([s, d], 1).ravel(), np.stack([d, s], 1).ravel()
    order = np.argsort(rows, kind="stable")
    rp, col, ww = g.export()
    assert np.array_equal(rp, np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n + 1))]).astype(np.uint64))
    assert np.array_equal(col, cols[order]) and np.array_equal(ww, np.repeat(w, 2)[order])
    inf = g.info()
    assert inf["n_slots"] == 2 * len(s) and inf["arena_used"] == 2 * len(s) + 2 * (n + 1)


def test_build_long_list_is_checked(dyg):  # noqa: F811
    """Lists over 65,536 edges are checked on the device."""
    m = 70_000
    s, d = np.arange(m, dtype=np.uint32), np.arange(1, m + 1, dtype=np.uint32)
    w = np.ones(m, np.float32)
    bad_w, bad_d = w.copy(), d.copy()
    bad_w[69_000], bad_d[66_000] = np.inf, m + 1
    for args in ((s, bad_d, w), (s, d, bad_w)):
        with pytest.raises(dyg.DygError) as e:
            dyg.Graph.from_edges(m + 1, *args)
        assert e.value.status == dyg.DYG_EINVAL
    assert dyg.Graph.from_edges(m + 1, s, d, w).info()["n_slots"] == 2 * m


def test_export_short_buffer(dyg):  # noqa: F811
    s, d, w = star(400, 300, np.random.default_rng(1))
    g = dyg.Graph.from_edges(400, s, d, w)
    rp0, col0, w0 = g.export()
    rp, col, ww = np.zeros(401, np.uint64), np.zeros(50, np.uint32), np.zeros(50, np.float32)
    assert dyg.lib().dyg_graph_export(g.handle, rp.ctypes.data, col.ctypes.data, ww.ctypes.data, 50) == 4
    assert np.array_equal(rp, rp0) and np.array_equal(col, col0[:50]) and np.array_equal(ww, w0[:50])


@pytest.mark.parametrize("transition", [0, 1])
@pytest.mark.parametrize("steps", [3, 5, 100, 256, 257])
def test_winner_paths_recorded_and_replayed(dyg, oracle, transition, steps):  # noqa: F811
    """Winners of one to 200 moves, with walks that keep their paths (up to 256
    steps) and walks whose winners are replayed; the long ones ask for more
    room than a call starts with, so their walks are repeated."""
    k, rng = 1000, np.random.default_rng(steps)
    # cycles of 3..200 vertices with a few chords
    sizes = np.where(np.arange(k) % 4 == 0, 200, rng.integers(3, 40, k))
    off = np.concatenate([[0], np.cumsum(sizes)])
    base, L = np.repeat(off[:-1], sizes), np.repeat(sizes, sizes)
    i = np.arange(off[-1]) - base
    gs, gd = (base + i).astype(np.uint32), (base + (i + 1) % L).astype(np.uint32)
    ch = np.flatnonzero(rng.random(len(gs)) < 0.02)
    gs = np.concatenate([gs, gs[ch]])
    gd = np.concatenate([gd, (base + (i + L // 2) % L)[ch]]).astype(np.uint32)
    ok = gs != gd
    gs, gd = gs[ok], gd[ok]
    gw = rng.uniform(0.5, 2.0, len(gs)).astype(np.float32)
    n, dele = int(off[-1]), off[:-1]
    G, H = dyg.Graph.from_edges(n, gs, gd, gw), dyg.Graph.from_edges(n, gs[dele], gd[dele], gw[dele])
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, gs[dele], gd[dele], gw[dele])
    p = dyg.WalkParams.make(walkers=64, max_steps=steps, transition=transition, heuristic_walkers=2)
    r = dyg.decremental_stream(G, H, gs[dele], gd[dele], p, batch_size=400)
    st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, gs[dele], gd[dele], p, batch_size=400)
    assert np.array_equal(r.status, st) and np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
    assert np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry) and np.array_equal(r.rec_kind, rk)
    same_graph(G, Go)
    same_graph(H, Ho)


# occurrences of one edge in a stream file: a single one, chains a lane folds
# (up to 32) and ones the block scans the file for, for edges that are new, in
# G only, and in both graphs
@pytest.mark.parametrize("times", [1, 2, 31, 32, 33, 700])
@pytest.mark.parametrize("more", [0, 300, 9000])
def test_stream_repeats(dyg, oracle, times, more):  # noqa: F811
    rng = np.random.default_rng(times + more)
    n = 500
    gs, gd, gw = star(n, 60, rng)
    in_h = rng.random(len(gs)) < 0.6
    hs, hd, hw = gs[in_h], gd[in_h], gw[in_h]
    only_g = np.flatnonzero(~in_h)[0]
    pick = [(gs[only_g], gd[only_g]), (hs[0], hd[0]), (5, 490), (7, 300)]
    e = np.array(pick * times + [tuple(rng.integers(0, n, 2)) for _ in range(more)], np.uint32)
    flip = rng.random(len(e)) < 0.5
    e[flip] = e[flip][:, ::-1]
    e = e[rng.permutation(len(e))]
    w = rng.uniform(0.1, 1.0, len(e)).astype(np.float32)
    G, H = dyg.Graph.from_edges(n, gs, gd, gw), dyg.Graph.from_edges(n, hs, hd, hw)
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, hs, hd, hw)
    p = dyg.WalkParams.make(threshold=5.0, walkers=32, max_steps=20)
    for k in range(2):   # the second file finds the table as the first left it
        r = dyg.stream_file(G, H, 0, e[:, 0].copy(), e[:, 1].copy(), w, p, first_update_id=k * len(e))
        st, cd, *_ = oracle.stream_file(Go, Ho, 0, e[:, 0].copy(), e[:, 1].copy(), w, p, first_uid=k * len(e))
        assert np.array_equal(r.status, st)
        assert np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
        same_graph(G, Go)
        same_graph(H, Ho)


def test_fresh_handles_on_a_stream_of_the_caller(dyg, oracle):  # noqa: F811
    """The first calls of new handles on a stream that the default stream does
    not wait for: workspaces are cleared on the stream that uses them."""
    import torch
    import dygrass_b200.workloads as wl
    W = wl.mesh_3d(12, inserts=400)
    Go, Ho = oracle.OGraph(W.n, W.g_src, W.g_dst, W.g_w), oracle.OGraph(W.n, W.h_src, W.h_dst, W.h_w)
    oracle.incremental(Ho, W.ins_src, W.ins_dst, W.ins_w, W.params, G=Go)
    st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, W.del_src, W.del_dst, W.dparams)
    for _ in range(4):
        s = torch.cuda.Stream()
        G, H = dyg.Graph.from_edges(W.n, W.g_src, W.g_dst, W.g_w), dyg.Graph.from_edges(W.n, W.h_src, W.h_dst, W.h_w)
        dyg.incremental_stream(H, W.ins_src, W.ins_dst, W.ins_w, W.params, G=G, stream=s.cuda_stream)
        r = dyg.decremental_stream(G, H, W.del_src, W.del_dst, W.dparams, stream=s.cuda_stream)
        assert np.array_equal(r.status, st) and np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry)
        same_graph(G, Go)
        same_graph(H, Ho)
        G.close()
        H.close()
