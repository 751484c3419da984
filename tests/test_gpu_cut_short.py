"""A grid barrier whose wait runs out: the call says so, no later launch of it
runs, and the graphs refuse updates until whole graphs are copied over them.
The wait is made to run out by arrivals on the barrier's counter that never
came; every block leaves at its limit."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import dyg, same_graph  # noqa: F401

pytestmark = pytest.mark.gpu
ESTATE = 5


def stall(dyg, g):  # noqa: F811
    f = dyg.lib().dyg_testing_stall_barrier
    f.argtypes, f.restype = [C.c_void_p, C.c_uint32], C.c_int
    assert f(g.handle, 8192) == 0


def hub_and_path(n, leaves, rng):
    s = np.concatenate([np.arange(n - 1), np.zeros(leaves, np.int64)]).astype(np.uint32)
    d = np.concatenate([np.arange(1, n), 2 + np.arange(leaves)]).astype(np.uint32)
    return s, d, rng.uniform(0.5, 2.0, len(s)).astype(np.float32)


@pytest.mark.parametrize("call", ["insert", "insert_weighted", "delete", "delete_weighted", "file_insert", "file_delete"])
@pytest.mark.parametrize("batches", [1, 3])
def test_barrier_that_runs_out(dyg, oracle, call, batches):  # noqa: F811
    rng = np.random.default_rng(7)
    # rows over 256 slots: weighted walks build their index, by a grid that
    # always meets at the barrier; 6,000 edges: commits of more than 16 blocks
    n, m = 12_000, 6_000
    gs, gd, gw = hub_and_path(n, 500, rng)
    es = np.concatenate([np.arange(m), np.zeros(200, np.int64)]).astype(np.uint32)
    ed = np.concatenate([np.arange(m) + 5000, 600 + np.arange(200)]).astype(np.uint32)
    ew = rng.uniform(0.5, 2.0, len(es)).astype(np.float32)
    G0, H0 = (dyg.Graph.from_edges(n, gs, gd, gw) for _ in range(2))
    G, H = G0.clone(), H0.clone()
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, gs, gd, gw)
    p = dyg.WalkParams.make(threshold=10.0, walkers=32, max_steps=8, transition=int("weighted" in call))
    dele = rng.permutation(len(gs))[:m]
    B = -(-m // batches)

    def go():
        if call.startswith("insert"):
            return dyg.incremental_stream(H, es, ed, ew, p, B, G=G)
        if call.startswith("delete"):
            return dyg.decremental_stream(G, H, gs[dele], gd[dele], p, batch_size=B)
        if call == "file_insert":
            return dyg.stream_file(G, H, 0, es, ed, ew, p)
        return dyg.stream_file(G, H, 1, gs[dele], gd[dele], None, p)

    stall(dyg, H if call.startswith("insert") else G)
    for _ in range(3):   # the call itself, and calls after it
        with pytest.raises(dyg.DygError) as e:
            go()
        assert e.value.status == ESTATE
    # the rows are still rows
    for g in (G, H):
        rp, col, w = g.export()
        assert np.all(col < n) and np.all(np.isfinite(w)) and np.all(w > 0)
    G.copy_from(G0)
    H.copy_from(H0)
    same_graph(G, Go)
    r = go()
    if call.startswith("insert"):
        fo, co, acc, _ = oracle.incremental(Ho, es, ed, ew, p, batch_size=B, G=Go)
        assert np.array_equal(r.found_at, fo) and np.array_equal(r.accepted, acc)
        got = r.conductance, co
    elif call.startswith("delete"):
        st, co, rx, ry, rk, _ = oracle.decremental(Go, Ho, gs[dele], gd[dele], p, batch_size=B)
        assert np.array_equal(r.status, st) and np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry)
        got = r.conductance, co
    else:
        op = int(call == "file_delete")
        a = (es, ed, ew) if not op else (gs[dele], gd[dele], None)
        st, co, *_ = oracle.stream_file(Go, Ho, op, *a, p)
        assert np.array_equal(r.status, st)
        got = r.conductance, co
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
    same_graph(G, Go)
    same_graph(H, Ho)


def test_split_calls_report_it(dyg):  # noqa: F811
    """Each call of a sharded batch says it too, and none walks through an
    index that was not finished."""
    import torch
    rng = np.random.default_rng(8)
    n, m = 12_000, 6_000
    gs, gd, gw = hub_and_path(n, 500, rng)
    G0 = dyg.Graph.from_edges(n, gs, gd, gw)
    G, H, L = G0.clone(), G0.clone(), dyg.lib()
    p = dyg.WalkParams.make(threshold=10.0, walkers=32, max_steps=8, transition=1)
    t = lambda a: torch.from_numpy(a.view(np.int32)).cuda()
    s, d, w = t(gs[:m].copy()), t(gd[:m].copy()), torch.ones(m, device="cuda")
    keys = torch.zeros(m, dtype=torch.int64, device="cuda")
    status, cond = torch.zeros(m, dtype=torch.int32, device="cuda"), torch.zeros(m, device="cuda")
    nw = C.c_uint32()
    nrec = C.c_uint64()
    q = lambda x: C.c_void_p(x.data_ptr())

    def restored(*stalled):
        G.copy_from(G0)
        H.copy_from(G0)
        for g in stalled:
            stall(dyg, g)

    walk = lambda: L.dyg_walk_keys(H.handle, q(s), q(d), q(w), None, 0, m, 0, m, 1, C.byref(p), q(keys), None)
    commit = lambda: L.dyg_incremental_commit_keys(H.handle, G.handle, q(s), q(d), q(w), m, q(keys), None, None, None, None)
    delete = lambda: L.dyg_decremental_delete(G.handle, H.handle, q(s), q(d), None, 0, m, q(status), q(cond),
                                              C.byref(nw), None)
    dwalk = lambda: L.dyg_decremental_walk_keys(G.handle, 0, nw.value, C.byref(p), q(keys), None)
    dcommit = lambda: L.dyg_decremental_commit_keys(G.handle, H.handle, C.byref(p), q(keys), nw.value, q(status), q(cond),
                                                    None, None, None, 0, C.byref(nrec), None)
    for call in (walk, commit):
        restored(H)
        assert call() == ESTATE and call() == ESTATE
        assert b"grid barrier" not in L.dyg_last_error_string()   # the second refusal is the graph's state
    restored(G)
    assert delete() == ESTATE and nw.value == 0
    for call in (dwalk, dcommit):
        restored()
        assert delete() == 0 and nw.value == m
        stall(dyg, G)
        assert call() == ESTATE and call() == ESTATE
    restored()
    assert [c() for c in (walk, commit)] == [0, 0]
    restored()
    assert [c() for c in (delete, dwalk, dcommit)] == [0, 0, 0]


@pytest.mark.parametrize("n", [10, 5000])
@pytest.mark.parametrize("call", ["export", "compact"])
def test_scan_that_runs_out(dyg, oracle, n, call):  # noqa: F811
    """Row offsets that were not all computed are not used: the call says so,
    and the next one works."""
    rng = np.random.default_rng(n)
    gs, gd, gw = hub_and_path(n, 3, rng)
    g, go = dyg.Graph.from_edges(n, gs, gd, gw), oracle.OGraph(n, gs, gd, gw)
    f = dyg.lib().dyg_testing_stall_scan
    f.argtypes, f.restype = [C.c_void_p], C.c_int
    for _ in range(2):
        assert f(g.handle) == 0
        with pytest.raises(dyg.DygError) as e:
            g.export() if call == "export" else g.compact()
        assert e.value.status == ESTATE
        same_graph(g, go)
        g.compact()
        same_graph(g, go)
