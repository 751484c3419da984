"""Many rows with many entries each in one batch: chains that are followed (32),
runs put in order by a warp (256) and by a block (4,096), rows a block scans the
list for (longer ones, and lists of up to 8,192 edges), against the CPU oracle."""
import numpy as np
import pytest

from test_gpu_parity import dyg, run_incr_both, same_graph  # noqa: F401

pytestmark = pytest.mark.gpu


def entries(rows, each, others, rng):
    """`each` edges from each of `rows` vertices to a pool, and `others` edges
    inside the pool; in random order and orientation.  Vertices: the rows, the
    pool."""
    pool = max(2 * each, 3000)
    s = np.concatenate([np.repeat(np.arange(rows), each), rows + rng.integers(0, pool, others)])
    d = np.concatenate([rows + np.concatenate([rng.permutation(pool)[:each] for _ in range(rows)]),
                        rows + rng.integers(0, pool, others)])
    flip = rng.random(len(s)) < 0.5
    s, d = np.where(flip, d, s), np.where(flip, s, d)
    o = rng.permutation(len(s))
    return rows + pool, s[o].astype(np.uint32), d[o].astype(np.uint32)


SHAPES = [(2, 32, 0), (2, 33, 0), (60, 33, 0), (60, 33, 9000), (400, 40, 0), (30, 255, 3000), (30, 256, 3000),
          (30, 257, 0), (30, 257, 3000), (40, 300, 0), (3, 4095, 0), (3, 4096, 0), (3, 4097, 0), (1, 9000, 500),
          (500, 9, 9000)]


@pytest.mark.parametrize("rows,each,others", SHAPES)
@pytest.mark.parametrize("deg", [0, 300])   # rows of up to 256 slots are moved by a warp
def test_append(dyg, oracle, rows, each, others, deg):  # noqa: F811
    rng = np.random.default_rng(rows * each + others + deg)
    n, es, ed = entries(rows, each, others, rng)
    base = np.arange(n - 1)
    hub = rng.integers(0, n, (min(rows, 40), deg)) if deg else np.empty((0, 0), np.int64)
    hs = np.concatenate([base, np.repeat(np.arange(len(hub)), deg)]).astype(np.uint32)
    hd = np.concatenate([base + 1, hub.ravel()]).astype(np.uint32)
    hw = rng.uniform(0.5, 2.0, len(hs)).astype(np.float32)
    ew = rng.uniform(0.5, 2.0, len(es)).astype(np.float32)
    p = dyg.WalkParams.make(threshold=3.0, walkers=32, max_steps=4)
    run_incr_both(dyg, oracle, n, hs, hd, hw, es, ed, ew, p, batch_size=len(es), with_g=(hs, hd, hw))


@pytest.mark.parametrize("rows,each,others", SHAPES)
@pytest.mark.parametrize("more", [0, 500])   # slots of the rows that stay
def test_delete(dyg, oracle, rows, each, others, more):  # noqa: F811
    rng = np.random.default_rng(rows * each + others + more)
    n, s, d = entries(rows, each, others, rng)
    stay = np.stack([np.repeat(np.arange(min(rows, 40)), more), rng.integers(0, n, min(rows, 40) * more)], 1)
    gs, gd = np.concatenate([s, stay[:, 0]]).astype(np.uint32), np.concatenate([d, stay[:, 1]]).astype(np.uint32)
    o = rng.permutation(len(gs))
    gs, gd = gs[o], gd[o]
    gw = rng.uniform(0.5, 2.0, len(gs)).astype(np.float32)
    in_h = rng.random(len(gs)) < 0.7
    hs, hd, hw = gs[in_h], gd[in_h], gw[in_h]
    # some edges twice, some that are not there
    ds = np.concatenate([s, s[:5], rng.integers(0, n, 5).astype(np.uint32)])
    dd = np.concatenate([d, d[:5], rng.integers(0, n, 5).astype(np.uint32)])
    o = rng.permutation(len(ds))
    ds, dd = ds[o], dd[o]
    G, H = dyg.Graph.from_edges(n, gs, gd, gw), dyg.Graph.from_edges(n, hs, hd, hw)
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, hs, hd, hw)
    p = dyg.WalkParams.make(walkers=32, max_steps=4, heuristic_walkers=1)
    for k in range(2):   # the second time everything is gone
        r = dyg.decremental_batch(G, H, ds, dd, p, first_update_id=k * len(ds))
        st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, ds, dd, p, first_uid=k * len(ds), single_batch=True)
        assert np.array_equal(r.status, st)
        assert np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
        assert np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry) and np.array_equal(r.rec_kind, rk)
        same_graph(G, Go)
        same_graph(H, Ho)


@pytest.mark.parametrize("keys,times,others", [(4, 32, 100), (4, 33, 100), (300, 40, 0), (300, 40, 9000), (60, 255, 0),
                                               (60, 256, 0), (60, 257, 0), (6, 4095, 0), (6, 4096, 0), (6, 4097, 0),
                                               (2, 9000, 3000)])
@pytest.mark.parametrize("tight", [False, True])
def test_file_repeats(dyg, oracle, keys, times, others, tight):  # noqa: F811
    """Edges repeated many times in a stream file: new ones, ones in G, ones in
    both graphs; `tight`: the new edges make G's arena grow, after the weights
    were added."""
    rng = np.random.default_rng(keys * times + others)
    n = 4000
    gs, gd = np.arange(n - 1, dtype=np.uint32), np.arange(1, n, dtype=np.uint32)
    gw = rng.uniform(0.5, 2.0, n - 1).astype(np.float32)
    in_h = rng.random(n - 1) < 0.5
    known = rng.choice(n - 1, keys, replace=False)
    pick = [(gs[k], gd[k]) if i % 3 else (rng.integers(0, n // 2), n // 2 + rng.integers(0, n // 2))
            for i, k in enumerate(known)]
    e = np.concatenate([np.repeat(np.array(pick, np.int64).reshape(-1, 2), times, 0), rng.integers(0, n, (others, 2))])
    flip = rng.random(len(e)) < 0.5
    e[flip] = e[flip][:, ::-1]
    e = e[rng.permutation(len(e))].astype(np.uint32)
    w = rng.uniform(0.1, 1.0, len(e)).astype(np.float32)
    kw = dict(slack_per_row=0, arena_headroom=0.0) if tight else {}
    G = dyg.Graph.from_edges(n, gs, gd, gw, **kw)
    H = dyg.Graph.from_edges(n, gs[in_h], gd[in_h], gw[in_h], **kw)
    Go, Ho = oracle.OGraph(n, gs, gd, gw), oracle.OGraph(n, gs[in_h], gd[in_h], gw[in_h])
    p = dyg.WalkParams.make(threshold=5.0, walkers=32, max_steps=10)
    for k in range(2):   # the second file finds the table as the first left it
        r = dyg.stream_file(G, H, 0, e[:, 0].copy(), e[:, 1].copy(), w, p, first_update_id=k * len(e))
        st, cd, *_ = oracle.stream_file(Go, Ho, 0, e[:, 0].copy(), e[:, 1].copy(), w, p, first_uid=k * len(e))
        assert np.array_equal(r.status, st)
        assert np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
        same_graph(G, Go)
        same_graph(H, Ho)
