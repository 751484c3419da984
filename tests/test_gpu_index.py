"""Weighted walks through rows on both sides of each line: what a lane reads at
once (8 slots), what it searches (32), what the warp does; with an index of the
rows in between and without (few and many walks on a graph with a hub row),
and weights where the fixed-point weights end (2^32 and more, under 2^-32)."""
import numpy as np
import pytest

from test_gpu_parity import dyg, run_incr_both, same_graph  # noqa: F401

pytestmark = pytest.mark.gpu


def rows_of(lengths, each, hub, rng):
    """`each` vertices of every length in `lengths`, joined to a pool of others; a
    hub row; a path through all vertices that are in none of these."""
    own = len(lengths) * each
    pool0, npool = own + 1, 4000
    s, d = [], []
    for i in range(own):
        s.append(np.full(lengths[i // each], i))
        d.append(pool0 + rng.choice(npool, lengths[i // each], replace=False))
    s.append(np.full(hub, own))
    d.append(pool0 + rng.choice(npool, hub, replace=False))
    s.append(np.arange(pool0, pool0 + npool - 1))
    d.append(np.arange(pool0 + 1, pool0 + npool))
    s, d = np.concatenate(s).astype(np.uint32), np.concatenate(d).astype(np.uint32)
    o = rng.permutation(len(s))
    return pool0 + npool, s[o], d[o]


@pytest.mark.parametrize("k", [1, 7, 600])
@pytest.mark.parametrize("hub", [0, 257, 1500])
@pytest.mark.parametrize("weights", ["plain", "huge", "tiny", "mixed"])
def test_weighted_rows(dyg, oracle, k, hub, weights):  # noqa: F811
    rng = np.random.default_rng(k + hub)
    n, s, d = rows_of([7, 8, 9, 31, 32, 33], 60, hub, rng)
    w = {"plain": rng.uniform(0.5, 2.0, len(s)),
         # 2^32 is the first weight that is cut off: sums of two wrap
         "huge": np.where(rng.random(len(s)) < 0.05, rng.choice([2.0**31, 2.0**32, 2.0**33, 1e20], len(s)), 1.0),
         # from 2^-32 on down a slot is never taken
         "tiny": rng.choice([2.0**-31, 2.0**-32, 2.0**-33, 1e-30], len(s)),
         "mixed": 2.0 ** rng.uniform(-40, 40, len(s))}[weights].astype(np.float32)
    es = rng.integers(0, 360, k).astype(np.uint32)
    ed = rng.integers(361, n, k).astype(np.uint32)
    ew = rng.uniform(0.01, 0.5, k).astype(np.float32)
    p = dyg.WalkParams.make(threshold=1e6, walkers=32, max_steps=40, transition=1)
    run_incr_both(dyg, oracle, n, s, d, w, es, ed, ew, p, batch_size=k)
    G, H = dyg.Graph.from_edges(n, s, d, w), dyg.Graph.from_edges(n, s, d, w)
    Go, Ho = oracle.OGraph(n, s, d, w), oracle.OGraph(n, s, d, w)
    dele = rng.choice(len(s), k, replace=False)
    r = dyg.decremental_batch(G, H, s[dele], d[dele], p)
    st, cd, rx, ry, rk, _ = oracle.decremental(Go, Ho, s[dele], d[dele], p, batch_size=k)
    assert np.array_equal(r.status, st)
    assert np.array_equal(r.conductance.view(np.uint32), cd.view(np.uint32))
    assert np.array_equal(r.rec_src, rx) and np.array_equal(r.rec_dst, ry) and np.array_equal(r.rec_kind, rk)
    same_graph(G, Go)
    same_graph(H, Ho)
