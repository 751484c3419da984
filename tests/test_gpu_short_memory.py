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
