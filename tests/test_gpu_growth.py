"""A handle's workspace grows between calls: the corridor arrays of a
264,000-vertex road graph are made, or made again for more workers, by a call
whose other buffers suffice.  They are cleared on the call's own stream, which
does not wait for the default one.  Expected costs and delays are those of the
256-query fixture (integers: equality)."""
import numpy as np
import pytest

from golden_util import load_scale

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def road():
    return load_scale("c5_sample256")


def _check(fx, res, times):
    assert not res.status.any()
    want = [np.tile(np.array([q[k] for q in fx["queries"]]), times) for k in ("found", "cost", "delay")]
    np.testing.assert_array_equal(res.found.astype(bool), want[0])
    np.testing.assert_array_equal(res.cost, want[1].astype(np.float32))
    np.testing.assert_array_equal(res.delay, want[2].astype(np.float32))


@pytest.mark.parametrize("first", ["fewer", "no_bounds"])
def test_corridor_arrays_made_by_a_later_call(road, first):
    import vine_b200 as v
    fx = road
    g = v.Graph(fx["row_ptr"], fx["col"], fx["len"], fx["delay"])
    cfg = v.Config(use_bounds=1, policy="ar")
    if first == "fewer":  # one worker an SM, then two
        _check(fx, v.solve(g, *(np.tile(fx[k], 2) for k in ("src", "dst", "budget")), cfg), 2)
    else:
        res = v.solve(g, fx["src"], fx["src"], fx["budget"], v.Config())
        assert res.found.all() and not res.cost.any()
    _check(fx, v.solve(g, *(np.tile(fx[k], 4) for k in ("src", "dst", "budget")), cfg), 4)
    g.close()


def test_arrays_for_as_many_workers_as_queries(road):
    """Arrays are made for the queries of a call (16 workers at least, at most one an SM)
    and grow with them; smaller calls use what is there."""
    import vine_b200 as v
    fx = road
    g = v.Graph(fx["row_ptr"], fx["col"], fx["len"], fx["delay"])
    for n in (1, 16, 17, 3, 129, 256, 40):
        res = v.solve(g, fx["src"][:n], fx["dst"][:n], fx["budget"][:n], v.Config(use_bounds=1, policy="ar"))
        assert not res.status.any()
        for q, e in enumerate(fx["queries"][:n]):
            assert (float(res.cost[q]), float(res.delay[q])) == (e["cost"], e["delay"])
            assert res.path(q)[0] == e["src"] and res.path(q)[-1] == e["dst"]
    g.close()


def test_many_small_calls():
    """The copies of a handle's later calls go through a pinned block."""
    import vine_b200 as v
    w = v.Workload.generate(1, rows=12, cols=12, n_pairs=130)
    g = v.Graph(w.row_ptr, w.col, w.len, w.delay)
    cfg = v.Config(use_bounds=1, pool_labels=1 << 22)
    want = v.solve(g, w.src, w.dst, w.budget, cfg)
    for q in range(w.nq):
        n = 1 + q % 3
        res = v.solve(g, w.src[q:q + n], w.dst[q:q + n], w.budget[q:q + n], cfg)
        for i in range(len(res.cost)):
            assert res.found[i] == want.found[q + i] and res.cost[i] == want.cost[q + i]
            assert res.delay[i] == want.delay[q + i]
            assert not want.found[q + i] or len(res.path(i)) >= 1 and res.path(i)[-1] == w.dst[q + i]
    g.close()
