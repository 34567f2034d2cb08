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
