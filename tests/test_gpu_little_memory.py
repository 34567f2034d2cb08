"""Calls on a device that has little memory left: what the engine can do
without, it does without.  The rest of the device is held by one block, of
which the test leaves a stated number of bytes."""
import numpy as np
import pytest

from golden_util import load_scale

pytestmark = pytest.mark.gpu


@pytest.fixture
def leave():
    import torch
    held = []

    def fill(keep):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        held.append(torch.empty(max(1, free - keep), dtype=torch.uint8, device="cuda"))

    yield fill
    held.clear()
    torch.cuda.empty_cache()


@pytest.mark.parametrize("grown", [False, True])
def test_no_room_for_corridors(leave, grown):
    """2 GB hold neither the corridor arrays of a 264,000-vertex graph (6 GB)
    nor, where they exist, those of more workers: the call is answered without
    them, and so is the next one; with the memory back, it is answered too."""
    import torch
    import vine_b200 as v
    fx = load_scale("c5_sample256")
    want = [np.array([q[k] for q in fx["queries"]]) for k in ("found", "cost", "delay")]
    g = v.Graph(fx["row_ptr"], fx["col"], fx["len"], fx["delay"])
    small = dict(pool_labels=1 << 27, far_capacity=1 << 15)
    few = np.argsort(fx["budget"])[:48]
    cfg = v.Config(use_bounds=1, policy="ar", **small)

    def check(sel, times=1):
        pick = np.tile(sel, times)
        res = v.solve(g, fx["src"][pick], fx["dst"][pick], fx["budget"][pick], cfg)
        assert not res.status.any()
        np.testing.assert_array_equal(res.found.astype(bool), want[0][pick])
        np.testing.assert_array_equal(res.cost, want[1][pick].astype(np.float32))
        np.testing.assert_array_equal(res.delay, want[2][pick].astype(np.float32))

    if grown:
        check(few)
    else:  # makes everything but the corridor arrays
        assert v.solve(g, fx["src"], fx["src"], fx["budget"], v.Config(**small)).found.all()
    leave(2 << 30)
    for _ in range(2):
        check(few, 21)  # 1,008 queries: two workers an SM, where there is room
    torch.cuda.empty_cache()
    g.close()


@pytest.mark.parametrize("keep_mb", [1700, 2600])
def test_little_room_for_label_variants(leave, keep_mb):
    """Too little for the first arena of every worker: an arena of what is free."""
    import vine_b200 as v
    w = v.Workload.generate(1, rows=20, cols=20, n_pairs=200)
    g = v.Graph(w.row_ptr, w.col, w.len, w.delay)
    rng = np.random.default_rng(2)
    src, dst = rng.integers(0, 400, 200), rng.integers(0, 400, 200)
    limits = np.full(200, 300, np.float32), np.full(200, 30, np.float32)
    h = v.Graph(w.row_ptr, w.col, w.len, w.delay)
    want = v.solve_labels(h, "hop", src, dst, *limits)
    h.close()
    leave(keep_mb << 20)
    for _ in range(2):
        got = v.solve_labels(g, "hop", src, dst, *limits)
        np.testing.assert_array_equal(got.found, want.found)
        np.testing.assert_array_equal(got.cost, want.cost)
        np.testing.assert_array_equal(got.delay, want.delay)
    g.close()
