"""The variant engine with and without bounds, at the edges of the rule that
applies them, against a plain Python search that keeps every non-dominated
label.  Weights are integers or multiples of 0.25, so all sums are exact in
FP32 and the comparison is equality."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ["csp", "hop", "maxcost", "qos"]
START = 21474836.0


def _random_graph(n, m, seed, quarter):
    rng = np.random.default_rng(seed)
    arcs = sorted({(int(u), int(x)) for u, x in rng.integers(0, n, (m, 2)) if u != x} |
                  {(i, i + 1) for i in range(n - 1)})
    row = np.zeros(n + 1, np.int64)
    for u, _ in arcs:
        row[u + 1] += 1
    w = rng.integers(0, 60, (len(arcs), 2)).astype(np.float32)
    w = w * 0.25 if quarter else w
    return np.cumsum(row), np.array([a[1] for a in arcs], np.int32), w[:, 0].copy(), w[:, 1].copy()


def _expand(kind, l, ln, dl):
    d, r0, r1, r2 = l
    if kind == "qos":
        return d + ln, min(r0, dl), 0.0, 0.0
    return (d + ln, r0 + dl, r1 + 1 if kind != "csp" else 0.0, max(r2, ln) if kind == "maxcost" else 0.0)


def _feasible(kind, l, L, H, M):
    if kind == "qos":
        return not l[1] < L
    return not (l[1] > L or (kind != "csp" and l[2] > H) or (kind == "maxcost" and l[3] > M))


def _search(csr, kind, s, t, L, H, M):
    """Best feasible (d, delay or bandwidth, hop, maxcost) at t, or None."""
    row, col, ln, dl = csr
    flip = -1.0 if kind == "qos" else 1.0

    def dominates(a, b):
        return a[0] <= b[0] and flip * a[1] <= flip * b[1] and a[2] <= b[2] and a[3] <= b[3]

    first = (0.0, START if kind == "qos" else 0.0, 0.0, 0.0)
    if not _feasible(kind, first, L, H, M):
        return None
    store, todo = {s: [first]}, [(s, first)]
    while todo:
        u, l = todo.pop()
        if l not in store[u] or u == t:
            continue
        for j in range(row[u], row[u + 1]):
            c = _expand(kind, l, float(ln[j]), float(dl[j]))
            x = int(col[j])
            if not _feasible(kind, c, L, H, M) or any(dominates(o, c) for o in store.get(x, [])):
                continue
            store[x] = [o for o in store.get(x, []) if not dominates(c, o)] + [c]
            todo.append((x, c))
    return min(store[t], key=lambda l: (l[0], flip * l[1], l[2], l[3])) if store.get(t) else None


@pytest.mark.parametrize("quarter", [False, True], ids=["integral", "quarters"])
@pytest.mark.parametrize("kind", KINDS)
def test_matches_plain_search(kind, quarter):
    import vine_b200 as v
    csr = _random_graph(36, 150, 3, quarter)
    g = v.Graph(*csr)
    rng = np.random.default_rng(8)
    unit = 0.25 if quarter else 1.0
    limits = [(0, 3, 20), (8, 4, 30), (60, 5, 45), (150, 7, 59), (400, 100, 10000),
              (2.0 ** 24, 2.0 ** 24, 2.0 ** 24), (math.inf, math.inf, math.inf), (-1, 5, 5), (59, 0, 59)]
    q = [(int(rng.integers(36)), int(rng.integers(36)), *l) for l in limits for _ in range(6)]
    q.append((4, 4, 50, 5, 50))
    src, dst = [x[0] for x in q], [x[1] for x in q]
    L, H, M = (np.array([x[k] for x in q], np.float32) for k in (2, 3, 4))
    L, M = L * np.float32(unit), M * np.float32(unit)
    r = v.solve_labels(g, kind, src, dst, L, H, M)
    for i in range(len(q)):
        want = _search(csr, kind, src[i], dst[i], float(L[i]), float(H[i]), float(M[i]))
        assert bool(r.found[i]) == (want is not None), (i, q[i])
        if want is not None:
            got = (float(r.cost[i]), float(r.delay[i]), *map(float, r.extra[i]))
            assert got == want, (i, q[i])
            assert r.path(i)[0] == src[i] and r.path(i)[-1] == dst[i]
    g.close()


def test_small_first_arena_is_retried():
    """Weights in quarters give no bounds, so the far corner of the grid takes
    more labels than a worker's first arena holds; the answers are those of a
    call that sets its arena."""
    import vine_b200 as v
    w = v.Workload.generate(1, rows=44, cols=44, n_pairs=1)
    g = v.Graph(w.row_ptr, w.col, w.len * np.float32(0.25), w.delay * np.float32(0.25))
    src, dst = [0, 0, 50], [44 * 44 - 1, 3, 44 * 43]
    lim = dict(hop_limit=[110, 110, 110], paths=True)
    a = v.solve_labels(g, "hop", src, dst, [1100, 1100, 1100], **lim)
    b = v.solve_labels(g, "hop", src, dst, [1100, 1100, 1100], config=v.Config(pool_labels=1 << 26), stats=True, **lim)
    assert b.stats[:, 2].max() > 1 << 17, "no query needs more than the first arena"
    assert a.found.tolist() == b.found.tolist() == [1, 1, 1]
    np.testing.assert_array_equal(a.cost, b.cost)
    np.testing.assert_array_equal(a.delay, b.delay)
    np.testing.assert_array_equal(a.extra, b.extra)
    for i in range(3):
        assert a.path(i)[0] == src[i] and a.path(i)[-1] == dst[i]
    g.close()


@pytest.mark.parametrize("far", [1, 2, 4097, 4099])
def test_any_far_capacity(far):
    """A worker's pile starts at a multiple of 16 bytes whatever its capacity;
    piles of a few entries give no bounds and no room, which is a status."""
    import vine_b200 as v
    g = v.Graph(*_random_graph(36, 150, 3, False))
    rng = np.random.default_rng(8)
    src, dst = rng.integers(0, 36, 40), rng.integers(0, 36, 40)
    limits = (np.full(40, 40, np.float32), np.full(40, 7, np.float32), np.full(40, 59, np.float32))
    for kind in KINDS:
        want = v.solve_labels(g, kind, src, dst, *limits)
        got = v.solve_labels(g, kind, src, dst, *limits, config=v.Config(far_capacity=far), raise_on_error=False)
        ok = got.status == 0
        assert set(got.status.tolist()) <= {0, v._lib.VINE_ERR_CAPACITY} and (ok.all() or far < 4)
        np.testing.assert_array_equal(got.found[ok], want.found[ok])
        np.testing.assert_array_equal(got.cost[ok], want.cost[ok])
        np.testing.assert_array_equal(got.delay[ok], want.delay[ok])
    g.close()


def test_bandwidth_paths_past_2_24():
    """Two ways of equal bandwidth: 2^24 + 2 in two arcs, and 2^24 + 3 whose FP32
    sum along the path is 2^24.  Costs are FP32 sums, so the second is the answer,
    as in a search without bounds (halved weights).  The ring of short arcs makes
    the bound pass's buckets narrow."""
    import vine_b200 as v
    arcs = [(0, 1, 0, 9), (0, 7, 8388608, 9), (1, 8, 0, 9), (2, 3, 8388608, 9), (3, 4, 1, 9), (4, 5, 1, 9),
            (5, 6, 1, 9), (7, 6, 8388610, 9), (8, 2, 8388608, 9)]
    arcs += [(9 + i, 9 + (i + 1) % 4000, 1, 9) for i in range(4000)]
    row = np.searchsorted([a[0] for a in arcs], np.arange(9 + 4000 + 1))
    col, ln, dl = (np.array([a[k] for a in arcs]) for k in (1, 2, 3))
    for scale in (0.5, 1.0):
        g = v.Graph(row, col, ln * scale, dl)
        r = v.solve_labels(g, "qos", [0, 0, 0], [6, 3, 6], [9, 9, 10])
        assert r.found.tolist() == [1, 1, 0]
        assert r.cost[:2].tolist() == [16777216 * scale] * 2 and r.delay[:2].tolist() == [9, 9]
        assert r.path(0).tolist() == [0, 1, 8, 2, 3, 4, 5, 6]
        g.close()
