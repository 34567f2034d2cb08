"""Corridors: the two-sided search that cuts a query's graph down before the
label search, at the sizes where it can go wrong.

Every case compares cost, delay and feasibility with the CPU oracle's label
setting under exact Dijkstra bounds (cost and delay are integers: equality).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n, arcs):
    arcs = sorted(arcs)
    row = np.zeros(n + 1, np.int64)
    for a in arcs:
        row[a[0] + 1] += 1
    return (np.cumsum(row), np.array([a[1] for a in arcs], np.int32),
            np.array([a[2] for a in arcs], np.float32), np.array([a[3] for a in arcs], np.float32))


def _line(n, rng):
    """A path graph with a fast and a slow arc a step (both directions)."""
    out = []
    for i in range(n - 1):
        for u, x in ((i, i + 1), (i + 1, i)):
            out.append((u, x, int(rng.integers(1, 50)), int(rng.integers(50, 100))))
            out.append((u, x, int(rng.integers(50, 100)), int(rng.integers(1, 50))))
    return n, out


def _star(spokes, rng):
    """Source -> spokes -> sink and a few chords: two hubs of `spokes` arcs."""
    n, out = spokes + 2, []
    for i in range(spokes):
        out.append((0, 2 + i, int(rng.integers(1, 1000)), int(rng.integers(1, 1000))))
        out.append((2 + i, 1, int(rng.integers(1, 1000)), int(rng.integers(1, 1000))))
        if i % 7 == 0:
            out.append((2 + i, 2 + int(rng.integers(spokes)), int(rng.integers(0, 9)), int(rng.integers(0, 9))))
    return n, out


def _layers(width, depth, rng, w=100):
    """`depth` layers of `width` vertices, three arcs each to the next layer."""
    n, out = width * depth, []
    for d in range(depth - 1):
        for i in range(width):
            for _ in range(3):
                out.append((d * width + i, (d + 1) * width + int(rng.integers(width)),
                            int(rng.integers(0, w + 1)), int(rng.integers(0, w + 1))))
    return n, out


CASES = {
    # name: (maker, source, sink)
    "line2": (lambda r: _line(2, r), 0, 1),
    "line33": (lambda r: _line(33, r), 0, 32),
    "line700": (lambda r: _line(700, r), 3, 690),
    "star31": (lambda r: _star(31, r), 0, 1),       # one warp
    "star257": (lambda r: _star(257, r), 0, 1),     # hubs, shared by the block
    "star5000": (lambda r: _star(5000, r), 0, 1),   # queue past its shared part
    "layers": (lambda r: _layers(40, 30, r), 5, 29 * 40 + 7),
    "layers_wide": (lambda r: _layers(3000, 10, r), 5, 9 * 3000 + 9),  # shrinks in steps
    "heavy_arcs": (lambda r: _layers(30, 20, r, w=400000), 1, 19 * 30 + 2),
}


def _check(v, O, g, og, s, t, budgets, cfg):
    h_len, h_del = O.lower_bounds(og, t)
    src, dst = np.full(len(budgets), s, np.int32), np.full(len(budgets), t, np.int32)
    res = v.solve(g, src, dst, np.asarray(budgets, np.float32), cfg)
    for q, b in enumerate(budgets):
        want = O.solve_label_setting(og, s, t, float(b), h_len, h_del, use_incumbent=True)
        assert bool(res.found[q]) == want["found"], (q, b)
        if not want["found"]:
            continue
        assert (float(res.cost[q]), float(res.delay[q])) == (want["cost"], want["delay"]), (q, b)
        p = res.path(q)
        assert p[0] == s and p[-1] == t
        low_cost = low_delay = 0.0  # parallel arcs: the path's sums lie at or above these
        for u, x in zip(p[:-1], p[1:]):
            heads, ln, dl = g.out_edges(int(u))
            assert (heads == x).any()
            low_cost += float(ln[heads == x].min())
            low_delay += float(dl[heads == x].min())
        assert low_cost <= want["cost"] and low_delay <= want["delay"] <= b


@pytest.mark.parametrize("threads,table", [(512, 13), (128, 11), (64, 6)])
@pytest.mark.parametrize("name", list(CASES))
def test_matches_oracle(name, threads, table):
    import vine_b200 as v
    from oracle import oracle as O
    make, s, t = CASES[name]
    n, arcs = make(np.random.default_rng(17))
    csr = _graph(n, arcs)
    g, og = v.Graph(*csr), O.CsrGraph(*csr)
    lo = O.dijkstra(og, s, "delay")[0][t]
    hi = O.dijkstra(og, s, "len")[1][t]
    if not np.isfinite(lo):
        lo, hi = 50.0, 100.0
    budgets = [lo - 1, lo, lo + 0.5, lo + 0.1 * (hi - lo), lo + 0.5 * (hi - lo), hi, 2 * hi + 10,
               2.0 ** 24, np.inf]  # the last two: the whole-graph bounds
    cfg = v.Config(use_bounds=1, policy="ar", block_threads=threads, table_log2=table,
                   pool_labels=1 << 24)
    _check(v, O, g, og, s, t, budgets, cfg)
    _check(v, O, g, og, s, t, budgets, v.Config(use_bounds=1, sync_rounds=1, pool_labels=1 << 24))
    g.close()


def test_corridor_past_its_capacity():
    """70,000 equal two-arc ways: more vertices than a local graph holds, so
    the query is answered with the bounds over the whole graph."""
    import vine_b200 as v
    k = 70000
    n, arcs = k + 2, []
    for i in range(k):
        arcs += [(0, 2 + i, 5, 7), (2 + i, 1, 6, 8)]
    g = v.Graph(*_graph(n, arcs))
    res = v.solve(g, [0, 0], [1, 1], [15, 14], v.Config(use_bounds=1, pool_labels=1 << 24))
    assert res.found.tolist() == [1, 0]
    assert (res.cost[0], res.delay[0]) == (11, 15)
    g.close()


def test_costs_past_2_24():
    """A path cost of 2^24 or more goes to the whole-graph bounds; the same
    graph's cheaper sink does not."""
    import vine_b200 as v
    arcs = [(0, 1, 16000000, 3), (1, 2, 16000000, 3), (0, 2, 33000000 // 2, 9)]
    g = v.Graph(*_graph(3, arcs))
    res = v.solve(g, [0, 0, 0], [1, 2, 2], [10, 6, 9], v.Config(use_bounds=1, pool_labels=1 << 24))
    assert res.found.tolist() == [1, 1, 1]
    assert res.cost.tolist() == [16000000, 32000000, 16500000]
    assert res.delay.tolist() == [3, 6, 9]
    g.close()


def test_zero_weights_and_unreachable():
    import vine_b200 as v
    arcs = [(0, 1, 0, 0), (1, 2, 0, 0), (2, 0, 0, 0), (2, 3, 0, 4), (0, 3, 2, 0), (4, 0, 1, 1)]
    g = v.Graph(*_graph(5, arcs))
    cfg = v.Config(use_bounds=1, pool_labels=1 << 24)
    res = v.solve(g, [0, 0, 0, 0, 1], [2, 3, 3, 4, 1], [0, 0, 4, 1e6, 0], cfg)
    assert res.found.tolist() == [1, 1, 1, 0, 1]
    assert res.cost[:3].tolist() == [0, 2, 0] and res.delay[:3].tolist() == [0, 0, 4]
    g.close()


@pytest.mark.parametrize("name", ["line33", "star257", "layers", "layers_wide", "heavy_arcs"])
def test_pareto_sets(name):
    """The sink's Pareto set, of the delay corridor, against the oracle's label setting
    without cost bounds."""
    import vine_b200 as v
    from oracle import oracle as O
    make, s, t = CASES[name]
    n, arcs = make(np.random.default_rng(17))
    csr = _graph(n, arcs)
    g, og = v.Graph(*csr), O.CsrGraph(*csr)
    _, h_del = O.lower_bounds(og, t)
    lo, hi = O.dijkstra(og, s, "delay")[0][t], O.dijkstra(og, s, "len")[1][t]
    budgets = np.array([lo - 1, lo, lo + 0.3 * (hi - lo), hi, 2 * hi + 10, 2.0 ** 24], np.float32)
    for cfg in (v.Config(mode="pareto", pool_labels=1 << 24),
                v.Config(mode="pareto", policy="ar", block_threads=64, table_log2=6, pool_labels=1 << 24)):
        r = v.solve(g, [s] * len(budgets), [t] * len(budgets), budgets, cfg, pareto_stride=2048)
        for q, b in enumerate(budgets):
            want = O.solve_label_setting(og, s, t, float(b), None, h_del, use_incumbent=False)
            assert bool(r.found[q]) == want["found"] and r.pareto_n[q] == len(want["pareto"]), (q, b)
            front = want["pareto"]
            np.testing.assert_array_equal(r.pareto(q), front[np.argsort(front[:, 0])])
            if want["found"]:
                assert r.path(q)[0] == s and r.path(q)[-1] == t
    g.close()


def _beside(chain, ring):
    """A chain 0 .. chain of long fast arcs beside a ring of short slow ones."""
    out = [(i, i + 1, 10, 1) for i in range(chain)]
    first = chain + 1
    out += [(first + i, first + (i + 1) % ring, 1, 10) for i in range(ring)]
    return chain + 1 + ring, out


@pytest.mark.parametrize("one_launch", [0, 1])
def test_first_path_past_the_keys(one_launch):
    """The first search meets on a path whose key its weights cannot bound."""
    import vine_b200 as v
    from oracle import oracle as O
    n, arcs = _beside(40, 400)
    csr = _graph(n, arcs)
    g, og = v.Graph(*csr), O.CsrGraph(*csr)
    _check(v, O, g, og, 0, 40, [100, 105],
           v.Config(use_bounds=1, policy="ar", table_log2=13, ctas_per_sm=one_launch, pool_labels=1 << 24))
    g.close()


def _no_delay_forth(n):
    return n, [a for i in range(n - 1) for a in ((i, i + 1, 10, 0), (i + 1, i, 10, 5))]


def _fast_row(k, rng):
    """A k x k grid of slow streets with one fast, long row at its edge."""
    out = []
    for r in range(k):
        for c in range(k):
            for rr, cc in ((r, c + 1), (r + 1, c)):
                if rr < k and cc < k:
                    fast = r == 0 and rr == 0
                    for u, x in ((r * k + c, rr * k + cc), (rr * k + cc, r * k + c)):
                        out.append((u, x, 30, 1) if fast else
                                   (u, x, int(rng.integers(1, 10)), int(rng.integers(10, 31))))
    return k * k, out


@pytest.mark.parametrize("one_launch", [0, 1])
@pytest.mark.parametrize("name", ["beside", "no_delay_forth", "fast_row", "halves", "unreachable"])
def test_paths_longer_than_the_budget_suggests(name, one_launch):
    """The cheapest path within the budget costs many times what the budget
    and the mean weights suggest, or there is none at all."""
    import vine_b200 as v
    from oracle import oracle as O
    n, arcs, s, t, budgets = {
        "beside": lambda: (*_beside(40, 400), 0, 40, [39, 40, 41, 100]),
        "no_delay_forth": lambda: (*_no_delay_forth(41), 0, 40, [0, 0.5, 3]),
        "fast_row": lambda: (*_fast_row(60, np.random.default_rng(4)), 0, 59, [58, 59, 60, 100]),
        # three arcs: the first and the last third fit the first search's keys, two do not
        "halves": lambda: (4004, [(0, 1, 50, 1), (1, 2, 50, 1), (2, 3, 50, 1)] +
                           [(4 + i, 4 + (i + 1) % 4000, 1, 1) for i in range(4000)], 0, 3, [2, 3, 4]),
        "unreachable": lambda: (*_beside(40, 400), 0, 45, [10, 1000, 1e6]),
    }[name]()
    csr = _graph(n, arcs)
    g, og = v.Graph(*csr), O.CsrGraph(*csr)
    _check(v, O, g, og, s, t, budgets,
           v.Config(use_bounds=1, policy="ar", table_log2=13, ctas_per_sm=one_launch, pool_labels=1 << 24))
    g.close()


@pytest.mark.parametrize("mode,far", [("pareto", 1024), ("pareto", 0), ("optimal", 1024)])
def test_searches_that_do_not_fit_the_piles(mode, far):
    """Waves hold labels that the bucketed search drops earlier, in half of its piles:
    a query that does not fit is searched again without its corridor within the
    call, which needs no retry.  Such piles held these queries before there were corridors."""
    import vine_b200 as v
    from oracle import oracle as O
    w = v.Workload.generate(1, rows=30, cols=30, n_pairs=24, alpha=(1.0,))
    og, g = O.CsrGraph(w.row_ptr, w.col, w.len, w.delay), w.graph()
    cfg = v.Config(mode=mode, use_bounds=int(mode == "optimal"), ctas_per_sm=1, far_capacity=far, pool_labels=1 << 27)
    res = v.solve(g, w.src, w.dst, w.budget, cfg, pareto_stride=512 if mode == "pareto" else 0)
    assert not res.status.any() and res.retried == 0
    for q in range(w.nq):
        s, t, b = int(w.src[q]), int(w.dst[q]), float(w.budget[q])
        h_len, h_del = O.lower_bounds(og, t)
        want = O.solve_label_setting(og, s, t, b, h_len if mode == "optimal" else None, h_del,
                                     use_incumbent=mode == "optimal")
        assert bool(res.found[q]) == want["found"]
        if want["found"]:
            assert (float(res.cost[q]), float(res.delay[q])) == (want["cost"], want["delay"])
            assert res.path(q)[0] == s and res.path(q)[-1] == t
        if mode == "pareto":
            front = want["pareto"]
            assert res.pareto_n[q] == len(front)
            np.testing.assert_array_equal(res.pareto(q), front[np.argsort(front[:, 0])])
    g.close()


@pytest.mark.parametrize("width,threads", [(0.0, 512), (1.0, 128), (1e7, 512)])
def test_large_pareto_fronts(width, threads):
    """Loose budgets on a 60 x 60 grid: up to 194 labels a vertex are kept, over many
    waves, over waves of a single cost and in one wave."""
    import vine_b200 as v
    from oracle import oracle as O
    w = v.Workload.generate(1, rows=60, cols=60, n_pairs=6, query_seed=5, alpha=(1.0,))
    og, g = O.CsrGraph(w.row_ptr, w.col, w.len, w.delay), w.graph()
    cfg = v.Config(mode="pareto", bucket_width=width, block_threads=threads, pool_labels=1 << 28)
    res = v.solve(g, w.src, w.dst, np.floor(1.5 * w.budget), cfg, pareto_stride=1024)
    assert not res.status.any() and res.pareto_n.max() > 100
    for q in range(w.nq):
        _, h_del = O.lower_bounds(og, int(w.dst[q]))
        want = O.solve_label_setting(og, int(w.src[q]), int(w.dst[q]), float(np.floor(1.5 * w.budget[q])), None, h_del,
                                     use_incumbent=False)
        front = want["pareto"]
        assert res.pareto_n[q] == len(front)
        np.testing.assert_array_equal(res.pareto(q), front[np.argsort(front[:, 0])])
    g.close()


def test_ends_apart_by_a_small_part():
    """One end reaches a few vertices only, the other one a chain of 55,000: the
    search ends with the small part (it had walked the chain, 140 ms)."""
    import vine_b200 as v
    n = 60000
    row = np.minimum(np.arange(n + 1), n - 1)
    g = v.Graph(row, np.arange(1, n), np.ones(n - 1, np.float32), np.ones(n - 1, np.float32))
    src, dst = [5000, 5000, 10, n - 3, 0], [3, 4999, 12, n - 6, 40]
    res = v.solve(g, src, dst, [1e6] * 5, v.Config(use_bounds=1, pool_labels=1 << 24), stats=True)
    assert res.found.tolist() == [0, 0, 1, 0, 1] and res.cost[2] == 2 and res.cost[4] == 40
    # rounds: as many as the small part has vertices, and a bucket on
    assert res.stats[0, 5] < 200 and res.stats[1, 5] < 6000
    g.close()


@pytest.mark.parametrize("engine", ["batch", "plain"])
@pytest.mark.parametrize("width", [0.01, 0.3, 1.0])
def test_narrow_buckets_of_large_costs(engine, width):
    """The first bucket starts at the source's bound, where the next float is
    1 away: it holds the source whatever its width (budgets without corridors)."""
    import vine_b200 as v
    arcs = [(0, 1, 5000000, 3), (1, 2, 5000001, 4), (2, 3, 4000000, 5), (0, 3, 15000000, 1)]
    g = v.Graph(*_graph(4, arcs))
    cfg = v.Config(engine=engine, use_bounds=1, bucket_width=width, pool_labels=1 << 22)
    res = v.solve(g, [0, 0, 1], [3, 3, 3], [2.0 ** 24, np.inf, 2.0 ** 25], cfg)
    assert res.found.tolist() == [1, 1, 1]
    assert res.cost.tolist() == [14000001, 14000001, 9000001] and res.delay.tolist() == [12, 12, 9]
    g.close()
