"""Calls with bounds run their corridors first, with up to four workers an
SM, and answer what does not fit them in a second launch.  Costs,
delays and feasibility are compared with the CPU oracle's label setting (all
of them integers: equality)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(width, depth, rng):
    n, arcs = width * depth, []
    for d in range(depth - 1):
        for i in range(width):
            for _ in range(3):
                arcs.append((d * width + i, (d + 1) * width + int(rng.integers(width)),
                             int(rng.integers(0, 101)), int(rng.integers(0, 101))))
    arcs.sort()
    row = np.searchsorted([a[0] for a in arcs], np.arange(n + 1))
    return (row.astype(np.int64), np.array([a[1] for a in arcs], np.int32),
            np.array([a[2] for a in arcs], np.float32), np.array([a[3] for a in arcs], np.float32))


@pytest.fixture(scope="module")
def case():
    """A layered graph, 26 queries and the oracle's answers to them."""
    from oracle import oracle as O
    csr, w, d = _layers(30, 25, np.random.default_rng(5)), 30, 25
    og, qs, want = O.CsrGraph(*csr), [], []
    for s, t in ((3, (d - 1) * w + 4), (40, 20 * w + 1), (7, 7), ((d - 1) * w, 2)):
        h_len, h_del = O.lower_bounds(og, t)
        lo = h_del[s] if np.isfinite(h_del[s]) else 50.0
        # the last two have no corridor: they are left to the second launch
        for b in ((-1.0, 0.0, 5.0) if s == t else (lo - 1, lo, lo + 40, lo * 1.3, lo * 2, 2.0 ** 24, np.inf)):
            qs.append((s, t, b))
            want.append(O.solve_label_setting(og, s, t, float(b), h_len, h_del, use_incumbent=True))
    return csr, qs, want


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _same(cost, delay, found, want, order):
    for q, k in enumerate(order):
        assert bool(found[q]) == want[k]["found"], q
        if want[k]["found"]:
            assert (float(cost[q]), float(delay[q])) == (want[k]["cost"], want[k]["delay"]), q


# 2^24 labels are fewer chunks than paired workers: some are left without
@pytest.mark.parametrize("pool", [1 << 24, 1 << 27])
@pytest.mark.parametrize("per_sm,extra", [(0, 1), (5, 0), (5, 1), (16, 0), (16, 1)])
def test_answers(case, per_sm, extra, pool):
    import vine_b200 as v
    csr, qs, want = case
    order = np.random.default_rng(9).integers(0, len(qs), per_sm * _sms() + extra)
    src, dst, bud = (np.array([qs[k][i] for k in order]) for i in range(3))
    g = v.Graph(*csr)
    for policy in ("ar", "fixed"):
        res = v.solve(g, src.astype(np.int32), dst.astype(np.int32), bud.astype(np.float32),
                      v.Config(use_bounds=1, policy=policy, pool_labels=pool, table_log2=13))
        _same(res.cost, res.delay, res.found, want, order)
        for q, k in enumerate(order):
            if want[k]["found"]:
                p = res.path(q)
                assert p[0] == src[q] and p[-1] == dst[q]
    g.close()


def test_invalid_queries_stay_invalid(case):
    import vine_b200 as v
    csr, qs, want = case
    n = 5 * _sms() + 30
    src, dst, bud = np.full(n, qs[2][0], np.int32), np.full(n, qs[2][1], np.int32), np.full(n, qs[2][2], np.float32)
    src[5], dst[70], bud[n - 1] = -1, len(csr[0]), np.nan
    g = v.Graph(*csr)
    with pytest.raises(v.VineError):
        v.solve(g, src, dst, bud, v.Config(use_bounds=1, pool_labels=1 << 27))
    g.close()


def test_captured_sequences_follow_the_workspace(case):
    """A captured small call, a larger one that grows the workspace, and the
    small one again; then the larger one captured and replayed."""
    import torch
    import vine_b200 as v
    csr, qs, want = case
    g = v.Graph(*csr)
    rng = np.random.default_rng(3)
    state = []
    for n in (40, 16 * _sms() + 1):
        order = rng.integers(0, len(qs), n)
        ins = [torch.tensor(np.array([qs[k][i] for k in order]), dtype=t, device="cuda")
               for i, t in enumerate((torch.int32, torch.int32, torch.float32))]
        out = {k: torch.empty(n, dtype=t, device="cuda") for k, t in
               (("cost", torch.float32), ("delay", torch.float32), ("found", torch.int32), ("status", torch.int32))}
        state.append((order, ins, out))
    s = torch.cuda.Stream()
    for which, captured in ((0, 1), (0, 1), (1, 0), (0, 1), (1, 1), (1, 1)):
        order, ins, out = state[which]
        for x in out.values():
            x.zero_()
        torch.cuda.synchronize()
        v.solve_device(g, *ins, out, v.Config(use_bounds=1, use_cuda_graph=captured, pool_labels=1 << 27), s.cuda_stream)
        s.synchronize()
        assert not out["status"].any()
        _same(out["cost"].cpu(), out["delay"].cpu(), out["found"].cpu(), want, order)
    g.close()


def test_captures_of_the_caller(case):
    """Calls captured by the caller, on the arrays of a small call (20 queries) and past
    them (40), replayed before and after larger calls have made others."""
    import torch
    import vine_b200 as v
    csr, qs, want = case
    g = v.Graph(*csr)
    rng = np.random.default_rng(7)
    cfg = v.Config(use_bounds=1, pool_labels=1 << 27)

    def call(n):
        order = rng.integers(0, len(qs), n)
        ins = [torch.tensor(np.array([qs[k][i] for k in order]), dtype=t, device="cuda")
               for i, t in enumerate((torch.int32, torch.int32, torch.float32))]
        out = {k: torch.empty(n, dtype=t, device="cuda") for k, t in
               (("cost", torch.float32), ("delay", torch.float32), ("found", torch.int32), ("status", torch.int32))}
        return order, ins, out

    def check(order, ins, out):
        torch.cuda.synchronize()
        assert not out["status"].any()
        _same(out["cost"].cpu(), out["delay"].cpu(), out["found"].cpu(), want, order)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        first = call(20)
        v.solve_device(g, *first[1], first[2], cfg, s.cuda_stream)
    check(*first)
    held = []
    for n in (20, 40):
        c, graph = call(n), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            v.solve_device(g, *c[1], c[2], cfg, s.cuda_stream)
        held.append((c, graph))
    for larger in (100, 5 * _sms() + 1):
        for c, graph in held:
            for x in c[2].values():
                x.zero_()
            graph.replay()
            check(*c)
        c = call(larger)
        torch.cuda.synchronize()
        v.solve_device(g, *c[1], c[2], cfg, s.cuda_stream)
        check(*c)
    for c, graph in held:
        for x in c[2].values():
            x.zero_()
        graph.replay()
        check(*c)
    del held, graph
    g.close()


@pytest.mark.parametrize("threads", [64, 512])
def test_calls_without_any_corridor(case, threads):
    """Budgets from 2^24 on: the first launch hands every query to the second."""
    import vine_b200 as v
    csr, qs, want = case
    some = [k for k, x in enumerate(qs) if x[2] >= 2.0 ** 24]
    order = np.array(some * 100)
    src, dst, bud = (np.array([qs[k][i] for k in order]) for i in range(3))
    g = v.Graph(*csr)
    cfg = v.Config(use_bounds=1, block_threads=threads, pool_labels=1 << 27, table_log2=13)
    for _ in range(3):
        res = v.solve(g, src.astype(np.int32), dst.astype(np.int32), bud.astype(np.float32), cfg)
        _same(res.cost, res.delay, res.found, want, order)
    g.close()
