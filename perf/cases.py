"""Performance cases: the work that users of the engine have it do.

Each case is a dict of plain values naming a family and its sizes.  The
graphs are the seeded workloads of this package (road lattices with
log-normal and with anti-correlated delays, the 4-neighbour grid, Chung-Lu);
a seed picks the queries: which source / sink pairs, in which order, and how
tight each delay budget is.  The graph itself stays, as a user's does.

  search   exact queries through ``solve`` (host arrays) or ``solve_device``
           (device tensors), with the engine's settings of the benchmark
           (reverse bounds, learned or AR bucket widths) or, ``tuning =
           "default"``, the class ``cspp`` with a default configuration, as
           the reference's callers use it
  pareto   every non-dominated (cost, delay) pair at the sink
  labels   the other label types: hop-constrained, max-cost, QoS bandwidth
  mlp      the scheduler network: training, gradients, predictions

Paths are asked for wherever a caller would want them and are packed by the
call, but not returned from ``run``: several paths may share the optimal
(cost, delay), and any of them is an answer.
"""
import functools
import heapq
import math

import numpy as np
import torch

import vine_b200 as v
from vine_b200 import scheduler

# Label arenas: large enough for every query drawn here, small enough for
# several handles on one device.
POOL_LARGE = 1 << 30
POOL_SMALL = 1 << 27


def listed():
    return [
        # The benchmark's workload: a night's batch of routing requests on a
        # city-sized road network, sinks 10 to 2000 hops away, every pair
        # asked with several delay budgets; inputs and outputs stay on the GPU.
        dict(name="road_batch_device", family="search", graph="road", rows=500, cols=528, hops=2000,
             pairs=1024, budgets=4, entry="device", tuning="learned"),
        # Random pairs across the same network at three tightness levels, from
        # host arrays and with paths: a what-if table for a planner.
        dict(name="road_pairs_host", family="search", graph="road", rows=500, cols=528, hops=0,
             pairs=32, budgets=3, entry="host", tuning="ar"),
        # One nearby destination, answered while somebody waits for it.
        dict(name="road_one_local", family="search", graph="road", rows=500, cols=528, hops=100,
             pairs=1, budgets=1, entry="host", tuning="ar"),
        # Fast roads cost more: delays anti-correlated with lengths give wide
        # Pareto fronts, the hard case for label setting.
        dict(name="anticorr_batch", family="search", graph="anticorr", rows=150, cols=150, hops=0,
             pairs=64, budgets=1, entry="host", tuning="ar"),
        # The smallest benchmark configuration: 16 pairs on the 100 x 100 grid.
        dict(name="grid_small", family="search", graph="grid", rows=100, cols=100, hops=0,
             pairs=16, budgets=1, entry="host", tuning="ar"),
        # The reference's own call sequence (labels, sinks, constraints,
        # solve()) with nothing configured.
        dict(name="grid_default", family="search", graph="grid", rows=45, cols=45, hops=0,
             pairs=16, budgets=1, entry="cspp", tuning="default"),
        # A power-law network (hubs, few hops), 64 queries.
        dict(name="chunglu_batch", family="search", graph="chunglu", rows=1, cols=100000, hops=6,
             pairs=64, budgets=1, entry="host", tuning="ar"),
        # The whole trade-off curve between cost and delay for a few pairs.
        dict(name="pareto_grid", family="pareto", graph="grid", rows=31, cols=31, hops=0,
             pairs=8, budgets=1),
        # Three or four criteria per label, on an odd-sized grid.
        dict(name="labels_maxcost", family="labels", kind="maxcost", graph="grid", rows=33, cols=33,
             hops=0, pairs=16, budgets=1),
        # Cheapest path over links of at least a given bandwidth.
        dict(name="labels_qos", family="labels", kind="qos", graph="road", rows=150, cols=151,
             hops=0, pairs=64, budgets=1),
        # One epoch of scheduler training, as the training recipe batches it.
        dict(name="mlp_train", family="mlp", op="train", rows=100000, batch=512),
        # Loss and gradient over a trace that somebody looks into.
        dict(name="mlp_loss_grad", family="mlp", op="loss_grad", rows=65536),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    what = rng.choice(["road", "road", "road", "anticorr", "grid", "default", "chunglu", "pareto",
                       "labels", "mlp"])
    if what == "road":
        queries = _log_int(rng, 1, 1024)
        pairs = min(queries, 192)
        hops = rng.choice([0, 1, 1, 1]) * _log_int(rng, 12, 2000)
        return dict(family="search", graph="road", rows=500, cols=528, hops=hops, pairs=pairs,
                    budgets=-(-queries // pairs), entry=rng.choice(["host", "device"]),
                    tuning=rng.choice(["ar", "learned"]))
    if what == "anticorr":
        side = _log_int(rng, 60, 180)
        return dict(family="search", graph="anticorr", rows=side, cols=side + rng.randrange(9),
                    hops=0, pairs=_log_int(rng, 1, 64), budgets=1,
                    entry=rng.choice(["host", "device"]), tuning=rng.choice(["ar", "learned"]))
    if what == "grid":
        side = _log_int(rng, 20, 120)
        return dict(family="search", graph="grid", rows=side, cols=side + rng.randrange(9), hops=0,
                    pairs=_log_int(rng, 1, 64), budgets=rng.choice([1, 3]),
                    entry=rng.choice(["host", "device"]), tuning=rng.choice(["ar", "learned"]))
    if what == "default":
        side = _log_int(rng, 12, 50)
        return dict(family="search", graph="grid", rows=side, cols=side + rng.randrange(9), hops=0,
                    pairs=_log_int(rng, 1, 32), budgets=1, entry="cspp", tuning="default")
    if what == "chunglu":
        return dict(family="search", graph="chunglu", rows=1, cols=_log_int(rng, 3000, 100000),
                    hops=rng.choice([4, 5, 6]), pairs=_log_int(rng, 1, 64), budgets=1,
                    entry=rng.choice(["host", "device"]), tuning=rng.choice(["ar", "learned"]))
    if what == "pareto":
        side = _log_int(rng, 10, 36)
        return dict(family="pareto", graph="grid", rows=side, cols=side + rng.randrange(9), hops=0,
                    pairs=_log_int(rng, 1, 16), budgets=1)
    if what == "labels":
        kind = rng.choice(["hop", "maxcost", "qos"])
        road = kind == "qos"
        side = _log_int(rng, 50, 180) if road else _log_int(rng, 12, 36)
        return dict(family="labels", kind=kind, graph="road" if road else "grid", rows=side,
                    cols=side + rng.randrange(9), hops=0, pairs=_log_int(rng, 1, 64 if road else 16),
                    budgets=1)
    op = rng.choice(["train", "loss_grad", "forward"])
    case = dict(family="mlp", op=op, rows=_log_int(rng, 30, 150000))
    if op == "train":
        case["batch"] = rng.choice([256, 512, 1024, 1500])
    return case


# ------------------------------------------------------------------- workloads


@functools.lru_cache(maxsize=8)
def _pool(graph, rows, cols, hops, pairs):
    """The graph and a pool of source / sink pairs with their tightest and
    loosest useful budgets (smallest delay; delay of the shortest path)."""
    config = {"road": 5 if hops else 2, "anticorr": 3, "grid": 1, "chunglu": 4}[graph]
    over = dict(n_pairs=max(64, pairs), query_seed=11)
    if graph == "chunglu":
        over.update(n=cols, m_target=20 * cols, hop_lo=3, hop_hi=hops)
    else:
        over.update(rows=rows, cols=cols)
        n = rows * cols
        if graph == "road":
            over.update(m_target=int(n * 733000 / 264000))
        if graph == "anticorr":
            over.update(m_target=int(n * 2.6))
        if hops:
            over.update(hop_lo=10, hop_hi=hops)
    tight = v.Workload.generate(config, alpha=(0.0,), **over)
    loose = v.Workload.generate(config, alpha=(1.0,), **over)
    ok = tight.budget >= 0
    return tight, tight.src[ok], tight.dst[ok], tight.budget[ok], loose.budget[ok]


def _queries(case, seed):
    w, src, dst, lo, hi = _pool(case["graph"], case["rows"], case["cols"], case["hops"], case["pairs"])
    rng = np.random.default_rng(seed)
    pick = np.resize(rng.permutation(len(src)), case["pairs"])
    pick = rng.permutation(np.repeat(pick, case["budgets"]))
    alpha = rng.uniform(0.1, 0.9, len(pick))
    budget = np.floor(lo[pick] + alpha * (hi[pick] - lo[pick])).astype(np.float32)
    return w, src[pick], dst[pick], budget


def _limits(case, w, src, dst, budget):
    """Limits of the other label types that bind for a part of the queries."""
    if case["kind"] == "qos":
        return dict(delay_limit=np.full(len(src), np.quantile(w.delay, 0.08), np.float32))
    cols = case["cols"]
    hops = np.abs(src // cols - dst // cols) + np.abs(src % cols - dst % cols)
    lim = dict(delay_limit=budget, hop_limit=np.ceil(1.15 * hops + 2).astype(np.float32))
    if case["kind"] == "maxcost":
        lim["maxcost_limit"] = np.full(len(src), 97.0, np.float32)
    return lim


def _mlp_data(case, seed):
    """Feature rows on the scale of real traces, with targets (log2 of a
    multiplier, gate)."""
    rng = np.random.default_rng(seed)
    x = np.abs(rng.normal(0.0, 1.0, (case["rows"], 16))).astype(np.float32)
    x *= np.array([8, 8, 8, 6, 12, 5, 1, 0.5, 0.5, 4, 1, 0.3, 0.3, 1, 0.5, 6], np.float32)
    gate = (rng.uniform(size=case["rows"]) < 0.3).astype(np.float32)
    y = np.stack([gate * rng.uniform(-1.5, 1.5, case["rows"]).astype(np.float32), gate], axis=1)
    return x, y.astype(np.float32)


def _mlp_params(seed):
    rng = np.random.default_rng([seed, 1])
    parts = [rng.uniform(-1, 1, n) * math.sqrt(6.0 / fan) * on
             for n, fan, on in ((1024, 16, 1), (64, 1, 0), (4096, 64, 1), (64, 1, 0), (128, 64, 1), (2, 1, 0))]
    return np.concatenate(parts).astype(np.float32)


# ------------------------------------------------------------------ the cases


def prepare(case, seed):
    if case["family"] == "mlp":
        x, y = _mlp_data(case, seed)
        return dict(case=case, mlp=v.MLP(params=_mlp_params(seed)), params=_mlp_params(seed), x=x, y=y)
    w, src, dst, budget = _queries(case, seed)
    g = w.graph()
    g.make_gpu_graph()
    st = dict(case=case, graph=g, src=src, dst=dst, budget=budget)
    pool = POOL_LARGE if case["pairs"] * case["budgets"] > 64 and case["hops"] != 6 else POOL_SMALL
    if case["family"] == "labels":
        st["limits"] = _limits(case, w, src, dst, budget)
        return st
    if case["family"] == "pareto":
        st["config"] = v.Config(mode="pareto", pool_labels=pool)
        return st
    if case["tuning"] == "default":
        st["config"] = v.Config(pool_labels=pool)
    elif case["tuning"] == "learned":
        st["mlp"] = scheduler.load()[0]
        st["config"] = scheduler.base_config(float(w.len.mean()), policy="mlp", mlp=st["mlp"], pool_labels=pool)
    else:
        st["config"] = scheduler.base_config(float(w.len.mean()), policy="ar", pool_labels=pool)
    if case["entry"] == "device":
        nq = len(src)
        st["src"], st["dst"], st["budget"] = (torch.from_numpy(a).cuda() for a in (src, dst, budget))
        st["out"] = dict(cost=torch.empty(nq, device="cuda"), delay=torch.empty(nq, device="cuda"),
                         found=torch.empty(nq, dtype=torch.int32, device="cuda"),
                         status=torch.empty(nq, dtype=torch.int32, device="cuda"),
                         path_offsets=torch.empty(nq + 1, dtype=torch.int64, device="cuda"),
                         path=torch.empty(nq * min(w.n, 8192), dtype=torch.int32, device="cuda"))
    return st


def run(state):
    case = state["case"]
    if case["family"] == "mlp":
        m = state["mlp"]
        if case["op"] == "forward":
            return dict(y=m.forward(state["x"]))
        if case["op"] == "loss_grad":
            loss, grad = m.loss_grad(state["x"], state["y"])
            return dict(loss=loss, grad=grad)
        # a fresh network each time, as the training recipe makes one
        m = v.MLP(params=state["params"])
        loss = m.train(state["x"], state["y"], epochs=1, batch=case["batch"], lr=1e-3, seed=3)
        return dict(loss=loss, params=m.params)
    g, src, dst = state["graph"], state["src"], state["dst"]
    if case["family"] == "labels":
        r = v.solve_labels(g, case["kind"], src, dst, **state["limits"])
        return dict(cost=r.cost, delay=r.delay, found=r.found, status=r.status, extra=r.extra)
    if case["family"] == "pareto":
        r = v.solve(g, src, dst, state["budget"], state["config"], pareto_stride=1024)
        return dict(cost=r.cost, delay=r.delay, found=r.found, n=r.pareto_n, d=r.pareto_d, dl=r.pareto_delay)
    if case["entry"] == "device":
        out = state["out"]
        v.solve_device(g, src, dst, state["budget"], out, state["config"])
        return {k: out[k] for k in ("cost", "delay", "found", "status")}
    if case["entry"] == "cspp":
        c = v.cspp(g, len(src), [v.c_label(int(s)) for s in src], [int(t) for t in dst],
                   [v.c_constraint(float(b)) for b in state["budget"]], config=state["config"])
        c.solve()
        return dict(cost=c.cost_l, delay=c.delay_l, found=c.found_l, status=c.status_l)
    r = v.solve(g, src, dst, state["budget"], state["config"])
    return dict(cost=r.cost, delay=r.delay, found=r.found, status=r.status)


def work(case):
    """Inputs read once and outputs written once; for the network its
    multiply-adds, forward and (with gradients) twice that backward."""
    if case["family"] == "mlp":
        n, flops = case["rows"], 2 * (16 * 64 + 64 * 64 + 64 * 2)
        passes = {"forward": 1, "loss_grad": 3, "train": 4}[case["op"]]
        return {"bytes": n * 4 * 18 + 2 * 4 * 5378, "flops": n * flops * passes}
    n = case["rows"] * case["cols"]
    m = n * {"road": 733434 / 264000, "anticorr": 2.6, "grid": 4, "chunglu": 18}[case["graph"]]
    nq = case["pairs"] * case["budgets"]
    return {"bytes": 4 * (n + 1) + 12 * m + 12 * nq + 16 * nq, "flops": 0}


# --------------------------------------------------------------- exact answers


def _mlp_exact(case, seed):
    x, y = (torch.from_numpy(a).double() for a in _mlp_data(case, seed))
    p = torch.from_numpy(_mlp_params(seed)).double().requires_grad_()
    w1, b1, w2, b2, w3, b3 = torch.split(p, [1024, 64, 4096, 64, 128, 2])
    h = torch.relu(x @ w1.view(64, 16).T + b1)
    h = torch.relu(h @ w2.view(64, 64).T + b2)
    out = h @ w3.view(2, 64).T + b3
    if case["op"] == "forward":
        return dict(y=out.detach().numpy())
    # mean over rows of the squared error summed over both outputs
    loss = ((out - y) ** 2).sum() / case["rows"]
    loss.backward()
    return dict(loss=float(loss.detach()), grad=p.grad.numpy())


def _adjacency(w):
    fwd = [[] for _ in range(w.n)]
    rev = [[] for _ in range(w.n)]
    row, col, ln, dl = w.row_ptr.tolist(), w.col.tolist(), w.len.tolist(), w.delay.tolist()
    for u in range(w.n):
        for j in range(row[u], row[u + 1]):
            fwd[u].append((col[j], ln[j], dl[j]))
            rev[col[j]].append((u, ln[j], dl[j]))
    return fwd, rev


def _dijkstra(adj, s, which, radius=math.inf):
    dist, heap = {s: 0.0}, [(0.0, s)]
    while heap:
        d, u = heapq.heappop(heap)
        if d > dist[u]:
            continue
        for arc in adj[u]:
            nd = d + arc[which]
            if nd <= radius and nd < dist.get(arc[0], math.inf):
                dist[arc[0]] = nd
                heapq.heappush(heap, (nd, arc[0]))
    return dist


def _label_setting(adj, s, t, budget, limit, h_len, h_del, front):
    """Non-dominated (cost, delay) pairs at t in order of cost, the first one
    alone unless `front`; None past `limit` labels."""
    heap, best, found, seen = [(h_len.get(s, math.inf), 0.0, 0.0, s)], {}, [], 0
    if h_del.get(s, math.inf) > budget:
        return []
    while heap:
        _, dl, d, u = heapq.heappop(heap)
        if dl >= best.get(u, math.inf):
            continue
        best[u] = dl
        if u == t:
            found.append((d, dl))
            if not front:
                break
            continue
        seen += 1
        if seen > limit:
            return None
        for x, a, b in adj[u]:
            nl = dl + b
            if x in h_del and nl + h_del[x] <= budget and nl < best.get(x, math.inf):
                heapq.heappush(heap, (d + a + h_len[x], nl, d + a, x))
    return found


def _qos_best(adj, s, t, floor):
    best, heap = {s: (0.0, -21474836.0)}, [(0.0, -21474836.0, s)]
    while heap:
        d, nb, u = heapq.heappop(heap)
        if (d, nb) > best[u]:
            continue
        if u == t:
            return d, -nb
        for x, a, b in adj[u]:
            key = (d + a, max(nb, -b))
            if b >= floor and key < best.get(x, (math.inf, 0.0)):
                best[x] = key
                heapq.heappush(heap, (*key, x))
    return math.inf, math.inf


def exact(case, seed):
    if case["family"] == "mlp":
        return None if case["op"] == "train" else _mlp_exact(case, seed)
    w, src, dst, budget = _queries(case, seed)
    nq = len(src)
    if w.n > 25000 or nq * w.n > 2000000:
        return None
    if case["family"] == "labels":
        if case["kind"] != "qos":
            return None
        fwd, _ = _adjacency(w)
        floor = float(_limits(case, w, src, dst, budget)["delay_limit"][0])
        got = [_qos_best(fwd, int(s), int(t), floor) for s, t in zip(src, dst)]
        return dict(cost=np.array([g[0] for g in got]), delay=np.array([g[1] for g in got]),
                    found=None, status=None, extra=None)
    fwd, rev = _adjacency(w)
    cost, delay = np.full(nq, np.inf), np.full(nq, np.inf)
    d, dl = np.zeros((nq, 1024)), np.zeros((nq, 1024))
    left = 400000
    for q in range(nq):
        h_del = _dijkstra(rev, int(dst[q]), 2, float(budget[q]))
        h_len = _dijkstra(rev, int(dst[q]), 1)
        front = _label_setting(fwd, int(src[q]), int(dst[q]), float(budget[q]), left, h_len, h_del,
                               case["family"] == "pareto")
        if front is None:
            return None
        left -= 1000
        if front:
            cost[q], delay[q] = front[0]
            front = np.array(front[:1024])
            d[q, :len(front)], dl[q, :len(front)] = front[:, 0], front[:, 1]
    out = dict(cost=cost, delay=delay, found=None)
    if case["family"] == "pareto":
        return dict(out, n=None, d=d, dl=dl)
    return dict(out, status=None)
