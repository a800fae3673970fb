"""The work that users of this framework have it do, as cases to be timed.

Every case goes through the package's public entry points, as a program that
matches queries on a resident data graph calls them: single queries, batches,
local counts, embeddings, candidate spaces, set intersections, and the learned
cardinality estimator in both directions.  Data graphs have the shapes of the
package's own configurations (asdmatch_b200/specs.py): the small ones are made
from the seed, the two large ones are the resident data set (one graph for
every seed; the queries walked on them are the inputs).

Exact counts of large queries go past any time a user waits, so cases whose
queries can have many matches set a count limit, as the collection of training
targets does: a query then has an exact count, a proven overflow, or the status
"limit reached"; its count means something only in the first case.
"""
import functools
import math

import numpy as np
import torch

import asdmatch_b200 as A
from asdmatch_b200 import specs

LARGE = {"C1": specs.C1, "C4": specs.C4}
SMALL = {"C0": specs.C0, "C0D": specs.C0D}
FEATURES = 44  # the estimator's node features
HIDDEN = 128


def listed():
    return [
        # one 8-vertex query on a graph of 3,112 vertices and 71 labels: an interactive lookup, where latency and
        # launches are all there is
        {"name": "count_small", "kind": "count", "graph": "C0", "n": 3112, "size": 8, "density": 0,
         "limit": 10 ** 8},
        # one 6-vertex query on the resident graph of 3.77M vertices that has an exact count within reach
        {"name": "count_large", "kind": "count", "graph": "C1", "n": 0, "size": 6, "density": 0, "limit": 10 ** 11},
        # 200 selective 8-vertex queries on the small graph, one call: the batched form of count_small
        {"name": "batch_small", "kind": "batch", "graph": "C0", "n": 3112, "queries": 200, "size_min": 8,
         "size_max": 8, "limit": 0},
        # 64 queries of 6 to 8 vertices on the small graph with 8 labels: 10^3 to 10^8 matches each, counted exactly
        {"name": "batch_dense", "kind": "batch", "graph": "C0D", "n": 3112, "queries": 64, "size_min": 6,
         "size_max": 8, "limit": 0},
        # the mixed batch on the large resident graph, 4 to 32 vertices: the headline workload
        {"name": "batch_large", "kind": "batch", "graph": "C1", "n": 0, "queries": 512, "size_min": 4,
         "size_max": 32, "limit": 10 ** 8},
        # local counts (a |Vg| x |Vq| matrix) of one query, as the command line's -c asks for them
        {"name": "local_small", "kind": "local", "graph": "C0D", "n": 3112, "queries": 1, "size_min": 6,
         "size_max": 6},
        # batched local counts on the graph of 1M vertices and 10M edges
        {"name": "local_large", "kind": "local", "graph": "C4", "n": 0, "queries": 8, "size_min": 4, "size_max": 5},
        # the sorted embeddings of one query, up to two million rows
        {"name": "embed", "kind": "embed", "graph": "C0D", "n": 3112, "size": 6, "rows_min": 400_000,
         "rows_max": 2_000_000},
        # candidate spaces of four queries on the large graph, read back by a caller that plans by itself
        {"name": "space", "kind": "space", "graph": "C1", "n": 0, "queries": 4, "size_min": 4, "size_max": 16},
        # k-way intersections of sorted lists of uneven lengths, batched
        {"name": "intersect", "kind": "intersect", "sets": 256, "lists": 3, "len_min": 16, "len_max": 20_000},
        # estimates of 4,096 sub-queries, the estimator's evaluation batch
        {"name": "predict", "kind": "predict", "graphs": 4096, "size_max": 6},
        # one optimiser step on 256 sub-queries, the estimator's training batch
        {"name": "train", "kind": "train", "graphs": 256, "size_max": 6},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["count", "count", "batch", "batch", "batch", "local", "local", "embed", "space", "intersect",
                       "predict", "train"])
    if kind == "count":
        if rng.random() < 0.5:
            return {"kind": kind, "graph": "C0", "n": _log_int(rng, 1000, 50_000), "size": rng.randint(4, 16),
                    "density": 0, "limit": 10 ** 8}
        return {"kind": kind, "graph": "C1", "n": 0, "size": rng.randint(4, 8), "density": rng.choice([0, 1, 2]),
                "limit": 10 ** 11}
    if kind == "batch":
        where = rng.choice(["C0", "C0D", "C1"])
        if where == "C0":
            size = rng.randint(4, 12)
            return {"kind": kind, "graph": where, "n": _log_int(rng, 1000, 50_000), "queries": _log_int(rng, 2, 400),
                    "size_min": size, "size_max": min(12, size + rng.randint(0, 4)), "limit": 10 ** 8}
        if where == "C0D":
            size = rng.randint(4, 7)
            return {"kind": kind, "graph": where, "n": rng.randint(1500, 3500), "queries": _log_int(rng, 4, 64),
                    "size_min": size, "size_max": size + 1, "limit": 10 ** 8}
        size = rng.randint(4, 24)
        return {"kind": kind, "graph": where, "n": 0, "queries": _log_int(rng, 4, 400), "size_min": size,
                "size_max": rng.randint(size, 32), "limit": 10 ** 8}
    if kind == "local":
        size = rng.randint(4, 5)
        if rng.random() < 0.5:
            return {"kind": kind, "graph": "C0D", "n": rng.randint(1500, 4000), "queries": rng.randint(1, 16),
                    "size_min": size, "size_max": size + 1}
        return {"kind": kind, "graph": "C4", "n": 0, "queries": rng.randint(1, 8), "size_min": 4, "size_max": size}
    if kind == "embed":
        lo = _log_int(rng, 100, 200_000)
        return {"kind": kind, "graph": "C0D", "n": rng.randint(2500, 3500), "size": rng.randint(4, 6), "rows_min": lo,
                "rows_max": 10 * lo}
    if kind == "space":
        size = rng.randint(4, 16)
        return {"kind": kind, "graph": rng.choice(["C1", "C4"]), "n": 0, "queries": rng.randint(1, 8),
                "size_min": size, "size_max": min(16, size + rng.randint(0, 8))}
    if kind == "intersect":
        top = _log_int(rng, 100, 50_000)
        return {"kind": kind, "sets": _log_int(rng, 1, 256), "lists": rng.randint(2, 6),
                "len_min": _log_int(rng, 1, top), "len_max": top}
    if kind == "predict":
        return {"kind": kind, "graphs": _log_int(rng, 1, 8192), "size_max": rng.randint(3, 8)}
    return {"kind": "train", "graphs": _log_int(rng, 16, 2048), "size_max": rng.randint(3, 8)}


# ---- inputs -----------------------------------------------------------------

def _chung_lu(spec):
    return A.HostGraph.chung_lu(spec["n"], spec["m"], spec["gamma"], spec["nlabels"], spec["zipf_s"], spec["seed"])


@functools.lru_cache(maxsize=2)
def _large_graph(name):
    return _chung_lu(LARGE[name])


def _host_graph(case, seed):
    if case["graph"] in LARGE:
        return _large_graph(case["graph"])
    spec = dict(SMALL[case["graph"]])
    spec["m"] = int(round(spec["m"] * case["n"] / spec["n"]))
    spec["n"], spec["seed"] = case["n"], 17 * seed + 5
    return _chung_lu(spec)


def _walk(g, size, density, seed):
    """The query of the first walk from `seed` on that gives one of this size and density."""
    while True:
        try:
            return g.random_walk_query(size, seed, density)
        except A.AsdmError as e:
            if e.code != A.ERR_INVALID:
                raise
            seed += 1


def _queries(g, case, seed):
    """Sizes uniform over the case's range, in a mixed order that is the same for every seed."""
    span = case["size_max"] - case["size_min"] + 1
    sizes = [case["size_min"] + i * 2654435761 % 2 ** 32 % span for i in range(case["queries"])]
    return [_walk(g, s, 0, 1_000_000 * (seed + 1) + 1000 * i) for i, s in enumerate(sizes)]


def _counted_query(dg, g, case, seed, least, most):
    """The first walk whose match count is in [least, most]; the largest count up to `most` where none is."""
    best = None
    for i in range(400):
        q = _walk(g, case["size"], case.get("density", 0), 1_000_000 * (seed + 1) + 1000 * i)
        try:
            rows = A.count_query(dg, q, time_limit_s=1.0, count_limit=most).count
        except A.AsdmError:
            continue
        if best is None or rows > best[0]:
            best = (rows, q)
        if rows >= least:
            break
    return best[1] if best else q


def _lists(case, seed):
    """Sorted lists for set intersections: lengths log-uniform, the lists of a set drawn from one range of ids."""
    rng = np.random.default_rng([seed, case["sets"], case["lists"]])
    out = []
    for _ in range(case["sets"]):
        lens = np.exp(rng.uniform(np.log(case["len_min"]), np.log(case["len_max"] + 1), case["lists"])).astype(int)
        top = 4 * int(lens.max()) + 8
        out.append([np.unique(rng.integers(0, top, max(1, int(k)), dtype=np.uint32)) for k in lens])
    return out


def _subqueries(case, seed):
    """A batch of random connected sub-queries with features of the estimator's kinds and ranges: a one-hot label,
    scaled logarithms of set and list sizes, degrees, sizes; (x, adj_off, adj, node_graph, target)."""
    rng = np.random.default_rng([seed, case["graphs"], case["size_max"]])
    sizes = rng.integers(3, case["size_max"] + 1, case["graphs"])
    n = int(sizes.sum())
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    node_graph = np.repeat(np.arange(case["graphs"]), sizes)
    local = np.arange(n) - first[node_graph]
    # a random tree (every vertex hangs on an earlier one) and, in half of the graphs, one more edge
    child = np.nonzero(local > 0)[0]
    parent = first[node_graph[child]] + (rng.random(len(child)) * local[child]).astype(np.int64)
    more = np.nonzero((rng.random(case["graphs"]) < 0.5) & (sizes >= 4))[0]
    a, b = first[more], first[more] + sizes[more] - 1
    pairs = np.unique(np.concatenate([np.stack([parent, child], 1), np.stack([a, b], 1)]), axis=0)
    both = np.concatenate([pairs, pairs[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    adj_off = np.concatenate([[0], np.cumsum(np.bincount(both[:, 0], minlength=n))]).astype(np.uint32)
    adj = both[:, 1].astype(np.uint32)
    x = np.zeros((n, FEATURES), np.float32)
    x[np.arange(n), np.minimum(rng.geometric(0.2, n) - 1, 31)] = 1
    x[:, 32:40] = rng.uniform(-0.3, 1.0, (n, 8))
    x[:, 40] = 1
    x[:, 41] = sizes[node_graph] / 16
    x[:, 42:44] = rng.integers(0, 3, (n, 2)) / 8
    target = rng.uniform(1.0, 25.0, case["graphs"]).astype(np.float32)
    return x, adj_off, adj, node_graph.astype(np.uint32), target


def _weights(seed):
    """Model parameters in the estimator's order: three 128 x 256 layers, their biases, the readout and its bias."""
    rng = np.random.default_rng([seed, 11])
    a, ao = math.sqrt(6 / (3 * HIDDEN)), math.sqrt(6 / (HIDDEN + 1))
    return np.concatenate([rng.uniform(-a, a, 3 * HIDDEN * 2 * HIDDEN), rng.uniform(-0.1, 0.1, 3 * HIDDEN),
                           rng.uniform(-ao, ao, HIDDEN), [0.5]]).astype(np.float32)


LEARNING_RATE = 1e-3
MOST_IDS = 4_000_000  # candidates of a query that a caller of `space` keeps


def prepare(case, seed):
    torch.cuda.current_device()
    kind = case["kind"]
    if kind == "intersect":
        return {"kind": kind, "lists": _lists(case, seed), "sizes": np.zeros(case["sets"], np.uint32),
                "rows": np.zeros((case["sets"], case["len_max"]), np.uint32)}
    if kind in ("predict", "train"):
        est = A.Estimator(FEATURES)
        est.set_params(_weights(seed))
        return {"kind": kind, "est": est, "batch": _subqueries(case, seed), "graphs": case["graphs"]}
    g = _host_graph(case, seed)
    dg = A.DeviceGraph(g)
    state = {"kind": kind, "dg": dg}
    if kind == "count":
        state["query"] = _counted_query(dg, g, case, seed, 1, case["limit"] // 10)
        state["limit"] = case["limit"]
    elif kind == "batch":
        state["batch"] = A.BatchInput(_queries(g, case, seed))
        state["limit"] = case["limit"]
    elif kind == "embed":
        state["query"] = _counted_query(dg, g, case, seed, case["rows_min"], case["rows_max"])
        state["table"] = np.zeros((case["rows_max"], case["size"]), np.uint32)
    else:
        state["queries"] = _queries(g, case, seed)
    if kind == "space":
        # |C(u)|, the candidate-edge totals and the candidates, a row per query
        state["sizes"] = np.zeros((case["queries"], 32), np.uint32)
        state["totals"] = np.zeros((case["queries"], 32 * 31), np.uint64)
        state["ids"] = np.zeros((case["queries"], MOST_IDS), np.uint32)
    return state


# ---- one pass ---------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "count":
        try:
            return [A.OK, A.count_query(state["dg"], state["query"], count_limit=state["limit"]).count]
        except A.AsdmError as e:  # past the limit, or a proven overflow
            return [e.code, 0]
    if kind == "batch":
        b = state["batch"]
        A.run_batch_ex(state["dg"], b, count_limit=state["limit"])
        return {"status": b.status.copy(), "counts": np.where(b.status == A.OK, b.counts, 0)}
    if kind == "local":
        if len(state["queries"]) == 1:
            r = A.match(state["dg"], state["queries"][0], A.MODE_LOCAL)
            return {"counts": np.array([r.count], np.uint64), "local": [r.local_counts]}
        counts, status, local = A.run_batch_local(state["dg"], state["queries"])
        return {"counts": counts, "status": status, "local": local}
    if kind == "embed":
        r = A.match(state["dg"], state["query"], A.MODE_EMBED)
        table = state["table"]
        table[:r.count] = r.embeddings
        return {"count": r.count, "rows": table}
    if kind == "space":
        sizes, totals, ids = state["sizes"], state["totals"], state["ids"]
        for i, cs in enumerate(A.candidate_spaces(state["dg"], state["queries"])):
            sizes[i, :cs.q.n] = cs.sizes()
            edges = cs.edge_totals()
            totals[i, :len(edges)] = edges
            at = 0
            for u in range(cs.q.n):
                c = cs.candidate_set(u)[:MOST_IDS - at]
                ids[i, at:at + len(c)] = c
                at += len(c)
            cs.close()
        return {"sizes": sizes, "totals": totals, "ids": ids}
    if kind == "intersect":
        sizes, rows = state["sizes"], state["rows"]
        for i, found in enumerate(A.leapfrog_join(state["lists"])):
            sizes[i] = len(found)
            rows[i, :len(found)] = found
        return {"sizes": sizes, "rows": rows}
    x, adj_off, adj, node_graph, target = state["batch"]
    est = state["est"]
    if kind == "predict":
        return est.predict(x, adj_off, adj, node_graph, state["graphs"])
    loss = est.train_step(x, adj_off, adj, node_graph, target, lr=LEARNING_RATE)
    return {"loss": loss, "params": est.params()}


# ---- what a pass cannot do without --------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "intersect":
        lo, hi = case["len_min"], case["len_max"] + 1
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        return {"bytes": int(4 * case["sets"] * (case["lists"] + 0.25) * mean), "flops": 0}
    if kind in ("predict", "train"):
        nodes = case["graphs"] * (3 + case["size_max"]) / 2
        layer = 2 * nodes * 2 * HIDDEN * HIDDEN  # one product of a layer
        params = 3 * 2 * HIDDEN * HIDDEN + 4 * HIDDEN + 1
        batch = 4 * (nodes * (FEATURES + 4) + 2 * case["graphs"])
        if kind == "predict":
            return {"bytes": int(batch + 4 * params), "flops": int(3 * layer)}
        # forward, weight gradients, input gradients (not of the first layer); parameters and both moments read
        # and written
        return {"bytes": int(batch + 24 * params), "flops": int(8 * layer)}
    # the data graph's lists and labels, once; counts cost nothing beside them
    spec = LARGE.get(case["graph"]) or SMALL[case["graph"]]
    n = case["n"] or spec["n"]
    m = spec["m"] * n / spec["n"]
    total = 8 * m + 8 * n
    size = case.get("size", (case.get("size_min", 0) + case.get("size_max", 0)) / 2)
    if kind == "local":
        total += 8 * n * size * case["queries"]
    if kind == "embed":
        total += 4 * size * math.sqrt(case["rows_min"] * case["rows_max"])
    return {"bytes": int(total), "flops": 0}


# ---- computed numbers in 64 bits ----------------------------------------------

def exact(case, seed):
    if case["kind"] not in ("predict", "train"):
        return None  # whole numbers
    x, adj_off, adj, node_graph, target = _subqueries(case, seed)
    p = _weights(seed).astype(np.float64)
    n, ng, h = len(x), case["graphs"], HIDDEN
    wsize = h * 2 * h
    W = [p[k * wsize:(k + 1) * wsize].reshape(h, 2 * h) for k in range(3)]
    bias = [p[3 * wsize + k * h:3 * wsize + (k + 1) * h] for k in range(3)]
    wo, bo = p[3 * wsize + 3 * h:3 * wsize + 4 * h], p[-1]
    src = np.repeat(np.arange(n), np.diff(adj_off.astype(np.int64)))

    def around(v):  # sum over a node's neighbours
        out = np.zeros_like(v)
        np.add.at(out, src, v[adj])
        return out

    def per_graph(v):
        out = np.zeros((ng, v.shape[1]))
        np.add.at(out, node_graph, v)
        return out

    H = np.zeros((n, h))
    H[:, :FEATURES] = x
    X, Z = [], []
    for k in range(3):
        X.append(np.concatenate([H, around(H)], 1))
        Z.append(X[k] @ W[k].T + bias[k])
        H = np.maximum(Z[k], 0)
    pooled = per_graph(H)
    y = pooled @ wo + bo
    if case["kind"] == "predict":
        return y
    r = y - target
    dy = 2 * r / ng
    dW, db = [None] * 3, [None] * 3
    dH = dy[node_graph][:, None] * wo
    for k in (2, 1, 0):
        dZ = np.where(Z[k] > 0, dH, 0)
        dW[k], db[k] = dZ.T @ X[k], dZ.sum(0)
        if k:
            dX = dZ @ W[k]
            dH = dX[:, :h] + around(dX[:, h:])
    g = np.concatenate([w.ravel() for w in dW] + db + [dy @ pooled, [dy.sum()]])
    # the first step of Adam: both moments start at zero
    return {"loss": float(np.mean(r * r)), "params": p - LEARNING_RATE * g / (np.abs(g) + 1e-8)}
