"""The workloads the engine's speed is measured on, through its public entry points.

Every case is one of the calls a user of the engine makes:

  pipeline   an edge list to communities: convert_edges, run, labels_from_device
             (what `convert` followed by `main-gpu` does), the list in pinned host
             memory or on the device
  text       the `convert` tool: the edge-list text to the binary-format arrays
  graph      `main-gpu`: a graph in the binary format to communities
  iteration  one step of the loop of `main-gpu` on a resident graph, from labels
             the caller holds (labels in, labels and statistics out)
  wcc        the score and statistics of a caller's labelling of a resident graph
  batch      many graphs in one call of each stage
  served     graphs of mixed sizes joining a resident set, stepped until all left

Graphs come from the repository's seeded generators: planted partition (mean
degree 8 to 40, mixing 0.05 to 0.4), R-MAT (0.57/0.19/0.19/0.05, edge factor 8
to 16) and Chung-Lu with planted communities (skewed degrees), from the smallest
served request (1,000 vertices) to R-MAT scale 22 and 4 M-vertex Chung-Lu.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "het-scd_gb300"))

import scd_gb300  # noqa: E402
import scdgen  # noqa: E402

INVALID = scd_gb300.INVALID_LABEL


# ---- the cases -----------------------------------------------------------------

def _planted(n, degree=20.0, mu=0.1):
    return {"graph": "planted", "n": n, "degree": degree, "mu": mu}


def _rmat(scale, factor=16):
    return {"graph": "rmat", "scale": scale, "factor": factor}


def _chunglu(n, wmax=200000.0, mu=0.2):
    return {"graph": "chunglu", "n": n, "wmax": wmax, "mu": mu}


def listed():
    return [
        # the smallest request a serving process sees: launches, waits and allocations
        {"name": "pipeline-planted-1k", "call": "pipeline", "where": "host", **_planted(1000, 16.0)},
        # the plain CPU-and-GPU configuration (n = 10,000, mean internal degree 18, mixing 0.1)
        {"name": "pipeline-planted-10k", "call": "pipeline", "where": "host", **_planted(10000, 20.0)},
        # a large served request
        {"name": "pipeline-rmat-19", "call": "pipeline", "where": "host", **_rmat(19)},
        # the headline workload, edge list on the device
        {"name": "pipeline-rmat-22", "call": "pipeline", "where": "device", **_rmat(22)},
        # skewed degrees: hubs of tens of thousands of neighbours, long out-lists
        {"name": "pipeline-chunglu-4m", "call": "pipeline", "where": "device", **_chunglu(4000000)},
        # the `convert` tool on a text file's contents, arrays back to the host
        {"name": "text-planted-60k", "call": "text", **_planted(60001, 17.0, 0.25)},
        # `main-gpu` on a converted graph: upload, partition, loop
        {"name": "graph-planted-150k", "call": "graph", **_planted(150001, 24.0, 0.2)},
        # one iteration of `main-gpu`'s loop, the labels held by the caller
        {"name": "iteration-rmat-20", "call": "iteration", **_rmat(20)},
        # scoring a labelling from elsewhere (some vertices unlabelled)
        {"name": "wcc-chunglu-500k", "call": "wcc", **_chunglu(500000, 50000.0)},
        # planted graphs of the batched configuration (n log-uniform in [1,000, 200,000])
        {"name": "batch-96", "call": "batch", "count": 96, "nmax": 200000},
        # the served mix: small planted graphs and, one in eight, an R-MAT graph
        {"name": "served-32", "call": "served", "count": 32, "nmax": 50000, "scale": 17},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, most):
    kind = rng.choice(["planted", "planted", "rmat", "chunglu"])
    if kind == "planted":
        return _planted(_log_int(rng, 1000, min(most, 200000)), round(rng.uniform(8, 40), 2),
                        round(rng.uniform(0.05, 0.4), 3))
    if kind == "rmat":
        return _rmat(rng.randint(13, int(math.log2(most))), rng.randint(8, 16))
    return _chunglu(_log_int(rng, 20000, max(most, 20001)), round(math.exp(rng.uniform(math.log(1000), math.log(2e5)))),
                    round(rng.uniform(0.1, 0.4), 3))


def draw(rng):
    call = rng.choice(["pipeline", "pipeline", "pipeline", "text", "graph", "iteration", "wcc", "batch", "served"])
    if call == "batch":
        return {"call": call, "count": rng.randint(4, 96), "nmax": _log_int(rng, 4000, 200000)}
    if call == "served":
        return {"call": call, "count": rng.randint(4, 32), "nmax": _log_int(rng, 4000, 50000),
                "scale": rng.randint(13, 18)}
    if call == "pipeline":
        return {"call": call, "where": rng.choice(["host", "device"]), **_draw_graph(rng, 2 ** 21)}
    if call == "text":
        return {"call": call, **_draw_graph(rng, 2 ** 16)}
    return {"call": call, **_draw_graph(rng, 2 ** 20)}


# ---- inputs --------------------------------------------------------------------

def _edges(case, seed):
    kind = case["graph"]
    if kind == "planted":   # mean degree: internal + external
        return scdgen.planted(case["n"], case["degree"] * (1 - case["mu"]), case["mu"], 20, 100, seed=seed)
    if kind == "rmat":
        return scdgen.rmat(case["scale"], case["factor"], seed=seed)
    return scdgen.chunglu(case["n"], 2.1, 5.0, case["wmax"], case["mu"], 10, 500, seed=seed)


def _bounds(case):
    """Most vertices and records a graph of the case can have."""
    if case["graph"] == "planted":
        return case["n"], int(case["n"] * case["degree"] * 0.55) + 1000
    if case["graph"] == "rmat":
        return 2 ** case["scale"], 2 ** case["scale"] * case["factor"]
    return case["n"], case["n"] * 40


def _many(case, seed):
    """The edge lists of a batch (planted graphs of all densities) or of a served mix."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["count"]):
        n = int(np.exp(rng.uniform(np.log(1000), np.log(case["nmax"]))))
        if case["call"] == "batch":
            degree, mu = float(rng.uniform(8, 40)), float(rng.uniform(0.05, 0.4))
            out.append(scdgen.planted(n, degree * (1 - mu), mu, 20, 100, seed=seed * 1000 + i))
        elif i % 8 == 7:
            out.append(scdgen.rmat(case["scale"], 16, seed=seed * 1000 + i))
        else:
            out.append(scdgen.planted(n, 14.4, 0.1, 20, 100, seed=seed * 1000 + i))
    return out


def _pinned(arrays):
    """The arrays as views into one pinned host buffer (a receive buffer)."""
    buf = torch.empty(max(sum(a.size for a in arrays), 1), dtype=torch.int32, pin_memory=True)
    host, views, at = buf.numpy().view(np.uint32), [], 0
    for a in arrays:
        host[at:at + a.size] = a.reshape(-1)
        views.append(host[at:at + a.size].reshape(a.shape))
        at += a.size
    return buf, views


class _Graph:
    def __init__(self, d):
        self.__dict__.update(d)


def _text(pairs):
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "edges.txt")
        scdgen.write_text(path, pairs)
        with open(path, "rb") as f:
            return b"# undirected edges, one per line\n" + f.read()


def _converted(pairs):
    with scd_gb300.Engine(0) as eng:
        eng.convert_edges(pairs)
        return _Graph(eng.graph_download())


def _labelling(eng, seed):
    """A caller's labelling: the initial partition with a tenth of the vertices moved
    to a random community and a fiftieth unlabelled."""
    communities = eng.initial_partition()
    labels, rng = eng.current_labels(), np.random.default_rng(seed)
    r = rng.uniform(size=labels.size)
    labels = np.where(r < 0.1, rng.integers(0, max(communities, 1), labels.size), labels)
    return np.where(r > 0.98, INVALID, labels).astype(np.uint32)


def _result_buffers(case):
    """The buffers a caller keeps for its results, sized for any graph of the case:
    the entries beyond a result's own size stay as they are here."""
    call = case["call"]
    if call == "batch":
        return {"labels": torch.full((case["count"] * case["nmax"],), -1, dtype=torch.int32, pin_memory=True).numpy()}
    if call == "served":
        return {"labels": np.full(case["count"] * case["nmax"] + (case["count"] // 8 << case["scale"]), -1, np.int32)}
    n, records = _bounds(case)
    if call == "text":
        return {"indices": np.full(n + 1, -1, np.int32), "adj": np.full(2 * records, -1, np.int32),
                "tri": np.full(n, -1, np.int32), "tri_deg": np.full(n, -1, np.int32)}
    names = {"pipeline": ("labels",), "graph": ("labels",), "iteration": ("labels", "sizes", "ext", "int"),
             "wcc": ("sizes", "ext", "int")}[call]
    return {k: np.full(n, -1, np.int32) for k in names}


def _put(buffer, values):
    buffer[:values.size] = values.view(np.int32)
    return buffer


def prepare(case, seed):
    call = case["call"]
    state = {"call": call, "engine": scd_gb300.Engine(0), "out": _result_buffers(case)}
    if call in ("batch", "served"):
        state["buffer"], state["lists"] = _pinned(_many(case, seed))
        if call == "served":
            state["stage"] = scd_gb300.Engine(0)
            state["engine"].resident_init()
    elif call == "text":
        state["text"] = _text(_edges(case, seed))
    elif call == "pipeline":
        pairs = _edges(case, seed)
        if case["where"] == "host":
            state["buffer"], (state["pairs"],) = _pinned([pairs])
        else:
            state["device"] = torch.from_numpy(pairs.view(np.int32)).cuda()
    elif call == "graph":
        state["graph"] = _converted(_edges(case, seed))
    else:
        eng = state["engine"]
        eng.convert_edges(_edges(case, seed))
        state["labels"] = eng.initial_partition() and eng.current_labels() if call == "iteration" else \
            _labelling(eng, seed)
    torch.cuda.synchronize()
    return state


# ---- the calls -----------------------------------------------------------------

def _counts(r):
    return np.array([r["iterations"], r["initial_communities"], r["printed_communities"], r["distinct_communities"]],
                    np.int64)


TRACE = 64   # WCC values of a loop that are returned: initial, best, then one per iteration


def _trace(initial, best, per_iteration):
    out = np.zeros(TRACE)
    out[:2], k = (initial, best), min(len(per_iteration), TRACE - 2)
    out[2:2 + k] = per_iteration[:k]
    return out


def _communities(eng, out):
    r = eng.run()
    n, m, p_ext = eng.graph_info()
    return {"labels": _put(out["labels"], eng.labels_from_device()), "counts": _counts(r),
            "size": np.array([n, m], np.int64), "p_ext": p_ext, "wcc": _trace(r["initial_wcc"], r["best_wcc"], r["wcc"])}


def run(state):
    call, eng, out = state["call"], state["engine"], state["out"]
    if call == "pipeline":
        if "device" in state:
            eng.convert_edges(device_ptr=state["device"].data_ptr(), count=state["device"].shape[0])
        else:
            eng.convert_edges(state["pairs"])
        return _communities(eng, out)
    if call == "text":
        eng.convert_text(state["text"])
        d = eng.graph_download()
        return {k: _put(out[k], d[k]) for k in out}
    if call == "graph":
        eng.transfer_graph(state["graph"])
        return _communities(eng, out)
    if call == "iteration":
        eng.labels_to_device(state["labels"])
        w = eng.improve_labels()
        results = dict(zip(("sizes", "ext", "int"), eng.community_stats()), labels=eng.current_labels())
        return {"wcc": w, **{k: _put(out[k], results[k]) for k in out}}
    if call == "wcc":
        eng.labels_to_device(state["labels"])
        w = eng.compute_wcc()
        results = dict(zip(("sizes", "ext", "int"), eng.community_stats()))
        return {"wcc": w, **{k: _put(out[k], results[k]) for k in out}}
    if call == "batch":
        eng.batch_convert(state["lists"])
        results, _ = eng.batch_run()
        eng.batch_labels_all(out=out["labels"].view(np.uint32))
        return {"labels": out["labels"], "counts": np.concatenate([_counts(r) for r in results]),
                "wcc": np.array([[r["initial_wcc"], r["best_wcc"]] for r in results])}
    # served: four arrivals join, the set makes a step, and so on until every graph has left
    stage, waiting, held, done = state["stage"], list(state["lists"]), 0, {}
    order = []
    while waiting or held:
        if waiting:
            stage.batch_convert(waiting[:4])
            ids = eng.resident_add(stage)
            waiting, held, order = waiting[4:], held + len(ids), order + ids
        _, finished = eng.resident_step()
        if finished:
            for i, r, _, labels in eng.resident_take(cap=held, labels_cap=1 << 23):
                done[i] = (r, labels)
                held -= 1
    return {"labels": _put(out["labels"], np.concatenate([done[i][1] for i in order])),
            "counts": np.concatenate([_counts(done[i][0]) for i in order]),
            "wcc": np.array([[done[i][0]["initial_wcc"], done[i][0]["best_wcc"]] for i in order])}


# ---- what a pass cannot do without -----------------------------------------------

def _size(case):
    """(vertices, input records) of a case's graph, about."""
    if case["graph"] == "planted":
        return case["n"], int(case["n"] * case["degree"] / 2)
    if case["graph"] == "rmat":   # about a quarter of the ids keep an edge on a triangle
        return 2 ** case["scale"] // 3, int(2 ** case["scale"] * case["factor"] * 0.95)
    return case["n"], int(case["n"] * 13.5)


def work(case):
    """Bytes only (nothing here is arithmetic-bound): the inputs once and the outputs once."""
    call = case["call"]
    if call in ("batch", "served"):
        mean_n = (case["nmax"] - 1000) / math.log(case["nmax"] / 1000)
        n, e = mean_n * case["count"], mean_n * case["count"] * (12 if call == "batch" else 8)
        if call == "served":
            n += case["count"] // 8 * 2 ** case["scale"] // 3
            e += case["count"] // 8 * 2 ** case["scale"] * 15
        return {"bytes": 8 * e + 4 * n}
    n, e = _size(case)
    if call == "pipeline":
        return {"bytes": 8 * e + 4 * n}
    if call == "text":
        return {"bytes": 12 * e + 8 * e + 12 * n}
    if call == "graph":
        return {"bytes": 8 * e + 12 * n + 4 * n}
    if call == "iteration":
        return {"bytes": 8 * e + 12 * n + 8 * n}
    return {"bytes": 8 * e + 12 * n + 4 * n}


# ---- the same in plain numpy and torch ---------------------------------------------

# records beyond which the plain version takes too long: whole loops on planted
# graphs, on skewed ones, and single steps
MOST_PLANTED, MOST_SKEWED, MOST_STEP = 4_000_000, 4_500_000, 17_000_000


def _edge_triangles(n, src, dst):
    """Triangles on every edge src -> dst of an acyclic orientation."""
    dev = "cuda"
    src, dst = torch.as_tensor(src, device=dev), torch.as_tensor(dst, device=dev)
    keys, order = torch.sort(src * n + dst)
    src, dst = keys // n, keys % n
    beg = torch.searchsorted(src, torch.arange(n + 1, device=dev))
    length, count = beg[1:] - beg[:-1], torch.zeros_like(keys)
    step, walk = 1 << 16, length[dst]
    for lo in range(0, keys.numel(), step):
        e = torch.arange(lo, min(lo + step, keys.numel()), device=dev)
        w = walk[e]
        first = torch.cumsum(w, 0) - w
        own = torch.repeat_interleave(e, w)
        bc = beg[dst[own]] + torch.arange(own.numel(), device=dev) - torch.repeat_interleave(first, w)
        want = src[own] * n + dst[bc]
        ac = torch.searchsorted(keys, want).clamp(max=keys.numel() - 1)
        hit = keys[ac] == want
        for idx in (own[hit], bc[hit], ac[hit]):
            count.index_add_(0, idx, torch.ones_like(idx))
    back = torch.empty_like(count)
    back[order] = count
    return back.cpu().numpy()


def _plain_convert(pairs):
    flat = pairs.reshape(-1)
    ids, first, inverse = np.unique(flat, return_index=True, return_inverse=True)
    rank = np.empty(ids.size, np.int64)
    rank[np.argsort(first)] = np.arange(ids.size)
    a, b = rank[inverse].reshape(-1, 2).T
    n = ids.size
    key = np.unique((np.minimum(a, b) * n + np.maximum(a, b))[a != b])
    a, b = key // n, key % n
    deg = np.bincount(a, minlength=n) + np.bincount(b, minlength=n)
    up = (deg[b] > deg[a]) | ((deg[b] == deg[a]) & (b > a))
    cnt = _edge_triangles(n, np.where(up, a, b), np.where(up, b, a))
    tri = (np.bincount(a, cnt, n) + np.bincount(b, cnt, n)).astype(np.int64)
    a, b = a[cnt > 0], b[cnt > 0]
    tdeg = np.bincount(a, minlength=n) + np.bincount(b, minlength=n)
    order = np.lexsort((-np.arange(n), -tdeg))[:int((tdeg > 0).sum())]
    final = np.empty(n, np.int64)
    final[order] = np.arange(order.size)
    u, v = np.concatenate([final[a], final[b]]), np.concatenate([final[b], final[a]])
    s = np.lexsort((v, u))
    indices = np.concatenate([[0], np.cumsum(tdeg[order])])
    return {"n": order.size, "m": a.size, "indices": indices, "adj": v[s], "tri": tri[order], "tri_deg": tdeg[order]}


def _rows(g):
    deg = np.diff(np.asarray(g["indices"], np.int64))
    return deg, np.repeat(np.arange(g["n"]), deg), np.asarray(g["adj"], np.int64)


def _plain_partition(g):
    deg = np.diff(np.asarray(g["indices"], np.int64))
    cc = g["tri"] / (deg * (deg - 1.0))
    order = np.lexsort((np.arange(g["n"]), deg, cc))[::-1]
    labels, nxt, ind, adj = np.full(g["n"], -1, np.int64), 0, g["indices"], g["adj"]
    for p in order.tolist():
        if labels[p] < 0:
            row = adj[ind[p]:ind[p + 1]]
            labels[row[labels[row] < 0]] = nxt
            labels[p] = nxt
            nxt += 1
    return labels, nxt


def _plain_stats(g, labels, k):
    deg, src, adj = _rows(g)
    ok = labels[src] >= 0
    same = ok & (labels[src] == labels[adj])
    return (np.bincount(labels[labels >= 0], minlength=k), np.bincount(labels[src[ok & ~same]], minlength=k),
            np.bincount(labels[src[same]], minlength=k))


def _wrap(x):
    return x.astype(np.int32).astype(np.float64)


def _plain_gain(r, din, dout, cout, pin, pe):
    with np.errstate(all="ignore"):
        t = np.where(r > 0, (cout - din) / r.astype(float), 0.0)
        dp = _wrap(din * (din - 1)) * pin
        den = (dp + _wrap(dout * (dout - 1)) * pe + _wrap(dout * din) * pe) * ((din + dout) + 1.0 * (r - 1 - din))
        ga = np.where(den != 0, dp * (din + dout) / den, 0.0)
        rr, q = _wrap((r - 1) * (r - 2)) * pin * pin * pin, (r - 1) * pin
        two = (2 * (din - 1)) * pin
        tr, tt = t * (r - 1) * pin * pe, t * (t - 1) * pe
        den = (rr + two + tr + tt + dout * pe) * (q + 1 + t + 1.0 * (r - q - 1))
        gb = np.where(den != 0, two * (q + 1 + t) / den, 0.0)
        den = (rr + tt + tr) * (q + t + 1.0 * (r - q)) * (q + t + 1.0 * (r - q - 1))
        gc = np.where((den != 0) & (r + t > 0) & (r - 1 + t > 0), -rr * (q + t) * 1.0 / den, 0.0)
    return ga + din * gb + (r - din) * gc


def _plain_improve(g, pe, labels, stats):
    deg, src, adj = _rows(g)
    k = int(stats[0].size) + 1
    ok = labels[adj] >= 0
    key, f = np.unique(src[ok] * k + labels[adj[ok]], return_counts=True)
    p, l = key // k, key % k
    own = l == labels[p]
    size = stats[0][l] - own
    ext = stats[1][l] + np.where(own, 2 * f - deg[p], 0)
    internal = stats[2][l] // 2 - np.where(own, f, 0)
    with np.errstate(all="ignore"):
        pin = np.where(size > 1, 2.0 * internal / (size * (size - 1.0)), 0.0)
    gain = _plain_gain(size, f, deg[p] - f, ext, pin, pe)
    remove, best, where = np.zeros(g["n"]), np.zeros(g["n"]), np.zeros(g["n"], np.int64)
    remove[p[own]] = -gain[own]
    order = np.lexsort((l, -gain, p))
    first = order[np.unique(p[order], return_index=True)[1]]
    first = first[gain[first] > 0]
    best[p[first]], where[p[first]] = gain[first], l[first]
    insert = best + remove
    return np.where((insert > remove) & (insert > 0), where, np.where(remove > 0, -1, labels))


def _plain_wcc(g, labels, sizes):
    _, src, adj = _rows(g)
    keep = (src > adj) & (labels[src] >= 0) & (labels[src] == labels[adj])
    a, b, n = src[keep], adj[keep], g["n"]
    cnt = _edge_triangles(n, a, b) if a.size else np.zeros(0, np.int64)
    it = np.bincount(a, cnt, n) + np.bincount(b, cnt, n)
    itd = np.bincount(a[cnt > 0], minlength=n) + np.bincount(b[cnt > 0], minlength=n)
    size = np.where(labels >= 0, np.append(sizes, 0)[labels], 0)
    td = np.asarray(g["tri_deg"], np.int64)
    with np.errstate(all="ignore"):
        term = _wrap((it * td).astype(np.int64)) / (np.asarray(g["tri"], np.float64) * (td + 1.0 * (size - 1 - itd)))
    term = np.where((size > 2) & (td > 0) & np.isfinite(term), term, 0.0)
    return math.fsum(term.tolist()) / n if n else 0.0


def _plain_p_ext(g):
    deg = np.diff(np.asarray(g["indices"], np.int64))
    with np.errstate(all="ignore"):
        term = np.where(deg > 1, g["tri"] / (deg * (deg - 1.0)), 0.0)
    return float(math.fsum(term.tolist()) / g["n"])


def _plain_loop(g):
    pe = _plain_p_ext(g)
    labels, k = _plain_partition(g)
    stats = _plain_stats(g, labels, k)
    best = first = _plain_wcc(g, labels, stats[0])
    trace = []
    while True:
        labels = _plain_improve(g, pe, labels, stats)
        stats = _plain_stats(g, labels, k)
        trace.append(_plain_wcc(g, labels, stats[0]))
        if trace[-1] < best * 1.01:
            return pe, first, best, trace
        best = trace[-1]


def exact(case, seed):
    call = case["call"]
    if call in ("batch", "served"):
        lists = _many(case, seed)
        if sum(p.shape[0] for p in lists) > MOST_PLANTED:
            return None
        return {"labels": None, "counts": None,
                "wcc": np.array([_plain_loop(_plain_convert(p))[1:3] for p in lists])}
    most = MOST_STEP if call in ("iteration", "wcc") else MOST_PLANTED if case["graph"] == "planted" else MOST_SKEWED
    if call == "text" or _size(case)[1] > most:
        return None   # (text: whole numbers only)
    if call in ("pipeline", "graph"):
        pe, first, best, trace = _plain_loop(_plain_convert(_edges(case, seed)))
        return {"labels": None, "counts": None, "size": None, "p_ext": pe, "wcc": _trace(first, best, trace)}
    # the resident graph and the caller's labels are inputs of these calls
    state = prepare(case, seed)
    g, lab = state["engine"].graph_download(), state["labels"].astype(np.int64)
    labels = np.where(lab == INVALID, -1, lab)
    if call == "iteration":
        k = int(labels.max()) + 1
        labels = _plain_improve(g, _plain_p_ext(g), labels, _plain_stats(g, labels, k))
        return {"labels": None, "sizes": None, "ext": None, "int": None,
                "wcc": _plain_wcc(g, labels, np.bincount(labels[labels >= 0], minlength=k))}
    return {"sizes": None, "ext": None, "int": None, "wcc": _plain_wcc(g, labels, np.bincount(labels[labels >= 0]))}
