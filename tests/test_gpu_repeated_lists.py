"""The score of transferred graphs whose rows list entries twice, where a vertex's whole
out-list is longer than the register groups' and its internal one is not: every entry of a
partner's internal out-list counts, as the kernels for long lists count it, against plain loops.

The score is a sum of n terms of at most a few units each, so sums in another order differ by
at most n * 2^-53 of it."""
import numpy as np
import pytest

import oracle as O
import scd_gb300

pytestmark = pytest.mark.gpu


def _graph(members, centres, inner, stray, seed):
    """One community: `members` vertices, a hub above them that lists each of them twice, and
    `centres` vertices above the hub with `inner` members, the hub and, outside the community,
    `stray` unlabelled vertices in their out-lists."""
    rng = np.random.default_rng(seed)
    hub = members + stray
    n = hub + 1 + centres
    u, v = [np.repeat(np.full(members, hub), 2)], [np.repeat(np.arange(members), 2)]
    for a in range(hub + 1, n):
        mine = np.concatenate([rng.choice(members, inner, replace=False), members + np.arange(stray), [hub]])
        u.append(np.full(mine.size, a))
        v.append(mine)
    u, v = np.concatenate(u), np.concatenate(v)
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    labels = np.zeros(n, np.uint32)
    labels[members:hub] = scd_gb300.INVALID_LABEL
    deg = np.bincount(src, minlength=n)
    indices = np.concatenate([[0], np.cumsum(deg)])
    return O.Graph(n, src.size // 2, indices, dst[order], np.full(n, 2 * members), np.full(n, 500)), labels


def _score(g, labels):
    """Every centre a, entry b and entry c of b's list: a triangle if a lists c (no centre here
    lists an entry twice); the edges with a triangle by their place."""
    rows = [[int(w) for w in g.adj[g.indices[v]:g.indices[v + 1]] if w < v and labels[w] == labels[v]]
            if labels[v] != scd_gb300.INVALID_LABEL else [] for v in range(g.n)]
    count, found = np.zeros(g.n, np.int64), set()
    for a in range(g.n):
        place = {w: i for i, w in enumerate(rows[a])}
        for i, b in enumerate(rows[a]):
            for j, c in enumerate(rows[b]):
                if c in place:
                    count[[a, b, c]] += 1
                    found |= {(a, i), (b, j), (a, place[c])}
    degree = np.zeros(g.n, np.int64)
    for v, i in found:
        degree[v] += 1
        degree[rows[v][i]] += 1
    size = int((labels == 0).sum())
    on = labels == 0
    term = 2.0 * count[on] * g.tri_deg[on] / (g.tri[on] * (g.tri_deg[on] + (size - 1.0 - degree[on])))
    return float(term.sum() / g.n)


CASES = [(40, 50, 3, 40, 1), (40, 50, 8, 70, 2), (140, 9, 31, 10, 3), (140, 30, 30, 300, 4), (40, 9, 1, 1200, 5),
         (40, 3, 4, 9000, 6)]


@pytest.mark.parametrize("shape", CASES)
def test_every_entry_counts(shape):
    g, labels = _graph(*shape)
    want = _score(g, labels)
    with scd_gb300.Engine(0) as eng:
        eng.transfer_graph(g)
        eng.labels_to_device(labels)
        got = eng.compute_wcc()
    assert abs(got - want) <= g.n * 2.0 ** -53 * abs(want)


def test_beside_other_graphs_of_a_set():
    """A set holds such graphs and one of distinct rows: the loop of each as on its own."""
    graphs = [_graph(40, 50, 8, 70, 7)[0], _graph(140, 30, 30, 300, 8)[0]]
    distinct = _graph(40, 50, 8, 70, 9)[0]
    row = np.repeat(np.arange(distinct.n), np.diff(distinct.indices.astype(np.int64)))
    keep = np.ones(distinct.adj.size, bool)
    keep[1:] = (distinct.adj[1:] != distinct.adj[:-1]) | (row[1:] != row[:-1])
    indices = np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=distinct.n))])
    graphs.append(O.Graph(distinct.n, keep.sum() // 2, indices, distinct.adj[keep], distinct.tri, distinct.tri_deg))
    alone = []
    with scd_gb300.Engine(0) as eng:
        for g in graphs:
            eng.transfer_graph(g)
            alone.append((eng.run(), eng.labels_from_device()))
    with scd_gb300.Engine(0) as s, scd_gb300.Engine(0) as stage:
        s.resident_init()
        ids = []
        for g in graphs:
            stage.transfer_graph(g)
            ids += s.resident_add(stage)
        left, done = len(ids), {}
        while left:
            s.resident_step()
            for i, r, _, lab in s.resident_take():
                done[i] = (r, lab)
                left -= 1
    for i, (r, lab) in zip(ids, alone):
        assert done[i][0]["iterations"] == r["iterations"] and done[i][0]["best_wcc"] == r["best_wcc"]
        assert np.array_equal(done[i][1], lab)
