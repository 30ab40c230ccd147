"""Community statistics of transferred graphs of every form that is accepted, against
numpy counts over whole rows: symmetric ones (counted from the out-lists), and ones
with a one-way entry, a loop or a hub whose whole row is its out-list (counted from
the rows)."""
import numpy as np
import pytest

import scd_gb300

pytestmark = pytest.mark.gpu


class _Csr:
    def __init__(self, n, u, v):
        order = np.lexsort((v, u))
        u, v = u[order], v[order]
        if u.size % 2:   # the binary format holds 2m entries
            u, v = u[:-1], v[:-1]
        self.n, self.m = n, u.size // 2
        self.src, self.adj = u, v.astype(np.uint32)
        self.indices = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.uint32)
        self.tri = np.ones(n, np.int32)
        self.tri_deg = np.ones(n, np.int32)


def _graph(kind, n):
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, n, (2, 6 * n))
    keep = a != b
    key = np.unique(np.minimum(a, b)[keep] * n + np.maximum(a, b)[keep])
    a, b = key // n, key % n
    if kind == "hub":   # the largest id neighbours everyone: its out-list is its whole row
        a, b = np.concatenate([a, np.arange(n - 1)]), np.concatenate([b, np.full(n - 1, n - 1)])
        key = np.unique(a * n + b)
        a, b = key // n, key % n
    u, v = np.concatenate([a, b]), np.concatenate([b, a])
    if kind == "repeated":   # an edge listed twice in both of its rows
        u, v = np.concatenate([u, a[:5], b[:5]]), np.concatenate([v, b[:5], a[:5]])
    if kind == "one-way":
        u, v = u[:-2], v[:-2]
    if kind == "loop":
        u, v = np.concatenate([u, [3, 7]]), np.concatenate([v, [3, 7]])
    return _Csr(n, u, v)


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("symmetric", "repeated", "one-way", "loop") for n in
                                    (9, 129, 5000, 40000, 400000)] + [("hub", 9000)])
def test_statistics(kind, n):
    g = _graph(kind, n)
    rng = np.random.default_rng(1)
    k = max(n // 7, 2)
    labels = rng.integers(0, k, n).astype(np.uint32)
    labels[rng.uniform(size=n) < 0.1] = scd_gb300.INVALID_LABEL
    labels[0] = k - 1
    ok = labels[g.src] != scd_gb300.INVALID_LABEL
    same = ok & (labels[g.src] == labels[g.adj])
    valid = labels[labels != scd_gb300.INVALID_LABEL]
    want = (np.bincount(valid, minlength=k), np.bincount(labels[g.src[ok & ~same]], minlength=k),
            np.bincount(labels[g.src[same]], minlength=k))
    with scd_gb300.Engine(0) as eng:
        eng.transfer_graph(g)
        eng.labels_to_device(labels)
        for got, w in zip(eng.community_stats(), want):
            assert np.array_equal(got, w)
