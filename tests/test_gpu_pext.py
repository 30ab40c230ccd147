"""The index-ordered p_ext sum against the same additions in Python, one by one.

The kernel adds in integers of the running sum's unit and falls back to a real
addition at ties, at doublings of the sum and at terms it cannot round in
integers; the sequences below hold many of each.  Bit for bit.
"""
import numpy as np
import pytest

import scd_gb300

pytestmark = pytest.mark.gpu


class _Rows:
    """A graph of given degrees and tri (its rows are never walked by p_ext)."""

    def __init__(self, deg, tri):
        deg = np.minimum(np.asarray(deg, np.int64), len(deg))
        self.n = len(deg)
        if deg.sum() & 1:
            deg[-1] += 1 if deg[-1] < self.n else -1
        self.indices = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
        self.m = int(deg.sum()) // 2
        self.adj = np.concatenate([np.arange(d) for d in deg] or [[]]).astype(np.uint32)
        self.tri = np.asarray(tri, np.int32)
        self.tri_deg = deg.astype(np.int32)
        self.deg = deg


def _sequence(kind, n):
    rng = np.random.default_rng(n)
    deg = rng.integers(2, min(n, 40) + 1, n) if n > 1 else np.zeros(n, int)
    tri = (2.0 ** rng.uniform(0, 30.9, n)).astype(np.int64)
    if kind == "small":      # coefficients below 1, as converted graphs have them
        tri = (rng.uniform(0, 1, n) * deg * np.maximum(deg - 1, 0)).astype(np.int64)
    if kind == "zeros":      # leading zeros over more than one tile, and single ones after
        tri[: n * 3 // 4] = 0
        tri[rng.uniform(size=n) < 0.3] = 0
    if kind == "growing":    # the terms stay close to the sum: ties and doublings
        tri = np.minimum(2.0 ** (np.arange(n) * 30.9 / n), 2 ** 31 - 1).astype(np.int64)
        deg[:] = 2 if n > 1 else 0
        deg[::3] = min(n, 4) if n > 1 else 0
    if kind == "negative":   # the sum falls below zero and comes back
        tri = np.where(rng.uniform(size=n) < 0.5, -tri, tri)
    return deg, tri


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("wide", "small", "growing") for n in
                                    (1, 2, 31, 32, 33, 1000, 8191, 8224, 8225, 30000)] +
                         [("zeros", 40), ("zeros", 40000), ("negative", 700)])
def test_pext_equals_additions_one_by_one(kind, n):
    g = _Rows(*_sequence(kind, n))
    s = 0.0
    for d, t in zip(g.deg.tolist(), g.tri.tolist()):
        s += t / (d * (d - 1.0)) if d > 1 else 0.0
    with scd_gb300.Engine(0) as eng:
        eng.transfer_graph(g)
        assert eng.graph_info()[2] == s / n
