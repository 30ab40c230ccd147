"""Graphs of long out-lists fit the memory limit that their arrays and one pair of lists of their
vertices need: the lists that a score is counted from take nothing more.

Per vertex 100 bytes: the row offsets, triangles, degrees and out-degrees, the degree classes and
the counting buckets with an offset each, internal lengths, counts and degrees, two labellings and
the best, two sets of statistics, and the gains' records (24). Per edge 18: both directions of
the adjacency and of the internal lists, and the flags. Per row of more than 256 entries 8, and a
few words a graph and a block of 2048 vertices."""
import numpy as np
import pytest

import scd_gb300
import scdgen

pytestmark = pytest.mark.gpu
GRAPHS = {"2k": lambda: scdgen.planted(2000, 300.0, 0.1, 400, 600, seed=1),
          "20k": lambda: scdgen.planted(20000, 200.0, 0.1, 400, 600, seed=1), "rmat18": lambda: scdgen.rmat(18, 16, seed=1)}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_long_lists_fit(name):
    pairs = GRAPHS[name]()
    with scd_gb300.Engine(0) as eng:
        eng.convert_edges(pairs)
        n, m, _ = eng.graph_info()
        degree = np.diff(eng.graph_download()["indices"].astype(np.int64))
        want = eng.run()
        hubs = degree[degree > 4096]
        tables = (12 * 2 ** np.ceil(np.log2(2.0 * hubs)) + 8).sum()   # keys, counts and places of a hub's labels
        eng.set_memory_limit(int(100 * n + 18 * m + 8 * (degree > 256).sum() + 12 * (n // 2048 + 1) + tables + 400))
        eng.convert_edges(pairs)
        got = eng.run()
    assert list(got["wcc"]) == list(want["wcc"]) and got["iterations"] == want["iterations"]
