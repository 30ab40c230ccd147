"""The row-bitmap triangle count around a dense core against the hash-table walks.

Cores of sizes around the padding of a bit row (4096), random and bipartite (where no
edge of the core lies on a triangle inside it, so every one of its flags comes from
the vertices outside), with outside vertices of long and of short out-lists; and the
skewed generators. Graph bytes (tri, tri_deg, the kept edges) must be equal."""
import numpy as np
import pytest

import scd_gb300
import scdgen

pytestmark = pytest.mark.gpu


def _core_graph(k, inner, fringe, degree, bipartite, seed):
    """k core vertices with `inner` random edges among them (across two halves if
    bipartite), `fringe` outside vertices with `degree` core neighbours each, a tenth of
    them with 20, and sparse edges between outside vertices; ids shuffled."""
    rng = np.random.default_rng(seed)
    half = k // 2
    a = rng.integers(0, half if bipartite else k, inner)
    b = rng.integers(half, k, inner) if bipartite else rng.integers(0, k, inner)
    f = np.arange(fringe)
    deg = np.where(f % 10 == 0, 20, degree)
    out = k + np.repeat(f, deg)
    # a bipartite core's outside vertices see both halves
    into = rng.integers(0, k, out.size)
    e = rng.integers(k, k + fringe, (2, 3 * fringe))
    u = np.concatenate([a, out, e[0]])
    v = np.concatenate([b, into, e[1]])
    keep = u != v
    ids = rng.permutation(k + fringe).astype(np.uint32)
    pairs = np.stack([ids[u[keep]], ids[v[keep]]], 1)
    return np.sort(pairs, axis=1)


GRAPHS = [(f"core{k}{'-bipartite' if bip else ''}", lambda k=k, bip=bip: _core_graph(
    k, 150 * k, 40000, 120, bip, k)) for k in (2000, 4095, 4096, 4097, 8193, 17000) for bip in (False, True)] + [
    ("core33000", lambda: _core_graph(33000, 3_000_000, 60000, 130, False, 1)),
    ("rmat19", lambda: scdgen.rmat(19, seed=5)),
    ("rmat18-dense", lambda: scdgen.rmat(18, 40, seed=6)),
    ("chunglu1m", lambda: scdgen.chunglu(1_000_000, 2.1, 5.0, 100000.0, 0.2, 10, 500, seed=7)),
]


@pytest.mark.parametrize("name,make", GRAPHS, ids=[g[0] for g in GRAPHS])
def test_bitmaps_equal_walks(name, make):
    pairs = make()
    got = []
    for flags in (0, scd_gb300.FLAG_TC_HASH):
        with scd_gb300.Engine(0, flags=flags) as eng:
            eng.convert_edges(pairs)
            got.append(eng.graph_bytes())
    assert got[0] == got[1]
