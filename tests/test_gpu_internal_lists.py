"""WCC with internal out-lists of every length class: communities whose members' internal
out-lists run from nothing to a few thousand entries, around the limits of the kernels
that count them (32, 64, 512 partners a chunk, 1024), against the oracle.

The triangles a vertex is given are its internal ones, so that a count off by one shows
as 1 / (its triangles) in one of n terms of at most 1: above 1e-11 here, while a sum of n
terms in another order differs by at most n * 2^-53 (1e-12)."""
import numpy as np
import pytest

import oracle as O
import scd_gb300

pytestmark = pytest.mark.gpu


def _graph(sizes, density, stray, seed, n=None, ids=None):
    rng = np.random.default_rng(seed)
    n = n or sum(sizes)
    ids = rng.permutation(n) if ids is None else ids
    labels = np.full(n, scd_gb300.INVALID_LABEL, np.uint32)
    tri, us, vs, at = np.ones(n, np.int32), [], [], 0
    for k, s in enumerate(sizes):
        me = np.sort(ids[at:at + s])   # members of any id, so that out-lists mix
        at += s
        a = np.triu(rng.random((s, s)) < density, 1)
        sym = (a | a.T).astype(np.float32)
        tri[me] = np.maximum((sym @ sym * sym).sum(1) / 2, 1).astype(np.int32)
        labels[me] = k
        i, j = np.nonzero(a)
        us.append(me[i])
        vs.append(me[j])
    e = rng.integers(0, n, (2, stray))   # edges between communities lengthen the whole lists
    e = e[:, labels[e[0]] != labels[e[1]]]
    u, v = np.concatenate(us + [e[0]]), np.concatenate(vs + [e[1]])
    key = np.unique(np.minimum(u, v) * n + np.maximum(u, v))
    a, b = key // n, key % n
    u, v = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.lexsort((v, u))
    indices = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))])
    return O.Graph(n, a.size, indices, v[order], tri, np.bincount(u, minlength=n)), labels


@pytest.mark.parametrize("sizes,density,stray", [
    ([3, 5, 9, 17, 33, 34, 35], 1.0, 400), ([33, 65, 66, 129, 258], 1.0, 9000), ([33, 65, 130, 600], 0.5, 40000),
    ([513, 514, 1025, 1026], 1.0, 0), ([70, 1100, 2300], 0.95, 60000), ([4, 20, 40] * 30, 0.7, 200000)])
@pytest.mark.parametrize("retuned", [False, True])
def test_internal_lists(sizes, density, stray, retuned):
    g, labels = _graph(sizes, density, stray, len(sizes))
    want = O.wcc(g, labels, np.bincount(labels))
    _check(g, labels, want, retuned)


@pytest.mark.parametrize("size", [3, 8, 9, 16, 17, 32, 33])
@pytest.mark.parametrize("bits", [5, 6, 7])
def test_entries_of_one_slot(size, bits):
    """A community whose ids all share the slot of the register groups' tables (the upper
    bits of the multiplicative hash), with every second vertex of another one among them."""
    n = 64 << bits
    ids = np.arange(n)
    same = ids[(ids * 0x9E3779B1 % 2 ** 32) >> (32 - bits) == 5]
    ids = np.concatenate([same[:size], np.setdiff1d(ids, same)[: 2 * size]])
    g, labels = _graph([size, 2 * size], 0.8, 300, size, n, ids)
    _check(g, labels, O.wcc(g, labels, np.bincount(labels[labels != scd_gb300.INVALID_LABEL])), False)


def _check(g, labels, want, retuned):
    with scd_gb300.Engine(0) as eng:
        eng.transfer_graph(g)
        if retuned:   # the lists follow the buckets of another split
            eng.autotune()
        eng.labels_to_device(labels)
        got = [eng.compute_wcc() for _ in range(2)]
    assert got[0] == got[1]
    assert abs(got[0] - want) <= g.n * 2.0 ** -53 * abs(want)


def test_rows_that_are_all_out_list():
    """A community stored one way (every entry in the row of its larger id): the out-lists hold
    all entries of the graph, twice what they hold of a symmetric one, and the score, which is
    made from the out-lists, is the same."""
    n = 3001   # an even number of entries
    u, v = np.tril_indices(n, -1)
    first = np.concatenate([[0], np.cumsum(np.arange(n))])
    tri, labels = np.full(n, (n - 1) * (n - 2), np.int32), np.zeros(n, np.uint32)
    one_way = O.Graph(n, u.size // 2, first, v, tri, np.full(n, n - 1))
    both = np.tile(np.arange(n), (n, 1))[~np.eye(n, dtype=bool)]
    symmetric = O.Graph(n, u.size, np.arange(n + 1) * (n - 1), both, tri, np.full(n, n - 1))
    got = []
    for g in (one_way, symmetric):
        with scd_gb300.Engine(0) as eng:
            eng.transfer_graph(g)
            eng.labels_to_device(labels)
            got.append(eng.compute_wcc())
    assert got[0] == got[1]
