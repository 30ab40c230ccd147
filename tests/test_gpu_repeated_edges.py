"""One improvement of graphs whose rows list edges more than once or hold loops (a transferred
graph's may): communities denser than complete ones (p_in > 1), each seen once by vertices of
every degree class, against the oracle's labels."""
import numpy as np
import pytest

import oracle as O
import scd_gb300

pytestmark = pytest.mark.gpu


def _graph(degree, times, loops, shared, seed):
    """Communities of 3 to 5 vertices, complete, every inner edge listed `times` times, a loop
    at `loops` of the members of each; unlabelled probes of `degree` neighbours see one member
    of each of as many communities, and `shared` probes see the same communities."""
    rng = np.random.default_rng(seed)
    count, probes = degree, max(shared, 1)
    sizes = rng.integers(3, 6, count)
    first = probes + np.concatenate([[0], np.cumsum(sizes)])
    n = int(first[-1])
    labels = np.full(n, scd_gb300.INVALID_LABEL, np.uint32)
    labels[probes:] = np.repeat(np.arange(count), sizes)
    u, v = [], []
    for k in range(count):
        me = np.arange(first[k], first[k + 1])
        a, b = np.triu_indices(me.size, 1)
        u.append(np.repeat(me[a], times))
        v.append(np.repeat(me[b], times))
    for p in range(probes):
        u.append(np.full(count, p))
        v.append(first[:-1] + rng.integers(0, 3, count))
    u, v = np.concatenate(u), np.concatenate(v)
    loop = np.concatenate([first[k] + np.arange(loops) for k in range(count)]) if loops else np.zeros(0, np.int64)
    if loop.size % 2:   # the binary format holds 2m entries
        loop = loop[:-1]
    ids = rng.permutation(n)   # rows of any id order
    src = ids[np.concatenate([u, v, loop])]
    dst = ids[np.concatenate([v, u, loop])]
    order = np.lexsort((dst, src))
    moved = np.empty(n, np.uint32)
    moved[ids] = labels
    tri = rng.integers(1, 5, n)
    indices = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))])
    return O.Graph(n, src.size // 2, indices, dst[order], tri, np.ones(n)), moved


@pytest.mark.parametrize("alpha", [0.25, 1.0, 2.5, 7.5])
@pytest.mark.parametrize("degree", [2, 15, 31, 40, 256, 300, 1500, 3000, 5000])
@pytest.mark.parametrize("times,loops,shared", [(1, 2, 1), (2, 0, 1), (2, 1, 9), (3, 0, 4)])
def test_improve(degree, times, loops, shared, alpha):
    g, labels = _graph(degree, times, loops, shared, degree)
    nc = int(labels[labels != scd_gb300.INVALID_LABEL].max()) + 1
    with scd_gb300.Engine(0) as eng:
        eng.transfer_graph(g, alpha)
        eng.labels_to_device(labels)
        p_ext = eng.graph_info()[2]
        eng.improve_labels()
        got = eng.current_labels()
    want = O.improve(g, p_ext, labels, *O.collect_stats(g, labels, nc), alpha=alpha)
    assert np.array_equal(got, want)
