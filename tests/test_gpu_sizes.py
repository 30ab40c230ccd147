"""Whole conversions and partitions at the sizes where the scans and list builders
change form (one tile, one CTA, two launches, several tiles per CTA), against the
oracle.  A strip of triangles (edges i - i+1 and i - i+2) keeps every vertex, so
the vertex count is the length of most scans of a run; everything is equal bit
for bit."""
import numpy as np
import pytest

import oracle
import scd_gb300

pytestmark = pytest.mark.gpu


def _strip(n, seed):
    """A triangle strip of n vertices under shuffled ids, records shuffled."""
    rng = np.random.default_rng(seed)
    ids = rng.permutation(n).astype(np.uint32)
    i = np.arange(n)
    a = np.concatenate([ids[i[:-1]], ids[i[:-2]]])
    b = np.concatenate([ids[i[1:]], ids[i[2:]]])
    pairs = np.stack([np.minimum(a, b), np.maximum(a, b)], 1)
    return pairs[rng.permutation(len(pairs))]


# one scan tile: n + 1 <= 2048; one CTA: n + 1 <= 16384; more than one tile per CTA: n >= 2490368
@pytest.mark.parametrize("n", [3, 2046, 2047, 2048, 2049, 4096, 16383, 16384, 16385, 100000, 2490367, 2490400])
def test_strip_of_every_scan_form(n):
    pairs = _strip(n, n)
    ref, _ = oracle.convert(pairs)
    assert ref.n == n
    with scd_gb300.Engine(0) as eng:
        eng.convert_edges(pairs)
        assert eng.graph_bytes() == ref.to_bytes()
        labels, nc = oracle.initial_partition(ref)
        assert eng.initial_partition() == nc
        assert np.array_equal(eng.current_labels(), labels)
        sizes, ext, internal = oracle.collect_stats(ref, labels, nc)
        for got, want in zip(eng.community_stats(), (sizes, ext, internal)):
            assert np.array_equal(got, want)
