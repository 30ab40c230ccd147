"""Rows at the lengths and row counts where the row sorts change form (513 and 4097
entries; a bitmap of the row numbers in one range, in several, and the radix sort
beyond), repeated records included, against the oracle's convert bit for bit."""
import numpy as np
import pytest

import oracle
import scd_gb300

pytestmark = pytest.mark.gpu


def _hubs(lengths, repeats, extra, seed):
    """A hub of each length whose neighbours form a path (so every edge is on a
    triangle), `repeats` of its records twice, and `extra` single edges elsewhere."""
    rng = np.random.default_rng(seed)
    u, v, at = [], [], 0
    for length in lengths:
        hub, nb = at, at + 1 + np.arange(length)
        at += length + 1
        u += [np.full(length, hub), nb[:-1], np.full(repeats, hub)]
        v += [nb, nb[1:], rng.choice(nb, repeats)]
    u, v = np.concatenate(u), np.concatenate(v)
    ids = rng.permutation(at).astype(np.uint32)
    pairs = np.stack([np.minimum(ids[u], ids[v]), np.maximum(ids[u], ids[v])], 1).astype(np.uint32)
    pairs = pairs[rng.permutation(len(pairs))]
    if extra:
        single = (at + np.arange(2 * extra, dtype=np.uint32)).reshape(-1, 2)
        pairs = np.concatenate([pairs[: len(pairs) // 2], single, pairs[len(pairs) // 2:]])
    return pairs


RANGE = 54 * 1024 * 32   # row numbers of one bitmap range


@pytest.mark.parametrize("lengths,repeats,extra", [
    (list(range(1, 40)), 2, 0),
    (list(range(1, 40)) * 800, 2, 1000),   # 32 rows a warp
    ([31, 32, 33, 64, 65, 128, 129, 256, 257], 7, 0),
    ([511, 512, 513, 1023, 1024, 1025, 2048, 4095], 0, 0),
    ([505, 1000, 4089, 4096], 7, 0),
    ([4096, 4097, 4098, 5000, 20000], 9, 0),
    ([70000], 300, 0),
    ([6000, 9000], 11, RANGE // 2 - 7600),   # one range, just
    ([6000, 9000], 11, RANGE // 2),          # two
    ([6000, 9000], 11, 16 * RANGE // 2 + 5000),   # more than the bitmap takes
], ids=["short", "short-many", "warp", "radix", "radix-repeats", "bitmap", "long", "one-range", "two-ranges", "beyond"])
def test_rows_of_every_form(lengths, repeats, extra):
    pairs = _hubs(lengths, repeats, extra, 3)
    ref, _ = oracle.convert(pairs)
    with scd_gb300.Engine(0) as eng:
        eng.convert_edges(pairs)
        assert eng.graph_bytes() == ref.to_bytes()
