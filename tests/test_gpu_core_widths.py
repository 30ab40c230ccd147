"""The row-bitmap triangle count with a dense core of every row width, on either side of each
padding step and of the largest core, against the hash-table walks.

A core whose members all have the same degree, above every other vertex's, is chosen whole or
not at all, so the phase timer of the bitmap count says that exactly `k` members were taken.
Members are neighbours within a distance on a ring: at every distance, or at odd ones only,
where for an even `k` no triangle lies inside the core and every flag of its edges comes from
the vertices outside, each of which sees a hundred consecutive members."""
import numpy as np
import pytest

import scd_gb300

pytestmark = pytest.mark.gpu
MOST = 32768   # members


def _ring(k, odd, seed):
    degree = max(300, k // 50)   # enough that the bitmaps are worth it
    distance = np.arange(1, degree // 2 + 1)
    if odd:
        distance = 2 * distance - 1
    a = np.arange(k)
    u, v = [np.tile(a, distance.size)], [(a[None, :] + distance[:, None]).reshape(-1) % k]
    u.append(k + a // 100)   # outside
    v.append(a)
    # in any order: ids are numbered as they appear, and equal degrees are ordered by them
    pairs = np.stack([np.concatenate(u), np.concatenate(v)], 1).astype(np.uint32)
    return pairs[np.random.default_rng(seed).permutation(pairs.shape[0])]


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("k", [4095, 4096, 4097, 8192, 8193, 12289, 16384, 16385, 20481, 24577, 28672, 28673, MOST, MOST + 1])
def test_every_row_width(k, odd):
    pairs = _ring(k, odd, k)
    got = []
    for flags, cores in ((0, k <= MOST), (scd_gb300.FLAG_TC_HASH, 0)):
        with scd_gb300.Engine(0, flags=flags | scd_gb300.FLAG_PROFILE) as eng:
            eng.convert_edges(pairs)
            assert eng.profile("tc_dense")[1] == cores
            got.append(eng.graph_bytes())
    assert got[0] == got[1]
