"""Internal counts by the hash tables of the warp and CTA kernels where many ids of a table
start at few of its slots (the upper bits of the multiplicative hash agree), so that probes
walk long chains: internal out-lists of 33 to 64, to 1024 and of more entries, against the
oracle (the tolerance of tests/test_gpu_internal_lists.py)."""
import numpy as np
import pytest

import oracle as O
from test_gpu_internal_lists import _check, _graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,bits", [(45, 8), (65, 8), (66, 4), (300, 6), (1025, 5), (1400, 3)])
def test_long_chains(size, bits):
    n = 8 * size << bits
    ids = np.arange(n)
    same = ids[(ids * 0x9E3779B1 % 2 ** 32) >> (32 - bits) == 5]
    ids = np.concatenate([same[:size], np.setdiff1d(ids, same)[:size]])
    g, labels = _graph([size, size], 0.95, 50 * size, size, n, ids)
    valid = labels[labels != 0xffffffff]
    _check(g, labels, O.wcc(g, labels, np.bincount(valid)), False)
