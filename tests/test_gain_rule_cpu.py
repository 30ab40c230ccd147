"""A foreign label seen once has no positive gain where improve.cu leaves its interval
out (never_gains): the rule restated, against the oracle's gain model (CPU)."""
import numpy as np
import pytest

import oracle


def _never_gains(r, ext, p_in):
    return 1 <= r <= 46340 and ext >= 1 and p_in >= 0 and (r <= 2 or ext == 1 or ext - 1 >= r)


@pytest.mark.parametrize("alpha", [0.0, 0.25, 1.0, 7.5])
def test_label_seen_once_never_gains(alpha):
    rng = np.random.default_rng(int(alpha * 4))
    met = 0
    for _ in range(40000):
        r = int(rng.choice([1, 2, 3, int(2 ** rng.uniform(0, 15.5)), 46339, 46340]))
        pairs = r * (r - 1) // 2
        inner = int(rng.choice([0, pairs, rng.integers(0, pairs + 1), max(pairs - 1, 0)]))
        p_in = (2.0 * inner) / (r * (r - 1.0)) if r > 1 else 0.0
        ext = int(rng.choice([1, 2, r, r + 1, r + 2, int(2 ** rng.uniform(0, 30.9))]))
        deg = int(rng.choice([1, 2, int(2 ** rng.uniform(0, 18)), 46341, 46342, 200000]))   # products of deg wrap
        p_ext = float(rng.choice([0.0, 1e-12, rng.uniform(0, 1), 1.0]))
        if not _never_gains(r, ext, p_in):
            continue
        met += 1
        g = oracle.gain(r, 1, deg - 1, ext, p_in, p_ext, alpha)
        assert g <= 0.0, (r, ext, inner, deg, p_ext, alpha, g)
    assert met > 10000
