"""The rule by which improve.cu leaves a foreign label seen once out (csrc/gain_rule.cuh,
compiled for the host) against the oracle's gain model, with the p_in above 1 of communities
whose rows list an edge more than once or hold loops (CPU)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "gain_rule.cuh"
extern "C" int rule(int r, int ext, float lo, float hi) { return scd::seen_once_never_gains(r, ext, lo, hi); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "het-scd_gb300", "csrc"),
                    str(d / "rule.cpp"), "-o", str(d / "rule.so")], check=True)
    f = ctypes.CDLL(str(d / "rule.so")).rule
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_float, ctypes.c_float]
    return f


def _enclosure(x):
    """x rounded down and up to single precision."""
    f = np.float32(x)
    lo = f if float(f) <= x else np.nextafter(f, np.float32(-np.inf))
    hi = f if float(f) >= x else np.nextafter(f, np.float32(np.inf))
    return lo, hi


@pytest.mark.parametrize("alpha", [0.0, 0.25, 1.0, 1.5, 2.5, 7.5, 1e6])
def test_label_left_out_has_no_positive_gain(rule, alpha):
    rng = np.random.default_rng(int(alpha * 4))
    met, above = 0, 0
    for _ in range(40000):
        r = int(rng.choice([1, 2, 3, 4, 5, int(2 ** rng.uniform(0, 15.5)), 46339, 46340, 46341]))
        pairs = r * (r - 1) // 2
        inner = int(rng.choice([0, pairs - 1, pairs, pairs + 1, 2 * pairs, 3 * pairs, pairs + r, rng.integers(0, 4 * pairs + 1)]))
        p_in = (2.0 * inner) / (r * (r - 1.0)) if r > 1 else 0.0
        ext = int(rng.choice([0, 1, 2, r, r + 1, r + 2, int(2 ** rng.uniform(0, 30.9))]))
        deg = int(rng.choice([1, 2, int(2 ** rng.uniform(0, 18)), 46341, 46342, 200000]))   # products of deg wrap
        p_ext = float(rng.choice([0.0, 1e-12, 0.1, rng.uniform(0, 1), 1.0]))
        lo, hi = _enclosure(p_in)
        above += p_in > 1
        if not rule(r, ext, lo, hi):
            continue
        met += 1
        g = oracle.gain(r, 1, deg - 1, ext, p_in, p_ext, alpha)
        assert not g > 0.0, (r, ext, inner, deg, p_ext, alpha, g)
    assert met > 5000 and above > 5000


def test_full_communities_are_left_out(rule):
    """p_in of exactly 1, the densest that a converted graph has, is within the rule."""
    assert rule(3, 1, 1.0, 1.0) and rule(30, 31, 1.0, 1.0)
