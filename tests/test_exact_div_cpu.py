"""The integer division of the WCC terms (csrc/exact_div.cuh, compiled for the host) against
the FP64 division: equal bits over the ranges it is called with, at random operands and at
quotients that lie on, or one part beside, the middle of two doubles."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <random>
#include "exact_div.cuh"
static uint64_t n = 0, bad = 0;
static void check(uint64_t a, uint64_t b) {
    if (a < 1 || a >> 32 || b < 1 || b >> 53) return;
    n++;
    const double want = (double)a / (double)b, got = scd::exact_div((uint32_t)a, b);
    if (std::memcmp(&want, &got, 8) && bad++ < 5) std::printf("%llu / %llu\n", (unsigned long long)a, (unsigned long long)b);
}
int main() {
    std::mt19937_64 r(1);
    for (int i = 0; i < 4000000; i++) {
        const uint64_t a = (r() | 1ull << 63) >> (32 + r() % 32), b = (r() | 1ull << 63) >> (11 + r() % 53);
        check(a, b);
        // b just below, at and above the quotients a / 2^k and a 2^k, and equal leading bits
        for (int d = -2; d <= 2; d++) {
            check(a, (a << (r() % 22)) + d);
            check(a, b + d);
            check((b >> 21) + d, b);
        }
    }
    for (uint64_t a = 1; a < 2000; a++)
        for (uint64_t b = 1; b < 2000; b++) check(a, b);
    // quotients near the middle of two doubles: a 2^k = (2 m + 1) b / 2 + e for small e
    for (int i = 0; i < 2000000; i++) {
        const uint64_t b = (r() | 1ull << 63) >> (11 + r() % 33) | 1;
        const unsigned __int128 mid = (unsigned __int128)((r() >> 11 | 1ull << 52) * 2 + 1) * b;
        const uint64_t a = (uint64_t)(mid >> (64 + r() % 42));
        for (int d = -1; d <= 2; d++) check((a & 0xffffffffull) + d, b);
    }
    const uint64_t edge[] = {1, 2, 3, (1ull << 31) - 1, 1ull << 31, (1ull << 32) - 1, 1ull << 32, (1ull << 52) - 1, 1ull << 52,
                             (1ull << 53) - 1};
    for (uint64_t a : edge)
        for (uint64_t b : edge) check(a, b);
    std::printf("%llu checked, %llu differ\n", (unsigned long long)n, (unsigned long long)bad);
    return bad != 0;
}
"""


def test_equals_fp64_division(tmp_path):
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "het-scd_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout.split()[0]) > 10_000_000
