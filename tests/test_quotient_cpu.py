"""The quotient that a PageRank step uses in place of a division
(lpma_gb300/csrc/quotient.h), on the CPU against the division itself: every
out-degree that a key can have, ranks over the exponents that occur, ranks next
to multiples of the degree and the largest ones.  Fused multiply-adds are exact
in the same way on host and device."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdint>
#include <initializer_list>
#include <limits>
#include "quotient.h"
using lpma::quotient;
static uint64_t x = 88172645463325252ull;
static uint64_t rnd() { return x ^= x << 13, x ^= x >> 7, x ^= x << 17; }
static long wrong = 0;
static void check(double r, double n) {
    const double a = quotient(r, n, 1.0 / n), b = r / n;
    if (a != b && ++wrong < 5) std::printf("%a / %a: %a, not %a\n", r, n, a, b);
}
int main() {
    for (uint32_t n = 1; n <= 1u << 22; n++) {
        for (int t = 0; t < 6; t++) check(std::ldexp(1.0 + (double)(rnd() >> 12) * 0x1p-52, -(int)(rnd() % 60)), n);
        // next to a multiple of n, and of n / 2
        const double m = (double)n * (double)(rnd() >> 33), e = 1.0 + 0x1p-52;
        check(m, n), check(m * e, n), check(m / e, n), check((m + n * 0.5) * e, n), check(0.0, n);
    }
    for (double n : {1.0, 2.0, 3.0, 7.0, 4194304.0}) {
        check(-1.0, n), check(-0.3, n);
        check(std::numeric_limits<double>::max(), n), check(-std::numeric_limits<double>::max(), n);
    }
    std::printf("%ld\n", wrong);
    return 0;
}
"""


def test_quotient_is_the_division(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(PROGRAM)
    # no contraction of its own: the fused operations are the ones written
    subprocess.check_call([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "lpma_gb300", "csrc"),
                           str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.stdout.strip() == "0", out.stdout + out.stderr
