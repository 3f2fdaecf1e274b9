"""The integer form of the FP64 products (aspartik_gb300/csrc/soft64.cuh),
compiled on its own with the host C++ compiler, against exact rational
arithmetic: two row sums of four positive products each, multiplied and
rounded once.

Bound: a term is at most 2 units (truncated cross terms) and 1 unit
(alignment shift) of 2^-60 of the largest term low, so a sum of four is at
most 12 / 2^60 low, the product of two sums 24 / 2^60 = 0.1 units in the last
place; the product's own truncation loses less than 2 units of 2^-56 (0.125)
and the final rounding half a unit: below 0.75 units in the last place of the
smaller binade, so below 1 in every case."""

import os
import random
import shutil
import struct
import subprocess
import tempfile
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "soft64.cuh"
#include <cstdio>
using namespace b3g;
static SoftNum split(unsigned long long v) {
    return soft_split((uint32_t)(v >> 32), (uint32_t)v);
}
// sum of four products as the kernel forms it
static void dot(const unsigned long long *x, const unsigned long long *p, uint64_t &m,
                int32_t &e) {
    uint32_t s[4];
    for (int k = 0; k < 4; ++k) s[k] = split(x[k]).e + split(p[k]).e;
    const uint32_t top = soft_max2(soft_max2(s[0], s[1]), soft_max2(s[2], s[3]));
    m = 0;
    for (int k = 0; k < 4; ++k) {
        const SoftNum a = split(x[k]), b = split(p[k]);
        m += soft_shr(soft_prod(a.hi, a.lo, b.hi, b.lo), top - s[k]);
    }
    e = (int32_t)top - kSoftDotBias;
}
int main() {
    unsigned long long v[16];
    for (;;) {
        for (int k = 0; k < 16; ++k)
            if (std::scanf("%llx", v + k) != 1) return 0;
        uint64_t a, b;
        int32_t ea, eb;
        dot(v, v + 4, a, ea);
        dot(v + 8, v + 12, b, eb);
        bool ok, ok2;
        const uint64_t y = soft_mul_round(a, ea, b, eb, ok);
        const SoftNum t = split(v[0]); // a tip: one table entry
        const uint64_t z = soft_mul_round(((uint64_t)t.hi << 32) | t.lo,
                                          (int32_t)t.e - kSoftBias, b, eb, ok2);
        const uint64_t w = soft_scale(v[0], split(v[1]));
        std::printf("%016llx %d %016llx %d %016llx\n", (unsigned long long)y, ok,
                    (unsigned long long)z, ok2, (unsigned long long)w);
    }
}
"""


def bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def off(got, want):
    """Distance of a double from an exact value in units in the last place."""
    x = struct.unpack("<d", struct.pack("<Q", got))[0]
    ulp = Fraction(2) ** (((got >> 52) & 0x7FF) - 1075)
    return abs(Fraction(x) - want) / ulp


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("spread", [0, 4, 40, 200])
def test_products_of_sums(spread):
    rng = random.Random(7 + spread)
    rows = []
    for _ in range(3000):
        row = [rng.choice([1.0, 1.0 - 2.0 ** -53, 1.0 + 2.0 ** -52, rng.uniform(1.0, 2.0)]) *
               2.0 ** -rng.randint(0, spread) for _ in range(16)]
        rows.append(row)
    # results outside the normal range must be reported, not returned
    rows.append([2.0 ** -540] * 16)
    rows.append([2.0 ** 300] * 16)
    with tempfile.TemporaryDirectory() as d:
        src = os.path.join(d, "t.cpp")
        with open(src, "w") as f:
            f.write(PROGRAM)
        exe = os.path.join(d, "t")
        subprocess.run(["g++", "-O2", "-std=c++17",
                        "-I" + os.path.join(ROOT, "aspartik_gb300", "csrc"), src, "-o", exe],
                       check=True)
        text = "\n".join(" ".join(f"{bits(v):x}" for v in row) for row in rows)
        out = subprocess.run([exe], input=text, capture_output=True, text=True,
                             check=True).stdout.split("\n")
    for row, line in zip(rows[:-2], out):
        y, ok, z, ok2, w = line.split()
        f = [Fraction(v) for v in row]
        b = sum(f[8 + k] * f[12 + k] for k in range(4))
        assert ok == "1" and ok2 == "1"
        assert off(int(y, 16), sum(f[k] * f[4 + k] for k in range(4)) * b) < 1
        assert off(int(z, 16), f[0] * b) < 1
        assert off(int(w, 16), f[0] * f[1]) < 1
    assert out[len(rows) - 2].split()[1] == "0"
    assert out[len(rows) - 1].split()[1] == "0"
