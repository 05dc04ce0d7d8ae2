"""QuotExact::many and the constructor that takes a ready reciprocal
(mage_b200/csrc/gam_quot.cuh), compiled for the host: N quotients at once are
the IEEE quotients bit for bit, also where one operand of the group is out of
the fast range, zero of either sign, infinite or NaN. QuotExact::quick is the IEEE
quotient or says that it is not."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "gam_quot.cuh"
static uint64_t sm(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double bits(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
static bool same(double x, double y) { return memcmp(&x, &y, 8) == 0 || (x != x && y != y); }
int main(int argc, char** argv) {
    const long n = atol(argv[1]);
    uint64_t s = 7;
    long bad = 0;
    const double odd[8] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, 1e-200, 1e200};
    for (long i = 0; i < n; i++) {
        auto rnd = [&](int spread) {
            return bits((sm(s) & 0x800FFFFFFFFFFFFFull) | ((uint64_t)(1023 + (int)(sm(s) % (2 * spread)) - spread) << 52));
        };
        const double d = (i % 7 == 0) ? bits(sm(s)) : rnd(i % 2 ? 40 : 500);
        double a[5], q[5];
        for (int k = 0; k < 5; k++) a[k] = rnd(i % 3 ? 40 : 500);
        if (i % 5 == 0) a[sm(s) % 5] = odd[sm(s) % 8];
        gam::QuotExact(d, 1.0 / d).many<5>(a, q);
        for (int k = 0; k < 5; k++) bad += !same(q[k], a[k] / d);
        // quick: where it does not turn ok off it is the quotient, and it stays on in the ordinary range
        for (int k = 0; k < 5; k++) {
            bool ok = true;
            const double v = gam::QuotExact(d, 1.0 / d).quick(a[k], ok);
            bad += ok && !same(v, a[k] / d);
            bad += !ok && std::fabs(d) > 1e-13 && std::fabs(d) < 1e13 && std::fabs(a[k]) > 1e-13 && std::fabs(a[k]) < 1e13;
        }
    }
    printf("%ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_many_equals_division(tmp_path):
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I", os.path.join(ROOT, "mage_b200/csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "3000000"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
