"""csrc/quot.cuh on the host: quotients from a shared reciprocal equal the division operator's bits
over the declared ranges, from the worst reciprocal estimate the hardware may give (relative error
2^-22), including divisors next to a power of two, numerators whose quotient lies next to the middle
of two neighbours, exact quotients and signed zeros."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "quot.cuh"
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double unit(uint64_t mant) { uint64_t b = 0x3ff0000000000000ull | (mant & 0xfffffffffffffull); double d; memcpy(&d, &b, 8); return d; }
static long bad = 0, n = 0;
static void one(double a, double b) {
    const double est = 1.0 / b;
    const double errs[] = {0.0, 0x1p-22, -0x1p-22, 0x1.7p-24, -0x1.3p-25};
    for (double e : errs) {
        const da::quot::Recip r = da::quot::refine(b, est * (1.0 + e));
        for (double x : {a, -a}) {
            const double q = da::quot::div(x, r), w = x / b;
            ++n;
            if (memcmp(&q, &w, 8)) { if (++bad < 10) printf("%a / %a: %a, not %a\n", x, b, q, w); }
        }
    }
}
int main(int, char **v) {
    const int kind = v[1][0] - '0';
    for (int k = 0; k < 400000; ++k) {
        double b = unit(rnd()), a = unit(rnd());
        if (kind == 1) b = 2.0 - std::ldexp(1.0 + (rnd() % 4096), -52);   // just below a power of two
        if (kind == 1 && (k & 1)) a = 2.0 - std::ldexp(1.0 + (rnd() % 4096), -52);
        if (kind == 2) {
            // a next to b (2 q + 1 ulp) / 2: the quotient next to the middle of two neighbours
            const double q = unit(rnd());
            a = std::fma(b, q, b * 0x1p-53);
            if (k & 1) a = std::nextafter(a, (k & 2) ? 0.0 : 4.0);
        }
        if (kind == 3) a = b * (double)(1 + rnd() % 1000000);  // exact quotients
        if (kind == 4) { a = (k & 1) ? 0.0 : std::ldexp(a, -780 + (int)(rnd() % 1560)); b = std::ldexp(b, -120 + (int)(rnd() % 240)); }
        one(a, b);
    }
    printf("%ld quotients, %ld differ\n", n, bad);
    return bad != 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("quot")
    (d / "q.cpp").write_text(SRC)
    exe = str(d / "q")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-x", "c++", "-I",
                    os.path.join(ROOT, "discrete_adjoint_b200", "csrc"), str(d / "q.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("kind", ["any", "divisor below a power of two", "middle of two neighbours", "exact",
                                  "whole range"])
def test_quotients_equal_the_operator(program, kind):
    k = ["any", "divisor below a power of two", "middle of two neighbours", "exact", "whole range"].index(kind)
    r = subprocess.run([program, str(k)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
