"""csrc/quot.cuh on the host, from the estimates that the hardware's reciprocal is documented to allow: it
reads the upper 32 bits of the divisor and returns the upper 32 bits of a result, so that a divisor with a
full lower word is off by up to 2^-20 twice; and from perturbations up to 2^-19 beyond any of it.  The quotients
equal the division operator's bits, and the reciprocal is within half an ulp."""
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
static uint64_t s = 0x9E3779B97F4A7C15ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double unit(uint64_t mant) { uint64_t b = 0x3ff0000000000000ull | (mant & 0xfffffffffffffull); double d; memcpy(&d, &b, 8); return d; }
static double upper(double v) { uint64_t b; memcpy(&b, &v, 8); b &= 0xffffffff00000000ull; memcpy(&v, &b, 8); return v; }
static long bad = 0, n = 0;
static void one(double a, double b, int kind) {
    const double cut = upper(1.0 / upper(b));
    double est[6];
    int k = 0;
    if (kind < 3) {
        est[k++] = cut;
        // an estimate off by some units of its last kept bit
        est[k++] = upper(cut * (1.0 + 0x1p-21));
        est[k++] = upper(cut * (1.0 - 0x1p-21));
    } else {
        for (double e : {0x1p-19, -0x1p-19, 0x1.fp-20, -0x1.6p-20}) est[k++] = (1.0 / b) * (1.0 + e);
    }
    for (int j = 0; j < k; ++j) {
        const da::quot::Recip r = da::quot::refine(b, est[j]);
        // |b y - 1| of the nearest double, with the margin that the quotients need
        const double res = std::fabs(std::fma(b, r.y, -1.0)), best = std::fabs(std::fma(b, 1.0 / b, -1.0));
        int eb; std::frexp(b, &eb);
        const double half = std::ldexp(b, -eb + 1) * 0x1p-54 * (1.0 + 0x1p-50);
        ++n;
        if (!(res <= std::fmax(best, half)) && ++bad < 10) printf("1 / %a from %a: %a\n", b, est[j], r.y);
        for (double x : {a, -a}) {
            const double q = da::quot::div(x, r), w = x / b;
            if (memcmp(&q, &w, 8) && ++bad < 10) printf("%a / %a from %a: %a, not %a\n", x, b, est[j], q, w);
        }
    }
}
int main(int, char **v) {
    const int kind = v[1][0] - '0';
    for (int k = 0; k < 400000; ++k) {
        double b = unit(rnd()), a = unit(rnd());
        if (kind != 0) {
            uint64_t w; memcpy(&w, &b, 8); w |= 0xffffffffull; memcpy(&b, &w, 8);  // the whole lower word is cut off
        }
        if (kind == 2) b = 2.0 - std::ldexp(1.0 + (rnd() % 65536), -52);
        if (k & 1) {  // the quotient next to the middle of two neighbours
            const double q = unit(rnd());
            a = std::fma(b, q, b * 0x1p-53);
            if (k & 2) a = std::nextafter(a, (k & 4) ? 0.0 : 4.0);
        }
        if (k & 8) { const int e = -120 + (int)(rnd() % 240); a = std::ldexp(a, e); b = std::ldexp(b, e / 2); }
        one(a, b, kind);
    }
    printf("%ld estimates, %ld differ\n", n, bad);
    return bad != 0;
}
"""
KINDS = ["any divisor", "full lower word", "below a power of two", "perturbed by 2^-19"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("recip")
    (d / "r.cpp").write_text(SRC)
    exe = str(d / "r")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-x", "c++", "-I",
                    os.path.join(ROOT, "discrete_adjoint_b200", "csrc"), str(d / "r.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("kind", KINDS)
def test_quotients_from_cut_estimates(program, kind):
    r = subprocess.run([program, str(KINDS.index(kind))], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
