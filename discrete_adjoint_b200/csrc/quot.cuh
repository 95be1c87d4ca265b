// FP64 quotients that share a divisor, correctly rounded without a branch.
//
// The step divides by the same value several times over (the three components of an HLL flux by
// sr - sl, a cell's slopes by its centre distances, hu, hv and the slopes by h), and the reference's
// bits need every quotient rounded as the division operator rounds it.  The operator costs a
// reciprocal of its own each time and a range test with a branch, which also keeps the compiler from
// interleaving neighbouring quotients: one after another they are most of a cell's latency.  Here
// the reciprocal is formed once per divisor and each quotient is one multiplication and four fused
// multiply-adds (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34, 1990):
//   q0 = a y,  r0 = b q0 - a,  q1 = q0 - r0 y,  r1 = b q1 - a,  q = q1 - r1 y.
// With y within half an ulp of 1/b, q1 is within one ulp of a/b; then r1 is exact, and q is a/b
// rounded to nearest: where a/b lies next to the middle m of two neighbours, q1 is half an ulp
// away, so q1 - r1 y before its rounding differs from a/b by at most 2^-54 |b y - 1| (b scaled to
// [1, 2), a/b to [1/2, 2)), less than 2^-106 / b, the least distance of a/b to m.  The residuals are
// taken with this sign so that a zero numerator keeps its sign.
//
// Valid while nothing underflows or overflows.  The callers guarantee it: the state is zero or
// within [2^-150, 2^100] (ordinary, below), the mesh's distances and g_z within [2^-40, 2^40]
// and k act/pass zero or within [2^-60, 2^60] (checked once on the host); every numerator is then
// zero or within [2^-760, 2^760], every divisor within [2^-250, 2^250] and every quotient zero or above
// 2^-910.  Anything else takes the division operator.
//
// Three quotients of one divisor, chained, one warp: 112 cycles a round against 382 with the operator.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define DA_QUOT_FN __device__ __forceinline__
#else
#include <cmath>
#define DA_QUOT_FN inline
#endif

namespace da {
namespace quot {

struct Recip {
    double b, y;  // divisor (positive), 1/b
};

#ifdef __CUDACC__
DA_QUOT_FN double mul(double a, double b) { return __dmul_rn(a, b); }
DA_QUOT_FN double mul_add(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
DA_QUOT_FN double mul(double a, double b) { return a * b; }
DA_QUOT_FN double mul_add(double a, double b, double c) { return std::fma(a, b, c); }
#endif

// 1/b from an estimate y0.  The hardware's is documented to read the upper 32 bits of b and to return the
// upper 32 bits of its result, the others zero: each cut costs up to 2^-20, taken as |e| < 2^-19 in all.
// Two steps of Goldschmidt's iteration (Applications of division by convergence, MIT, 1964: y (1 + e) (1 + e^2),
// whose factors do not wait for one another) leave e^4 < 2^-76 and the rounding of two results, an ulp; a
// Newton step (Markstein's, as above) from there leaves 2^-104 before its own rounding, which is y within
// half an ulp (and 2^-51 of that).  Three Newton steps are one multiply-add longer in their chain.
DA_QUOT_FN Recip refine(double b, double y0) {
    const double e = mul_add(-b, y0, 1.0);
    const double y1 = mul_add(e, y0, y0), e2 = mul(e, e);
    const double y2 = mul_add(e2, y1, y1);
    return Recip{b, mul_add(mul_add(-b, y2, 1.0), y2, y2)};
}

// a / b, rounded to nearest
DA_QUOT_FN double div(double a, const Recip &r) {
    const double q0 = mul(a, r.y);
    const double q1 = mul_add(mul_add(r.b, q0, -a), -r.y, q0);
    return mul_add(mul_add(r.b, q1, -a), -r.y, q1);
}

#ifdef __CUDACC__
DA_QUOT_FN Recip recip(double b) {
    double y0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
    return refine(b, y0);
}

// v is zero or of a magnitude within [2^-150, 2^100]
DA_QUOT_FN bool ordinary(double v) {
    constexpr unsigned lo = (1023u - 150u) << 20, hi = (1023u + 100u) << 20;
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) - lo <= hi - lo || v == 0.0;
}
#endif

}  // namespace quot
}  // namespace da
