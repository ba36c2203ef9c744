// sc_ddmath.cuh -- natural logarithm and arctangent evaluated in
// double-double arithmetic and rounded once to double.
//
// The integrated Green's function (FFTPoissonSolver.cpp:472-493) cancels
// eight antiderivative values per mesh point, so a one-ulp difference in a
// single log or atan moves the field by about 1e-11 of its maximum.  Two
// libraries that round differently (glibc on the host, CUDA on the device)
// therefore disagree at that level.  These versions carry about 2^-100 of
// relative accuracy until the last rounding, so they return the correctly
// rounded result except when the exact value lies within roughly 2^-20 ulp
// of a rounding boundary; they use only +, -, *, /, sqrt-free fma, and table
// reads (the quick atan also an approximate reciprocal), and log_dd and
// atan_dd give the same bits on the host and on the device.  atan_fast, which
// has no rounding test, need not: its reciprocal and its table row may differ.
//
// Methods:
//   * error-free transformations TwoSum (Knuth), Fast2Sum (Dekker) and
//     TwoProd by fused multiply-add; double-double add / multiply / divide
//     after Dekker (1971) and the QD library's "accurate" variants.
//   * log: x = 2^k m, m in [sqrt(1/2), sqrt(2)); c = round(64 m) / 64;
//     log x = k log 2 + log c + log1p((m - c) / c)  (table-driven, after
//     Tang, "Table-driven implementation of the logarithm function", 1990).
//   * atan: s = |x| or 1/|x|; c = round(64 s) / 64;
//     atan s = atan c + atan((s - c) / (1 + s c)); pi/2 - atan(1/|x|) for |x| > 1.
//   Tables of log(j/64) and atan(j/64) as (hi, lo) pairs come from mpmath at
//   200 bits (gen_ddmath_tables.py).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SC_DDM_HD __host__ __device__ __forceinline__
#define SC_DDM_TABLE static __device__ const
#else
#define SC_DDM_HD static inline
#define SC_DDM_TABLE static const
#endif

#include "sc_ddmath_tables.h"

namespace sc {
namespace ddm {

struct dd {
    double hi, lo;
};

SC_DDM_HD dd two_sum(double a, double b) {
    const double s = a + b;
    const double bb = s - a;
    const double e = (a - (s - bb)) + (b - bb);
    return dd{s, e};
}

// requires |a| >= |b| (or a == 0)
SC_DDM_HD dd fast_two_sum(double a, double b) {
    const double s = a + b;
    const double e = b - (s - a);
    return dd{s, e};
}

SC_DDM_HD dd two_prod(double a, double b) {
    const double p = a * b;
    return dd{p, fma(a, b, -p)};
}

SC_DDM_HD dd neg(dd a) { return dd{-a.hi, -a.lo}; }

// "Sloppy" double-double addition: relative error about 2^-105 (|a| + |b|) /
// |a + b|.  Every sum below either has no cancellation, or (the residuals of
// div) only needs its result to 2^-53 relative.
SC_DDM_HD dd add(dd a, dd b) {
    dd s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return fast_two_sum(s.hi, s.lo);
}

SC_DDM_HD dd mul(dd a, dd b) {
    dd p = two_prod(a.hi, b.hi);
    p.lo += a.hi * b.lo + a.lo * b.hi;
    return fast_two_sum(p.hi, p.lo);
}

SC_DDM_HD dd mul_d(dd a, double b) {
    dd p = two_prod(a.hi, b);
    p.lo += a.lo * b;
    return fast_two_sum(p.hi, p.lo);
}

// a / b from one hardware division: q1 = a.hi (1 / b.hi) is within a few ulp
// of the quotient, and two correction terms from the exact residuals
// a - b (q1 + q2) bring the result to about 2^-100 relative.
SC_DDM_HD dd div(dd a, dd b) {
    const double inv = 1.0 / b.hi;
    const double q1 = a.hi * inv;
    dd r = add(a, neg(mul_d(b, q1)));
    const double q2 = r.hi * inv;
    r = add(r, neg(mul_d(b, q2)));
    const double q3 = r.hi * inv;
    return add(fast_two_sum(q1, q2), dd{q3, 0.0});
}

SC_DDM_HD dd tab(const double (*t)[2], int i) { return dd{t[i][0], t[i][1]}; }

// log(x) for finite normal x > 0; other inputs go to the library function.
SC_DDM_HD double log_dd_full(double x) {
    if (!(x >= 2.2250738585072014e-308) || !(x <= 1.7976931348623157e308)) return log(x);
    uint64_t bits;
    memcpy(&bits, &x, sizeof bits);
    int k = (int)(bits >> 52) - 1023;
    bits = (bits & 0x000fffffffffffffull) | 0x3ff0000000000000ull;
    double m;
    memcpy(&m, &bits, sizeof m);  // [1, 2)
    if (m > 1.4142135623730951) {
        m = m * 0.5;
        k += 1;
    }
    const int j = (int)rint(m * 64.0);  // 45 .. 91
    const double c = (double)j / 64.0;
    const double u = m - c;  // exact (Sterbenz)
    // t = u / c: th from the tabulated reciprocal, tl from the exact residual
    const double rc = kLogRcp[j - kLogJ0];
    const double th = u * rc;
    const double tl = fma(-th, c, u) * rc;
    const dd t = fast_two_sum(th, tl);     // |t| < 0.0112
    // log1p t = t - t^2/2 + t^3/3 + t^4 (-1/4 + t/5 - ... - t^8/12)
    const double h = t.hi;
    double p = -1.0 / 12.0;
    p = p * h + 1.0 / 11.0;
    p = p * h - 1.0 / 10.0;
    p = p * h + 1.0 / 9.0;
    p = p * h - 1.0 / 8.0;
    p = p * h + 1.0 / 7.0;
    p = p * h - 1.0 / 6.0;
    p = p * h + 1.0 / 5.0;
    p = p * h - 1.0 / 4.0;
    const dd t2 = mul(t, t);
    const dd t3 = mul(t2, t);
    const double h2 = h * h;
    dd s = add(t, dd{-0.5 * t2.hi, -0.5 * t2.lo});
    s = add(s, mul(t3, dd{kThirdHi, kThirdLo}));
    s = add(s, dd{(h2 * h2) * p, 0.0});
    const double kd = (double)k;
    dd r = add(dd{kd * kLn2Hi, 0.0}, two_prod(kd, kLn2Lo));
    r = add(r, dd{kd * kLn2Lo2, 0.0});
    r = add(r, tab(kLogTab, j - kLogJ0));
    r = add(r, s);
    return r.hi;
}

// atan(x) for finite x; NaN and infinities go to the library function.
SC_DDM_HD double atan_dd_full(double x) {
    const double a = fabs(x);
    if (!(a <= 1.7976931348623157e308)) return atan(x);
    if (a < 9.3132257461547852e-10) return x;  // |x| < 2^-30: x^3/3 is below half an ulp of x
    // s = min(a, 1/a); c = j/64 near s; atan s = atan c + atan t with
    //   a <= 1: t = (a - c) / (1 + a c)
    //   a >  1: t = (1/a - c) / (1 + c/a) = (1 - a c) / (a + c)
    // numerator and denominator are exact double-doubles (TwoProd, TwoSum).
    const bool inv = a > 1.0;
    const double s = inv ? 1.0 / a : a;
    const int j = (int)rint(s * 64.0);  // 0 .. 64
    const double c = (double)j / 64.0;
    dd num, den;
    if (inv) {
        const dd ac = two_prod(a, c);
        num = add(dd{1.0, 0.0}, neg(ac));
        den = two_sum(a, c);
    } else {
        num = dd{a - c, 0.0};  // exact (Sterbenz, or c = 0)
        den = add(dd{1.0, 0.0}, two_prod(a, c));
    }
    const dd t = div(num, den);  // |t| < 2^-7
    // atan t = t - t^3/3 + t^5 (1/5 - t^2/7 + t^4/9 - t^6/11)
    const double h = t.hi, h2 = h * h;
    double p = -1.0 / 11.0;
    p = p * h2 + 1.0 / 9.0;
    p = p * h2 - 1.0 / 7.0;
    p = p * h2 + 1.0 / 5.0;
    const dd t3 = mul(mul(t, t), t);
    dd r = add(t, mul(t3, dd{-kThirdHi, -kThirdLo}));
    r = add(r, dd{(h2 * h2 * h) * p, 0.0});
    r = add(r, tab(kAtanTab, j));
    if (inv) r = add(dd{kPiHalfHi, kPiHalfLo}, neg(r));
    return x < 0.0 ? -r.hi : r.hi;
}

// ---------------------------------------------------------------- quick phase
// Ziv's strategy (as in CRlibm, Daramy-Loirat et al.): a cheaper evaluation
// hi + lo with a proven error bound E; when hi + (lo - E) and hi + (lo + E)
// round to the same double, that double is the correctly rounded result,
// otherwise the full double-double evaluation above decides.  log and atan of
// a double other than log 1, atan 0 are transcendental, never exactly halfway
// between two doubles, and the accepted values keep a distance from the
// boundaries at which the full evaluation is correctly rounded too, so both
// phases give the same bits.
//
// The Green's function evaluates three of each per mesh point and is bound by
// the FP64 pipe, so both reductions are chosen for few operations: exact
// arguments from one fused multiply-add, low parts added in double, one
// rounding test in place of a renormalisation.  About 23 FP64 operations for
// log and 33 for atan (the first form, a 64-interval reduction with TwoSums
// throughout, took about 60 and 80): the Green's-function phase 175 -> 134 us
// at 128^3 and 41.6 -> 35.4 us at 64^3, the same bits.
struct hilo {
    double hi, lo;
};

SC_DDM_HD uint64_t bits_of(double x) {
    uint64_t b;
    memcpy(&b, &x, sizeof b);
    return b;
}
SC_DDM_HD double double_of(uint64_t b) {
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
}

// Tang's table-driven scheme in the form with short tabulated reciprocals
// instead of a division (r = z rc - 1 in one fused multiply-add), the exponent
// and the table row read from the bits of x less those of the first interval's
// start, as Arm's Optimized Routines (S. Nagy, 2018) publish it; the intervals,
// reciprocals and tables are our own (gen_ddmath_tables.py).
// log x = k log 2 - log rc + log1p r for finite normal x: z = x 2^-k in
// [0.707, 1.414), rc a short reciprocal of z's interval (kLogQ), r = z rc - 1
// exact, |r| <= 2^-7.  k log 2 (high part) - log rc (high part) is exact
// (both multiples of 2^-42); log1p r - r = r^2 (-1/2 + r/3 - ... + r^7/9) in
// double.  exact: the sum s + r is an exact Fast2Sum (|s| >= 2^-7 or s == 0).
// Error of hi + lo, where exact holds: the truncation of log1p below 2^-73,
// the polynomial r^2 (...) < 2^-15 with at most 1.6 2^-53 of it, two
// additions to lo (|lo| < 2^-14.9) 2^-68 each: together below 2^-66.3 (the
// largest seen over 2e7 arguments is 2^-67.5).
constexpr double kLogQuickErr = 0x1p-64;
SC_DDM_HD hilo log_hilo(double x, bool& exact) {
    const uint64_t b = bits_of(x);
    const uint32_t h = (uint32_t)(b >> 32);
    const uint32_t t = h - kLogQOff;
    const int k = (int32_t)t >> 20;
    const int i = (int)(t >> 13) & 127;
    const double z = double_of(((uint64_t)(h - (t & 0xfff00000u)) << 32) | (uint32_t)b);
    const double rc = kLogQ[i][0], th = kLogQ[i][1], tl = kLogQ[i][2];
    const double r = fma(z, rc, -1.0);
    double p = fma(r, 1.0 / 9.0, -1.0 / 8.0);
    p = fma(r, p, 1.0 / 7.0);
    p = fma(r, p, -1.0 / 6.0);
    p = fma(r, p, 1.0 / 5.0);
    p = fma(r, p, -1.0 / 4.0);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -0.5);
    // k as a double: 2^52 + 2^31 + k has k + 2^31 in its low word (no conversion)
    const double kd = double_of((uint64_t)0x43300000u << 32 | ((uint32_t)k ^ 0x80000000u)) - (0x1p52 + 0x1p31);
    const double s = fma(kd, kLn2Hi, th);
    exact = ((uint32_t)(bits_of(s) >> 32) & 0x7fffffffu) >= 0x3f800000u || s == 0.0;
    const double hi = s + r;
    double lo = fma(kd, kLn2Lo, tl);
    lo = fma(r * r, p, lo);
    lo += r - (hi - s);
    return hilo{hi, lo};
}

// Quick log: false where the rounding is undecided.
SC_DDM_HD bool log_quick(double x, double& out) {
    bool exact;
    const hilo v = log_hilo(x, exact);
    out = v.hi + (v.lo + kLogQuickErr);
    return exact && out == v.hi + (v.lo - kLogQuickErr);
}

// Reciprocal of d in [1, 2^31] to 2^-51: an approximation r to 2^-20 and one
// step r (1 + e + e^2), e = 1 - d r, of Chebyshev's third-order iteration for
// the zero of 1/x - d.
SC_DDM_HD double rcp_approx(double d) {
    double r;
#ifdef __CUDA_ARCH__
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
#else
    r = (double)(1.0f / (float)d);
#endif
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// atan a for 2^-30 <= a <= 2^30: c = j/128 near a (a <= 1) or near 1/a;
//   a <= 1: atan a = atan c + atan t,        t = (a - c) / (1 + a c)
//   a >  1: atan a = (pi/2 - atan c) + atan t, t = (a c - 1) / (a + c)
// with |t| < 1.01 2^-8.  The numerator is exact in one fused multiply-add (c
// has 8 bits, the difference cancels at least as many), the denominator is
// dh + dl exactly, and t = th + tl to 2^-100 from the residual; atan t - t =
// t^3 (-1/3 + t^2/5 - t^4 (1/7 - d)) in double, d = 0.92 of the next term's
// t^2/9 at |t| = 2^-8, which leaves a truncation below 2^-69 t.  Error of
// hi + lo relative to hi: below 2^-67.5 (largest for c = 0, where the tail
// t^3/3 < 2^-17.5 t carries at most 3 2^-53 of itself; for c >= 1/128 the
// tail is below 2^-18.5 hi; the largest seen over 2e7 arguments is 2^-67.8).
constexpr double kAtanQuickEps = 0x1p-66;
SC_DDM_HD hilo atan_hilo(double a) {
    const bool inv = (uint32_t)(bits_of(a) >> 32) >= 0x3ff00000u;  // a >= 1, on the integer units
    const float f = (float)a;
    // a float quotient a few ulp off may pick the neighbour of round(128 / a)
#ifdef __CUDA_ARCH__
    const int j = __float2int_rn(inv ? __fdividef(128.0f, f) : 128.0f * f);
#else
    const int j = (int)rintf(inv ? 128.0f / f : 128.0f * f);
#endif
    const int row = inv ? j + 129 : j;
    const double th0 = kAtanQ[row][0], tl0 = kAtanQ[row][1];
    // j / 128: 2^45 + j / 128 has j in its low word
    const double c = double_of((uint64_t)0x42c00000u << 32 | (uint32_t)j) - 0x1p45;
    const double u = inv ? a : 1.0, w = inv ? 1.0 : a;
    const double num = inv ? fma(a, c, -1.0) : a - c;
    const double dh = fma(w, c, u);
    const double dl = fma(w, c, u - dh);
    const double rd = rcp_approx(dh);
    const double t = num * rd;
    const double tl = fma(-t, dl, fma(-t, dh, num)) * rd;
    const double t2 = t * t;
    double q = fma(t2, -1.0 / 7.0 + 0.92 * 0x1p-16 / 9.0, 1.0 / 5.0);
    q = fma(t2, q, -1.0 / 3.0);
    const double hi = th0 + t;
    double lo = fma(t2 * t, q, tl);
    lo += tl0;
    lo += t - (hi - th0);
    return hilo{hi, lo};
}

// Quick atan for 2^-30 <= |x| <= 2^30: false where the rounding is undecided.
SC_DDM_HD bool atan_quick(double x, double& out) {
    const hilo v = atan_hilo(fabs(x));
    const double r = v.hi + fma(v.hi, kAtanQuickEps, v.lo);
    out = copysign(r, x);
    return r == v.hi + fma(v.hi, -kAtanQuickEps, v.lo);
}

// Correctly rounded log and atan (the quick phase, else the full evaluation).
// The ranges are tested on the high word: x positive, normal and finite (log
// 1 is undecided in the quick phase); 2^-30 <= |x| < 2^30.
SC_DDM_HD bool log_range(double x) { return (uint32_t)(bits_of(x) >> 32) - 0x00100000u < 0x7fe00000u; }
SC_DDM_HD bool atan_range(double x) {
    return ((uint32_t)(bits_of(x) >> 32) & 0x7fffffffu) - 0x3e100000u < 0x41d00000u - 0x3e100000u;
}

SC_DDM_HD double log_dd(double x) {
    double r;
    if (log_range(x) && log_quick(x, r)) return r;
    return log_dd_full(x);
}

SC_DDM_HD double atan_dd(double x) {
    double r;
    if (atan_range(x) && atan_quick(x, r)) return r;
    return atan_dd_full(x);
}

// The same reductions without the rounding test (the mixed form): hi + lo
// rounded once, of the arguments the quick phases take.  By their error bounds
// within 0.5001 ulp for atan and for log where |log x| >= 2, within 0.513 for
// log nearer 1 (largest seen: 0.50001, 0.50001 and 0.5055;
// tests/ddmath_fast_check.cpp).
SC_DDM_HD double log_fast(double x) {
    if (!log_range(x)) return log(x);
    bool exact;
    const hilo v = log_hilo(x, exact);
    return v.hi + v.lo;
}

SC_DDM_HD double atan_fast(double x) {
    if (!atan_range(x)) return atan(x);
    const hilo v = atan_hilo(fabs(x));
    return copysign(v.hi + v.lo, x);
}

}  // namespace ddm
}  // namespace sc
