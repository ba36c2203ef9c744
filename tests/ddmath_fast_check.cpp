// Host build of log_fast / atan_fast (sc_ddmath.cuh), the evaluations without
// a rounding test, against quad precision.  Prints the largest errors in ulps:
//   <log, |log x| >= 2> <log, everywhere> <atan, 2^-30 <= |x| < 2^30>
// over random mantissas and exponents (not exp(u): its log is within 2^-53 of
// the double u, a quarter of an ulp at most), arguments next to 1 and every table interval.
#include <quadmath.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "sc_ddmath.cuh"

// |v - exact| in units of the last place of the rounded exact value
static double ulps(double v, __float128 exact) {
    const double r = std::fabs((double)exact);
    const double ulp = std::nextafter(r, INFINITY) - r;
    return (double)(fabsq((__float128)v - exact) / ulp);
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    std::mt19937_64 g(54321);
    std::uniform_real_distribution<double> mant(1.0, 2.0), w(-1.0 / 128, 1.0 / 128);
    std::uniform_int_distribution<int> xl(-43, 43), xa(-30, 29);
    double far = 0.0, all = 0.0, at = 0.0;
    auto check_log = [&](double x) {
        if (!(x > 0.0) || x == 1.0) return;
        const __float128 q = logq((__float128)x);
        const double e = ulps(sc::ddm::log_fast(x), q);
        all = std::max(all, e);
        if (fabsq(q) >= 2) far = std::max(far, e);
    };
    auto check_atan = [&](double y) {
        if (sc::ddm::atan_range(y)) at = std::max(at, ulps(sc::ddm::atan_fast(y), atanq((__float128)y)));
    };
    for (long i = 0; i < n; ++i) {
        check_log(std::ldexp(mant(g), xl(g)));
        check_log(1.0 + 2.0 * w(g));
        check_log((90 + (int)(i % 93)) / 128.0 + w(g));
        check_atan(((i & 1) ? -1.0 : 1.0) * std::ldexp(mant(g), xa(g)));
        const double y = (int)(i % 129) / 128.0 + w(g) / 2;
        check_atan(y);
        if (y != 0.0) check_atan(1.0 / y);
    }
    std::printf("%.6f %.6f %.6f\n", far, all, at);
    return 0;
}
