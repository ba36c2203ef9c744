// sc_exact.cuh -- order-independent (exact) sums of doubles on the device.
//
// Every double v with |v| < 2^55 becomes the 128-bit integer
// trunc(v * 2^72); integer addition is exact and associative, so a sum over
// particles does not depend on the order the particles are visited in (the
// particle arrays are reordered by cell every few steps).  The total is
// rounded to a double once.  Parts below 2^-72 (2e-22) are dropped, far
// below the rounding of any sum the step forms.
#pragma once

#include <cstdint>

#include "sc_common.cuh"

namespace sc {

using i128 = __int128;
using u128 = unsigned __int128;

constexpr int kExFrac = 72;

__device__ __forceinline__ i128 ex_from(double v) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const int e = (int)((bits >> 52) & 0x7ff);
    if (e == 0) return 0;  // zero or subnormal
    const unsigned long long m = (bits & 0xfffffffffffffull) | (1ull << 52);
    // v = m * 2^(e - 1075); fixed = m * 2^(e - 1075 + kExFrac)
    const int sh = e - 1075 + kExFrac;
    u128 mag;
    if (sh >= 0)
        mag = sh < 75 ? ((u128)m << sh) : ((u128)m << 74);  // |v| >= 2^55 saturates (out of contract)
    else
        mag = sh > -53 ? (u128)(m >> (-sh)) : (u128)0;
    return (bits >> 63) ? -(i128)mag : (i128)mag;
}

// The same fixed point accumulated per thread in two 64-bit words, value
// hi 2^36 + lo in units of 2^-72, for |v| < 2^10: hi gains floor(|v| 2^36)
// and lo the next 36 bits, each with v's sign.  Adding 2^16 (2^-20) with
// rounding towards zero leaves the bits above 2^-36 (2^-72) in the
// mantissa field, so two additions and two subtractions replace the 128-bit
// shift and addition of ex_from (about 18 operations per value against 35).
// hi grows by less than 2^46 per value, lo by less than 2^36: 2^16 values per
// thread fit.  Larger values (and NaN) go to `big`, four 64-bit counters per value in
// shared memory that take the 32-bit chunks of ex_from's integer.
struct ExAcc {
    long long hi, lo;
};

// All NV values at once: the rare path appears once in the caller's code.
template <int NV>
__device__ __forceinline__ void ex_add(ExAcc (&acc)[NV], const double (&v)[NV], unsigned long long* big) {
    bool fits = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) fits = fits && fabs(v[k]) < 1024.0;
    if (fits) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const double a = fabs(v[k]);
            const double m = __dadd_rz(a, 0x1p16);
            const double q = __dadd_rz(a - (m - 0x1p16), 0x1p-20);
            const long long sign = __double_as_longlong(v[k]) >> 63;
            acc[k].hi += ((__double_as_longlong(m) & 0xfffffffffffffll) ^ sign) - sign;
            acc[k].lo += ((__double_as_longlong(q) & 0xfffffffffffffll) ^ sign) - sign;
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < NV; ++k) {
            double x = v[0];
#pragma unroll
            for (int j = 1; j < NV; ++j) x = k == j ? v[j] : x;
            const u128 t = (u128)ex_from(x);
#pragma unroll
            for (int j = 0; j < 4; ++j) atomicAdd(big + 4 * k + j, (unsigned long long)(unsigned)(t >> (32 * j)));
        }
    }
}

__device__ __forceinline__ i128 ex_value(const ExAcc& acc) { return ((i128)acc.hi << 36) + (i128)acc.lo; }

// correctly rounded double of x * 2^-kExFrac
__device__ __forceinline__ double ex_to_double(i128 x) {
    const bool neg = x < 0;
    const u128 m = neg ? (u128)(-x) : (u128)x;
    const unsigned long long hi = (unsigned long long)(m >> 64), lo = (unsigned long long)m;
    double r;
    if (hi == 0) {
        r = __ull2double_rn(lo) * 0x1p-72;
    } else {
        const int lz = __clzll(hi);
        const unsigned long long top = lz ? ((hi << lz) | (lo >> (64 - lz))) : hi;
        const unsigned long long rest = lo << lz;
        unsigned long long mant = top >> 11;
        const unsigned long long rem = top & 0x7ffull;
        if (rem > 0x400ull || (rem == 0x400ull && (rest != 0 || (mant & 1ull)))) mant += 1;
        // mant 2^(75 - lz - kExFrac): a product with a power of two, exact
        r = (double)mant * __longlong_as_double((long long)(1023 + 75 - kExFrac - lz) << 52);
    }
    return neg ? -r : r;
}

__device__ __forceinline__ i128 ex_shfl_down(i128 v, int off) {
    const u128 u = (u128)v;
    const unsigned long long lo = __shfl_down_sync(0xffffffffu, (unsigned long long)u, off);
    const unsigned long long hi = __shfl_down_sync(0xffffffffu, (unsigned long long)(u >> 64), off);
    return (i128)(((u128)hi << 64) | lo);
}

// ---------------------------------------------------------------- deposit
// Exact sums of the scattered charges: each charge v (|v| <= |q dt|) becomes
// the integer t = rint(v * 2^(52 - E)) with 2^E > 2 |q dt|, so |t| < 2^51;
// the sums are integer additions, exact, so any order gives the same total,
// which is rounded to a double once.  The rounding of t is at most 2^-52 of
// one particle's charge.
// correctly rounded double of the 128-bit accumulator (lo, hi), times unit
__device__ __forceinline__ double acc_to_double(unsigned long long lo, unsigned long long hi, double unit) {
    const long long shi = (long long)hi;
    if (shi == ((long long)lo < 0 ? -1 : 0)) return __ll2double_rn((long long)lo) * unit;  // fits in 64 bits
    const bool neg = shi < 0;
    unsigned long long mlo = lo, mhi = hi;
    if (neg) {
        mlo = ~mlo + 1ull;
        mhi = ~mhi + (mlo == 0 ? 1ull : 0ull);
    }
    const int lz = __clzll(mhi);
    const unsigned long long top = lz ? ((mhi << lz) | (mlo >> (64 - lz))) : mhi;
    const unsigned long long rest = mlo << lz;
    unsigned long long mant = top >> 11;
    const unsigned long long rem = top & 0x7ffull;
    if (rem > 0x400ull || (rem == 0x400ull && (rest != 0 || (mant & 1ull)))) mant += 1;
    const double r = (double)mant * __longlong_as_double((long long)(1023 + 75 - lz) << 52);  // mant 2^(75 - lz)
    return (neg ? -r : r) * unit;
}

// The charge density of one node from its accumulator (L, H) = H 2^32 + L:
// (exact node sum) / dT * tmp2 (PartBunch.cpp:496, :510-511).  Only a
// product and a quotient: no contraction can change its rounding.  rdT: RN(1
// / dT), or 0 to divide (dT below 2^-70, where div_rcp does not hold); an
// empty node skips the quotient.
__device__ __forceinline__ double node_density(ulonglong2 a, double unit, double dT, double rdT, double tmp2) {
    if ((a.x | a.y) == 0ull) return 0.0 * tmp2;
    const i128 w = ((i128)(long long)a.y << 32) + (i128)a.x;
    double s = acc_to_double((unsigned long long)w, (unsigned long long)(w >> 64), unit);
    s = rdT != 0.0 ? div_rcp(s, dT, rdT) : s / dT;
    s *= tmp2;
    return s;
}

}  // namespace sc
