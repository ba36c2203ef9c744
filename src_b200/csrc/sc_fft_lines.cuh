// sc_fft_lines.cuh -- complex arithmetic, radix butterflies and the
// register-resident line transform shared by the FFT translation units
// (sc_fft.cu, sc_fft_plane.cu).  Both are compiled without FMA contraction,
// so every kernel that shares these butterflies rounds identically.
#pragma once

#include <type_traits>

#include "sc_internal.h"

namespace sc {
namespace {

template <typename T>
struct CT;
template <>
struct CT<double> {
    using type = double2;
};
template <>
struct CT<float> {
    using type = float2;
};
template <typename T>
using Cx = typename CT<T>::type;

template <typename C>
__device__ __forceinline__ C cadd(C a, C b) {
    return {a.x + b.x, a.y + b.y};
}
template <typename C>
__device__ __forceinline__ C csub(C a, C b) {
    return {a.x - b.x, a.y - b.y};
}
// Complex product with its two fused multiply-adds written out.  The file is
// compiled without FMA contraction (-fmad=false), so every kernel that shares
// these butterflies rounds identically, whatever the surrounding code: the
// staged, register-resident and batched transforms give the same bits.
__device__ __forceinline__ float fmx(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmx(double a, double b, double c) { return fma(a, b, c); }
template <typename C>
__device__ __forceinline__ C cmul(C a, C b) {
    return {fmx(a.x, b.x, -(a.y * b.y)), fmx(a.x, b.y, a.y * b.x)};
}

// ---------------------------------------------------------------- butterflies
// R-point DFT in registers; forward uses exp(-2 pi i / R).
template <typename T, int R, bool INV>
__device__ __forceinline__ void dft(Cx<T>* v) {
    using C = Cx<T>;
    if constexpr (R == 2) {
        C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4) {
        C t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
        C t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
        v[0] = cadd(t0, t2);
        v[2] = csub(t0, t2);
        if constexpr (!INV) {
            v[1] = C{t1.x + t3.y, t1.y - t3.x};
            v[3] = C{t1.x - t3.y, t1.y + t3.x};
        } else {
            v[1] = C{t1.x - t3.y, t1.y + t3.x};
            v[3] = C{t1.x + t3.y, t1.y - t3.x};
        }
    } else if constexpr (R == 3) {
        const T s = INV ? (T)0.86602540378443864676 : (T)-0.86602540378443864676;
        C t1 = cadd(v[1], v[2]);
        C d = csub(v[1], v[2]);
        C t2 = C{v[0].x - (T)0.5 * t1.x, v[0].y - (T)0.5 * t1.y};
        v[0] = cadd(v[0], t1);
        v[1] = C{t2.x - s * d.y, t2.y + s * d.x};
        v[2] = C{t2.x + s * d.y, t2.y - s * d.x};
    } else if constexpr (R == 8) {
        // 2 x 4: a_k = x_k + x_{k+4}, b_k = (x_k - x_{k+4}) W8^k; X_{2m} = DFT4(a), X_{2m+1} = DFT4(b)
        const T h = (T)0.70710678118654752440;
        C a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            a[k] = cadd(v[k], v[k + 4]);
            b[k] = csub(v[k], v[k + 4]);
        }
        // W8^1 = (1 - i)/sqrt2 (forward), W8^2 = -i, W8^3 = -(1 + i)/sqrt2; conjugates for the inverse
        if constexpr (!INV) {
            b[1] = C{h * (b[1].x + b[1].y), h * (b[1].y - b[1].x)};
            b[2] = C{b[2].y, -b[2].x};
            b[3] = C{h * (b[3].y - b[3].x), -h * (b[3].x + b[3].y)};
        } else {
            b[1] = C{h * (b[1].x - b[1].y), h * (b[1].y + b[1].x)};
            b[2] = C{-b[2].y, b[2].x};
            b[3] = C{-h * (b[3].x + b[3].y), h * (b[3].x - b[3].y)};
        }
        dft<T, 4, INV>(a);
        dft<T, 4, INV>(b);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            v[2 * m] = a[m];
            v[2 * m + 1] = b[m];
        }
    } else if constexpr (R == 5) {
        const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
        const T s1 = INV ? (T)0.95105651629515357212 : (T)-0.95105651629515357212;
        const T s2 = INV ? (T)0.58778525229247312917 : (T)-0.58778525229247312917;
        C a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
        C a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
        C x0 = v[0];
        C r1 = C{x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y};
        C r2 = C{x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y};
        C i1 = C{s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y};
        C i2 = C{s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y};
        v[0] = C{x0.x + a1.x + a2.x, x0.y + a1.y + a2.y};
        v[1] = C{r1.x - i1.y, r1.y + i1.x};
        v[4] = C{r1.x + i1.y, r1.y - i1.x};
        v[2] = C{r2.x - i2.y, r2.y + i2.x};
        v[3] = C{r2.x + i2.y, r2.y - i2.x};
    }
}

// R-point DFT of inputs whose upper half v[R/2 .. R-1] is zero (the
// zero-padded half of a forward transform's first stage).
template <typename T, int R, bool INV>
__device__ __forceinline__ void dft_half(Cx<T>* v) {
    using C = Cx<T>;
    if constexpr (R == 2) {
        v[1] = v[0];
    } else if constexpr (R == 4) {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[2] = csub(a, b);
        if constexpr (!INV) {
            v[1] = C{a.x + b.y, a.y - b.x};
            v[3] = C{a.x - b.y, a.y + b.x};
        } else {
            v[1] = C{a.x - b.y, a.y + b.x};
            v[3] = C{a.x + b.y, a.y - b.x};
        }
    } else {
        static_assert(R == 8, "half-input DFT for radix 2, 4, 8");
        const T h = (T)0.70710678118654752440;
        C a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = b[k] = v[k];
        if constexpr (!INV) {
            b[1] = C{h * (b[1].x + b[1].y), h * (b[1].y - b[1].x)};
            b[2] = C{b[2].y, -b[2].x};
            b[3] = C{h * (b[3].y - b[3].x), -h * (b[3].x + b[3].y)};
        } else {
            b[1] = C{h * (b[1].x - b[1].y), h * (b[1].y + b[1].x)};
            b[2] = C{-b[2].y, b[2].x};
            b[3] = C{-h * (b[3].x + b[3].y), h * (b[3].x - b[3].y)};
        }
        dft<T, 4, INV>(a);
        dft<T, 4, INV>(b);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            v[2 * m] = a[m];
            v[2 * m + 1] = b[m];
        }
    }
}

// ---------------------------------------------------------------- lines in registers
// The same Stockham transform of a 64-, 128- or 256-point line (plans 8 8;
// 4 4 8; 4 8 8: the same butterflies, twiddles and operation order as
// block_fft, so the same bits), computed by 8 threads of one warp with the
// data in registers: thread a holds elements a + 8m (m < L/8).  Those are
// exactly the inputs of the first stage's butterflies a + 8q; for 128 and 256
// points their outputs are in turn the inputs of the second stage's
// butterflies 4a + k, which leave elements (L/8)a .. (L/8)a + L/8 - 1 in the
// thread.  One exchange through the line's shared buffer (element p at
// p + p/(L/8): the 8 threads' accesses fall in distinct banks) gives thread a
// the inputs of the last stage's butterflies a + 8s, whose outputs are the
// elements a + 8m again.  No block barrier: the 8 threads of a line are a
// quarter of a warp.
//
// A 32-point line (plan 4 8) has 4 threads, thread a the elements a + 4m:
// the inputs of the first stage's butterflies a and a + 4, whose outputs go
// through the exchange to the single radix-8 butterfly a of the last stage.
//
// With 16 threads (256 points: k_dct_lines_reg) thread a holds the elements
// a + 16m: the inputs of four butterflies of the first stage, exchanged those
// of two of the second, exchanged again those of two of the last.
template <int L, int T = L == 32 ? 4 : 8>
struct LineGeo {
    static constexpr int TL = T;      // threads per line
    static constexpr int M = L / TL;  // elements per thread
    static constexpr int BUF = TL == 16 ? L + L / 8 : L + 8;  // exchange buffer elements of a line
    static constexpr int LINES = L >= 256 ? 8 : 16;           // lines per block
    static constexpr int NT = TL * LINES;
};
template <int L, int TL = LineGeo<L>::TL>
__device__ __forceinline__ int xidx(int p) {
    return p + p / (L == 32 || TL == 16 ? 8 : L / 8);
}

// What the exchange waits for: 0 the warp (the threads of a line are
// neighbours), 1 the block (they sit in different warps: the y passes, whose
// lanes run along x for coalesced columns), n > 1 the first n threads of the
// block (the others skip the transform).
template <int SYNC>
__device__ __forceinline__ void line_sync() {
    if constexpr (SYNC == 0)
        __syncwarp();
    else if constexpr (SYNC == 1)
        __syncthreads();
    else
        asm volatile("bar.sync 1, %0;" ::"n"(SYNC) : "memory");
}

template <typename T, bool INV, bool HALF_IN, int L, int SYNC = 0, int TL = LineGeo<L>::TL>
__device__ __forceinline__ void line_fft(Cx<T> (&v)[LineGeo<L, TL>::M], int a, Cx<T>* xs, const Cx<T>* __restrict__ tw) {
    using C = Cx<T>;
    constexpr int M = LineGeo<L, TL>::M;
    if constexpr (L == 32) {
        // stage 1: radix 4, Ns = 1; butterfly a + 4q reads elements a + 4q + 8r, writes 4 (a + 4q) + r
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            C u[4] = {v[q], v[q + 2], v[q + 4], v[q + 6]};
            if constexpr (HALF_IN)
                dft_half<T, 4, INV>(u);
            else
                dft<T, 4, INV>(u);
#pragma unroll
            for (int r = 0; r < 4; ++r) xs[xidx<L, TL>(4 * (a + 4 * q) + r)] = u[r];
        }
        line_sync<SYNC>();
        // last stage: radix 8, Ns = 4, step 1; butterfly a reads and writes elements a + 4r
        C u[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) u[r] = xs[xidx<L, TL>(a + 4 * r)];
#pragma unroll
        for (int r = 1; r < 8; ++r) {
            C t = __ldg(&tw[r * a]);
            if (INV) t.y = -t.y;
            u[r] = cmul(u[r], t);
        }
        dft<T, 8, INV>(u);
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = u[r];
        line_sync<SYNC>();
    } else if constexpr (TL == 16) {
        // stage 1: radix 4, Ns = 1; butterfly j = a + 16q reads elements j + 64r, writes 4j + r
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            C u[4] = {v[q], v[q + 4], v[q + 8], v[q + 12]};
            if constexpr (HALF_IN)
                dft_half<T, 4, INV>(u);
            else
                dft<T, 4, INV>(u);
#pragma unroll
            for (int r = 0; r < 4; ++r) xs[xidx<L, TL>(4 * (a + 16 * q) + r)] = u[r];
        }
        line_sync<SYNC>();
        // stage 2: radix 8, Ns = 4, step 8; butterfly j = a + 16q reads elements j + 32r and
        // writes 32 (j / 4) + j % 4 + 4r, once every butterfly of the line has read
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            C u[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) u[r] = xs[xidx<L, TL>(a + 16 * q + 32 * r)];
#pragma unroll
            for (int r = 1; r < 8; ++r) {
                C t = __ldg(&tw[r * (a % 4) * 8]);
                if (INV) t.y = -t.y;
                u[r] = cmul(u[r], t);
            }
            dft<T, 8, INV>(u);
#pragma unroll
            for (int r = 0; r < 8; ++r) v[q + 2 * r] = u[r];
        }
        line_sync<SYNC>();
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int r = 0; r < 8; ++r) xs[xidx<L, TL>((a + 16 * q) / 4 * 32 + a % 4 + 4 * r)] = v[q + 2 * r];
        line_sync<SYNC>();
        // last stage: radix 8, Ns = 32, step 1; butterfly j = a + 16q reads and writes elements j + 32r
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int j = a + 16 * q;
            C u[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) u[r] = xs[xidx<L, TL>(j + 32 * r)];
#pragma unroll
            for (int r = 1; r < 8; ++r) {
                C t = __ldg(&tw[r * j]);
                if (INV) t.y = -t.y;
                u[r] = cmul(u[r], t);
            }
            dft<T, 8, INV>(u);
#pragma unroll
            for (int r = 0; r < 8; ++r) v[q + 2 * r] = u[r];
        }
        line_sync<SYNC>();
    } else {
        C o[M];  // elements M a + i after the stages before the exchange
        if constexpr (L == 64) {
            // stage 1: radix 8, Ns = 1; butterfly a reads elements a + 8r
            C u[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) u[r] = v[r];
            if constexpr (HALF_IN)
                dft_half<T, 8, INV>(u);
            else
                dft<T, 8, INV>(u);
#pragma unroll
            for (int r = 0; r < 8; ++r) o[r] = u[r];
        } else {
            constexpr int R2 = L == 128 ? 4 : 8;   // second-stage radix
            constexpr int Q = M / 4;                // first-stage butterflies per thread
            C w[Q][4];
            // stage 1: radix 4, Ns = 1; butterfly a + 8q reads elements a + 8q + (L/4) r
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                C u[4];
                u[0] = v[q];
                u[1] = v[q + Q];
                if constexpr (HALF_IN) {
                    dft_half<T, 4, INV>(u);
                } else {
                    u[2] = v[q + 2 * Q];
                    u[3] = v[q + 3 * Q];
                    dft<T, 4, INV>(u);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) w[q][r] = u[r];
            }
            // stage 2: radix R2, Ns = 4, step L / (4 R2) = 8; butterfly 4a + k
            // reads the first stage's outputs 4a + k + (L/R2) r = output k of
            // butterfly a + 8r, and writes elements M a + k + 4r
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                C u[R2];
#pragma unroll
                for (int r = 0; r < R2; ++r) u[r] = w[r][k];
#pragma unroll
                for (int r = 1; r < R2; ++r) {
                    C t = __ldg(&tw[r * k * 8]);
                    if (INV) t.y = -t.y;
                    u[r] = cmul(u[r], t);
                }
                dft<T, R2, INV>(u);
#pragma unroll
                for (int r = 0; r < R2; ++r) o[k + 4 * r] = u[r];
            }
        }
#pragma unroll
        for (int i = 0; i < M; ++i) xs[xidx<L, TL>(M * a + i)] = o[i];
        line_sync<SYNC>();
        // last stage: radix 8, Ns = M, step 1; butterfly j = a + 8s reads
        // elements j + M r and writes them back in place
#pragma unroll
        for (int s2 = 0; s2 < M / 8; ++s2) {
            const int j = a + 8 * s2;
            C u[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) u[r] = xs[xidx<L, TL>(j + M * r)];
#pragma unroll
            for (int r = 1; r < 8; ++r) {
                C t = __ldg(&tw[r * j]);
                if (INV) t.y = -t.y;
                u[r] = cmul(u[r], t);
            }
            dft<T, 8, INV>(u);
#pragma unroll
            for (int r = 0; r < 8; ++r) v[s2 + (M / 8) * r] = u[r];  // element j + M r = a + 8 (s2 + (M/8) r)
        }
        line_sync<SYNC>();  // the buffer is free again
    }
}

}  // namespace
}  // namespace sc
