// sc_fft.cu -- open-boundary Hockney convolution on the doubled grid.
//
// The reference (FFTPoissonSolver.cpp:337-382) zero-pads rho into the doubled
// (2n)^3 grid, multiplies its unnormalised forward transform by that of the
// mirrored integrated Green's function and transforms back with 1/(2n)^3
// (FFT.hpp:726-732, :1706).  Here the same circular convolution is computed
// with batched radix FFTs in shared memory, pruned to the non-zero octant:
//
//   A  z: real -> half spectrum, columns (x<n0, y<n1), 2 real columns per complex FFT
//   B  y: forward, input rows y<n1 only
//   C  x: forward, multiply by the real spectrum of G, inverse; input and
//         output x<n0 only
//   D  y: inverse, outputs y<n1 only
//   E  z: half spectrum -> real, 2 columns per complex FFT, outputs z<n2 only,
//         times normFact (and the cell volume and 1/(4 pi eps0) for the
//         self-field path)
//
// Spectrum layout: spec[kz][ky][kx], kx fastest, kz in [0, n2].
// The mirrored Green's function G2 is even along every axis, so its
// transform is real and is the product of three cosine (DCT-I) transforms of
// G on (n0+1)(n1+1)(n2+1) points; it is built here from G with the same FFT
// stages applied to the even extension of each line.
//
// The staged kernels copy their lines global -> shared with cp.async (all
// copies of a block in flight at once, no register round trip), run Stockham
// radix stages in shared memory and write the pruned output; the k_*_lines
// kernels hold lines of 32 to 256 points in registers (sc_fft_lines.cuh), and
// sc_fft_plane.cu has the y and x passes of a plane in one kernel.  The transform
// lengths of the common meshes (2n = 32, 64, 96, 128, 256) are template
// constants, so the stage loops unroll and the index arithmetic folds; other
// lengths take the same kernels with the length read at run time.
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "sc_exact.cuh"
#include "sc_fft_lines.cuh"

namespace sc {
namespace {

// ---------------------------------------------------------------- cp.async
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
template <typename V>
__device__ __forceinline__ void cp_elem(V* smem, const V* gmem) {
    cp_async<(int)sizeof(V)>(smem, gmem);
}

// ---------------------------------------------------------------- plans
// Radix sequence of a length L = 2^p 3^a 5^b: radix-8 stages for the power of
// two (a remainder of 2 with an 8 becomes 4 x 4, so no radix-2 stage runs
// beside radix 8), then 3s and 5s.  nst = -1 when L has another factor.
struct RadixPlan {
    int nst;
    int r[12];
};
__host__ __device__ constexpr RadixPlan radix_plan(int L) {
    RadixPlan p{0, {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0}};
    if (L < 2) {
        p.nst = -1;
        return p;
    }
    int m = L, twos = 0;
    while (m % 2 == 0) {
        m /= 2;
        ++twos;
    }
    int e8 = twos / 3;
    const int rem = twos % 3;
    if (rem == 1 && e8 > 0) {
        e8 -= 1;
        p.r[p.nst++] = 4;
        p.r[p.nst++] = 4;
    } else if (rem == 1) {
        p.r[p.nst++] = 2;
    } else if (rem == 2) {
        p.r[p.nst++] = 4;
    }
    for (int i = 0; i < e8; ++i) p.r[p.nst++] = 8;
    while (m % 3 == 0 && p.nst < 12) {
        p.r[p.nst++] = 3;
        m /= 3;
    }
    while (m % 5 == 0 && p.nst < 12) {
        p.r[p.nst++] = 5;
        m /= 5;
    }
    if (m != 1) p.nst = -1;
    return p;
}
__host__ __device__ constexpr int min_radix(int L) {
    const RadixPlan p = radix_plan(L);
    int r = 16;
    for (int i = 0; i < p.nst; ++i) r = p.r[i] < r ? p.r[i] : r;
    return r;
}
// Complex transforms per block for a template length: the widest stage
// (L / min radix butterflies per transform) fills at most 256 threads, and
// at most 16 transforms share a block.  Length 0 (read at run time): 16.
__host__ __device__ constexpr int cols_for(int LT) {
    if (LT == 0) return 16;
    const int per = LT / min_radix(LT);
    int nc = 256 / per;
    if (nc > 16) nc = 16;
    if (nc < 1) nc = 1;
    return nc;
}
__host__ __device__ constexpr int threads_for(int LT) {
    if (LT == 0) return 256;
    const int t = cols_for(LT) * (LT / min_radix(LT));
    return t < 32 ? 32 : t;
}

// Shared-memory position of element i of a column: one empty slot after every
// 8 elements.  The first Stockham stages write with strides of R elements
// (R = 4 or 8, i.e. 64 or 128 bytes of complex double), which would put a
// warp's stores into one or two bank groups; the skew spreads them over all.
__host__ __device__ constexpr int sk(int i) { return i + (i >> 3); }

// One Stockham autosort butterfly (radix R): butterfly j of a column reads
// element j + r nb, r < R, applies the twiddles W^(r k step), k = j mod Ns,
// and writes element (j / Ns) Ns R + k + r Ns (positions through sk()).
// NZ < R: inputs r >= NZ are known zeros (NZ = R/2 only); NO < R: only
// outputs r < NO are needed; FIRST: Ns = 1, all twiddles are 1.
template <typename T, int R, bool INV, int NZ = R, int NO = R, bool FIRST = false>
__device__ __forceinline__ void butterfly(const Cx<T>* __restrict__ src, Cx<T>* __restrict__ dst, int j, int nb, int Ns,
                                          int step, const Cx<T>* __restrict__ tw) {
    using C = Cx<T>;
    static_assert(NZ == R || (2 * NZ == R && FIRST), "zero inputs only in a first stage");
    C v[R];
#pragma unroll
    for (int r = 0; r < NZ; ++r) v[r] = src[sk(j + r * nb)];
    const int k = FIRST ? 0 : j % Ns;
    if constexpr (!FIRST) {
#pragma unroll
        for (int r = 1; r < R; ++r) {
            C t = tw[r * k * step];
            if (INV) t.y = -t.y;
            v[r] = cmul(v[r], t);
        }
    }
    if constexpr (NZ == R)
        dft<T, R, INV>(v);
    else
        dft_half<T, R, INV>(v);
    const int base = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int r = 0; r < NO; ++r) dst[sk(base + r * Ns)] = v[r];
}

// Column stride: the L skewed elements (sk(L - 1) < L + L/8) plus one, so
// that the columns of a block also start in different banks.
__host__ __device__ constexpr int col_stride(int L) { return L + (L >> 3) + 1; }

// Pruning of a transform whose length is a template constant:
//   kPruneNone  full transform;
//   kPruneIn    the upper half of the input is zero (forward transforms of
//               the zero-padded doubled grid): the first stage reads half;
//   kPruneOut   only the lower half of the output is used (inverse
//               transforms back to the physical octant): the last stage
//               writes half.
constexpr int kPruneNone = 0, kPruneIn = 1, kPruneOut = 2;

// compile-time stage: length L, Ns, NC columns, NT threads
template <typename T, int R, bool INV, int L, int NS, int NC, int NT, int NZ, int NO>
__device__ __forceinline__ void stage_c(const Cx<T>* in, Cx<T>* out, const Cx<T>* tw) {
    constexpr int NB = L / R;
    constexpr int STEP = L / (NS * R);
    constexpr int CS = col_stride(L);
#pragma unroll
    for (int w0 = 0; w0 < NC * NB; w0 += NT) {
        const int w = w0 + (int)threadIdx.x;
        if ((NC * NB) % NT != 0 && w >= NC * NB) break;
        const int col = w / NB;
        const int j = w - col * NB;
        butterfly<T, R, INV, NZ, NO, NS == 1>(in + col * CS, out + col * CS, j, NB, NS, STEP, tw);
    }
}

template <typename T, bool INV, int L, int S, int NS, int NC, int NT, int PR>
__device__ __forceinline__ Cx<T>* stages_c(Cx<T>* a, Cx<T>* b, const Cx<T>* tw) {
    constexpr RadixPlan P = radix_plan(L);
    if constexpr (S == P.nst) {
        return a;
    } else {
        constexpr int R = P.r[S];
        constexpr bool even = R % 2 == 0;
        constexpr int NZ = (PR == kPruneIn && S == 0 && even && R <= 8) ? R / 2 : R;
        constexpr int NO = (PR == kPruneOut && S == P.nst - 1 && even) ? R / 2 : R;
        stage_c<T, R, INV, L, NS, NC, NT, NZ, NO>(a, b, tw);
        __syncthreads();
        return stages_c<T, INV, L, S + 1, NS * R, NC, NT, PR>(b, a, tw);
    }
}

// run-time stage (lengths without a template instance)
template <typename T, int R, bool INV>
__device__ __forceinline__ void stage_r(const Cx<T>* in, Cx<T>* out, int L, int Ns, int ncols, const Cx<T>* tw) {
    const int nb = L / R;
    const int step = L / (Ns * R);
    const int cs = col_stride(L);
    for (int w = threadIdx.x; w < ncols * nb; w += blockDim.x) {
        const int col = w / nb;
        const int j = w - col * nb;
        butterfly<T, R, INV>(in + col * cs, out + col * cs, j, nb, Ns, step, tw);
    }
}

// Complex FFT of NC columns (element i of column col at buf[col * col_stride(L) + sk(i)]); returns the buffer holding
// the result (buf or tmp).  The caller synchronises before the call.
// With a template length the transform is pruned as PR says (the caller
// then stages only the nonzero half, or reads only the lower half); with a
// run-time length it is always full.
template <typename T, bool INV, int LT, int NC, int NT, int PR = kPruneNone>
__device__ __forceinline__ Cx<T>* block_fft(Cx<T>* buf, Cx<T>* tmp, const FftPlan& pl, const Cx<T>* tw) {
    if constexpr (LT > 0) {
        return stages_c<T, INV, LT, 0, 1, NC, NT, PR>(buf, tmp, tw);
    } else {
        int Ns = 1;
        Cx<T>* a = buf;
        Cx<T>* b = tmp;
        for (int s = 0; s < pl.nst; ++s) {
            const int R = pl.r[s];
            if (R == 8)
                stage_r<T, 8, INV>(a, b, pl.L, Ns, NC, tw);
            else if (R == 4)
                stage_r<T, 4, INV>(a, b, pl.L, Ns, NC, tw);
            else if (R == 2)
                stage_r<T, 2, INV>(a, b, pl.L, Ns, NC, tw);
            else if (R == 3)
                stage_r<T, 3, INV>(a, b, pl.L, Ns, NC, tw);
            else
                stage_r<T, 5, INV>(a, b, pl.L, Ns, NC, tw);
            __syncthreads();
            Cx<T>* t = a;
            a = b;
            b = t;
            Ns *= R;
        }
        return a;
    }
}

template <typename V, int NT>
__device__ __forceinline__ void stage_twiddles(V* dst, const V* __restrict__ src, int L) {
    for (int e = threadIdx.x; e < L; e += NT) cp_elem(dst + e, src + e);
}

// elements of one tile: twiddles (L), buf and tmp (NC col_stride(L) + 2 NC each)
__host__ __device__ constexpr size_t tile_elems(int L, int nc) {
    return (size_t)L + 2 * ((size_t)nc * col_stride(L) + 2 * nc);
}

// ---------------------------------------------------------------- pass A
// 2 NC real columns (x) of one y per block, packed two per complex FFT.
// FULL: the z transform covers the data without zero padding (periodic z,
// L2 = n2); otherwise L2 = 2 n2 and the upper half is zero.  The half
// spectrum has L2/2 + 1 entries either way.
template <typename T, int LT, int NC, int NT, bool FULL = false>
__device__ __forceinline__ void fft_z_r2c_body(const T* __restrict__ rho, Cx<T>* __restrict__ spec, int n0, int n1, int n2,
                                               int L0, int L1, const FftPlan& pz, const Cx<T>* __restrict__ twz, int bx,
                                               int by) {
    using C = Cx<T>;
    constexpr int RC = 2 * NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L2 = LT > 0 ? LT : pz.L;
    const int CS = col_stride(L2);
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* buf = tw + L2;
    C* tmp = buf + NC * CS + RC;
    stage_twiddles<C, NT>(tw, twz, L2);
    const int y = by;
    const int x0 = bx * RC;
    for (int e = threadIdx.x; e < RC * (LT > 0 ? n2 : L2); e += NT) {  // the zero half is not staged when pruned
        const int xi = e % RC, z = e / RC;
        const int x = x0 + xi;
        T* slot = reinterpret_cast<T*>(&buf[(xi >> 1) * CS + sk(z)]) + (xi & 1);
        if (z < n2 && x < n0)
            cp_elem(slot, &rho[((size_t)z * n1 + y) * n0 + x]);
        else
            *slot = (T)0;
    }
    cp_async_wait_all();
    __syncthreads();
    const C* out = block_fft<T, false, LT, NC, NT, FULL ? kPruneNone : kPruneIn>(buf, tmp, pz, tw);
    const int K = L2 / 2;
    for (int e = threadIdx.x; e < RC * (K + 1); e += NT) {
        const int xi = e % RC, k = e / RC;
        const int x = x0 + xi;
        if (x >= n0) continue;
        const int q = xi >> 1;
        const C Z = out[q * CS + sk(k)];
        const C Zm = out[q * CS + sk(k == 0 ? 0 : L2 - k)];
        C r;
        if ((xi & 1) == 0)
            r = C{(T)0.5 * (Z.x + Zm.x), (T)0.5 * (Z.y - Zm.y)};
        else
            r = C{(T)0.5 * (Z.y + Zm.y), (T)-0.5 * (Z.x - Zm.x)};
        spec[((size_t)k * L1 + y) * L0 + x] = r;
    }
}
template <typename T, int LT, int NC, int NT, bool FULL = false>
__global__ void __launch_bounds__(NT, 1024 / NT) k_fft_z_r2c(const T* __restrict__ rho, Cx<T>* __restrict__ spec, int n0, int n1, int n2,
                                                  int L0, int L1, FftPlan pz, const Cx<T>* __restrict__ twz) {
    fft_z_r2c_body<T, LT, NC, NT, FULL>(rho, spec, n0, n1, n2, L0, L1, pz, twz, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------- pass B / D
// NC x-columns of one kz plane per block; rows y < n_in in, y < n_out out.
template <typename T, bool INV, int LT, int NC, int NT>
__device__ __forceinline__ void fft_y_body(Cx<T>* __restrict__ spec, int n0, int L0, int n_in, int n_out, const FftPlan& py,
                                           const Cx<T>* __restrict__ twy, int bx, int by) {
    using C = Cx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L1 = LT > 0 ? LT : py.L;
    const int CS = col_stride(L1);
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* buf = tw + L1;
    C* tmp = buf + NC * CS + 2 * NC;
    stage_twiddles<C, NT>(tw, twy, L1);
    const int kz = by;
    const int x0 = bx * NC;
    C* plane = spec + (size_t)kz * L1 * L0;
    for (int e = threadIdx.x; e < NC * ((LT > 0 && !INV) ? n_in : L1); e += NT) {
        const int xi = e % NC, yy = e / NC;
        const int x = x0 + xi;
        C* slot = &buf[xi * CS + sk(yy)];
        if (yy < n_in && x < n0)
            cp_elem(slot, &plane[(size_t)yy * L0 + x]);
        else
            *slot = C{(T)0, (T)0};
    }
    cp_async_wait_all();
    __syncthreads();
    const C* out = block_fft<T, INV, LT, NC, NT, INV ? kPruneOut : kPruneIn>(buf, tmp, py, tw);
    for (int e = threadIdx.x; e < NC * n_out; e += NT) {
        const int xi = e % NC, yy = e / NC;
        const int x = x0 + xi;
        if (x < n0) plane[(size_t)yy * L0 + x] = out[xi * CS + sk(yy)];
    }
}
template <typename T, bool INV, int LT, int NC, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_fft_y(Cx<T>* __restrict__ spec, int n0, int L0, int n_in, int n_out, FftPlan py,
                                              const Cx<T>* __restrict__ twy) {
    fft_y_body<T, INV, LT, NC, NT>(spec, n0, L0, n_in, n_out, py, twy, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------- pass C
// The forward transform and the multiplication run in TI, the inverse in TO.
// The mixed form takes TI = float, TO = double: rounding in the forward half
// is white noise in the spectrum, which the derivative of phi does not
// amplify, while rounding after the multiplication would be noise relative
// to phi itself and is kept at FP64.  `in` and `out` alias in the plain form;
// every block reads its rows before it writes them.
//
// CG: ghat holds complex values (the image charge's shifted G is not even in
// z, FFTPoissonSolver.cpp:316); the product is the complex one.
template <typename TI, typename TO, int LT, int NC, int NT, bool CG = false>
__device__ __forceinline__ void fft_x_conv_body(const Cx<TI>* in, Cx<TO>* out, const TI* __restrict__ ghat, int n0, int n1,
                                                int L1, int rows, const FftPlan& px, const Cx<TI>* __restrict__ twi,
                                                const Cx<TO>* __restrict__ two, int bx) {
    using CI = Cx<TI>;
    using CO = Cx<TO>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L0 = LT > 0 ? LT : px.L;
    const int CS = col_stride(L0);
    CO* tw_o = reinterpret_cast<CO*>(smem_raw);
    CI* tw_i = reinterpret_cast<CI*>(tw_o + L0);
    CO* bufo = reinterpret_cast<CO*>(tw_i + L0);
    CO* tmpo = bufo + NC * CS;
    stage_twiddles<CO, NT>(tw_o, two, L0);
    stage_twiddles<CI, NT>(tw_i, twi, L0);
    CI* bufi = reinterpret_cast<CI*>(bufo);
    CI* tmpi = reinterpret_cast<CI*>(tmpo);
    const int r0 = bx * NC;
    const int xs = LT > 0 ? n0 : L0;  // staged length: the zero half is not staged when pruned
    for (int e = threadIdx.x; e < NC * xs; e += NT) {
        const int ri = e / xs, x = e - ri * xs;
        const int r = r0 + ri;
        CI* slot = &bufi[ri * CS + sk(x)];
        if (r < rows && x < n0)
            cp_elem(slot, &in[(size_t)r * L0 + x]);
        else
            *slot = CI{(TI)0, (TI)0};
    }
    cp_async_wait_all();
    __syncthreads();
    const CI* f = block_fft<TI, false, LT, NC, NT, kPruneIn>(bufi, tmpi, px, tw_i);
    CO* g = (f == bufi) ? tmpo : bufo;
    CO* h = (f == bufi) ? bufo : tmpo;
    for (int e = threadIdx.x; e < NC * L0; e += NT) {
        const int ri = e / L0, kx = e - ri * L0;
        const int r = r0 + ri;
        if (r >= rows) continue;
        const int kz = r / L1;
        const int ky = r - kz * L1;
        const int gy = ky <= n1 ? ky : L1 - ky;
        const int gx = kx <= n0 ? kx : L0 - kx;
        const size_t gi = ((size_t)kz * (n1 + 1) + gy) * (n0 + 1) + gx;
        const CI v = f[ri * CS + sk(kx)];
        if constexpr (CG) {
            const CI gc = reinterpret_cast<const CI*>(ghat)[gi];
            g[ri * CS + sk(kx)] = CO{(TO)(v.x * gc.x - v.y * gc.y), (TO)(v.x * gc.y + v.y * gc.x)};
        } else {
            const TI gv = ghat[gi];
            g[ri * CS + sk(kx)] = CO{(TO)(v.x * gv), (TO)(v.y * gv)};
        }
    }
    __syncthreads();
    const CO* o = block_fft<TO, true, LT, NC, NT, kPruneOut>(g, h, px, tw_o);
    for (int e = threadIdx.x; e < NC * n0; e += NT) {
        const int ri = e / n0, x = e - ri * n0;
        const int r = r0 + ri;
        if (r < rows) out[(size_t)r * L0 + x] = o[ri * CS + sk(x)];
    }
}
template <typename TI, typename TO, int LT, int NC, int NT, bool CG = false>
__global__ void __launch_bounds__(NT, 1024 / NT) k_fft_x_conv(const Cx<TI>* in, Cx<TO>* out, const TI* __restrict__ ghat, int n0, int n1,
                                                   int L1, int rows, FftPlan px, const Cx<TI>* __restrict__ twi,
                                                   const Cx<TO>* __restrict__ two) {
    fft_x_conv_body<TI, TO, LT, NC, NT, CG>(in, out, ghat, n0, n1, L1, rows, px, twi, two, blockIdx.x);
}

// Pass C on rows of L = 2 n0 points: TL threads per row.  The forward
// transform leaves each thread the spectrum at a + TL m, exactly the inputs
// the inverse transform's first stages need from it.
template <typename TI, typename TO, bool CG, int L>
__device__ __forceinline__ void fft_x_conv_lines_body(const Cx<TI>* in, Cx<TO>* out, const TI* __restrict__ ghat, int n0,
                                                      int n1, int L1, int rows, const Cx<TI>* __restrict__ twi,
                                                      const Cx<TO>* __restrict__ two, int blk) {
    using CI = Cx<TI>;
    using CO = Cx<TO>;
    using G = LineGeo<L>;
    constexpr int M = G::M;
    __shared__ __align__(16) CO xbuf[G::LINES][G::BUF];
    const int li = threadIdx.x / G::TL, a = threadIdx.x % G::TL;
    const int r = blk * G::LINES + li;
    const bool live = r < rows;
    CI v[M];
#pragma unroll
    for (int m = 0; m < M; ++m)
        v[m] = (live && m < M / 2) ? in[(size_t)r * L + a + G::TL * m] : CI{(TI)0, (TI)0};
    const int kz = live ? r / L1 : 0;
    const int ky = live ? r - kz * L1 : 0;
    const int gy = ky <= n1 ? ky : L1 - ky;
    const size_t grow = ((size_t)kz * (n1 + 1) + gy) * (n0 + 1);
    // the row of G's spectrum is fetched before the forward transform, so its
    // latency hides behind the transform
    using GV = typename std::conditional<CG, CI, TI>::type;
    GV g[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int kx = a + G::TL * m;
        const int gx = kx <= n0 ? kx : L - kx;
        g[m] = live ? reinterpret_cast<const GV*>(ghat)[grow + gx] : GV{};
    }
    line_fft<TI, false, true, L>(v, a, reinterpret_cast<CI*>(xbuf[li]), twi);
    CO w[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const CI f = v[m];
        if constexpr (CG) {
            const CI gc = g[m];
            w[m] = CO{(TO)(f.x * gc.x - f.y * gc.y), (TO)(f.x * gc.y + f.y * gc.x)};
        } else {
            const TI gv = g[m];
            w[m] = CO{(TO)(f.x * gv), (TO)(f.y * gv)};
        }
    }
    line_fft<TO, true, false, L>(w, a, xbuf[li], two);
    if (!live) return;
#pragma unroll
    for (int m = 0; m < M / 2; ++m) out[(size_t)r * L + a + G::TL * m] = w[m];  // x < n0
}

template <typename TI, typename TO, bool CG, int L>
__global__ void __launch_bounds__(LineGeo<L>::NT) k_fft_x_conv_lines(const Cx<TI>* in, Cx<TO>* out,
                                                                   const TI* __restrict__ ghat, int n0, int n1, int L1,
                                                                   int rows, const Cx<TI>* __restrict__ twi,
                                                                   const Cx<TO>* __restrict__ two) {
    fft_x_conv_lines_body<TI, TO, CG, L>(in, out, ghat, n0, n1, L1, rows, twi, two, blockIdx.x);
}

// Passes B (forward, inputs y < L/2) and D (inverse, outputs y < L/2) on
// columns of L points along y: TL threads per column (in different warps),
// consecutive x of one plane per block.
// FP64 columns of 256 points take 16 threads of 128 registers: with 8 of 186
// pass D had 7 warps per SM waiting for its columns (issue 16 %).  128^3 step
// 903 -> 901 us, mixed 702 -> 694.
template <typename T, int L>
using YGeo = LineGeo<L, L == 256 && sizeof(T) == sizeof(double) ? 16 : LineGeo<L>::TL>;
template <typename T, int L>
constexpr int kYBlocks = YGeo<T, L>::TL == 16 ? 4 : 1;  // 128 registers with 16 threads per line

template <typename T, bool INV, int L>
__device__ __forceinline__ void fft_y_lines_body(Cx<T>* __restrict__ spec, int n0, int L0, int planes,
                                                 const Cx<T>* __restrict__ twy, int bx, int kz) {
    using C = Cx<T>;
    using G = YGeo<T, L>;
    constexpr int M = G::M;
    // lanes run along x (thread li + LINES a: column li, part a), so a warp
    // reads and writes whole rows of consecutive columns; the line buffers
    // are G::BUF + 1 apart, so the lines of one access fall in distinct banks
    __shared__ __align__(16) C xbuf[G::LINES][G::BUF + 1];
    const int li = threadIdx.x % G::LINES, a = threadIdx.x / G::LINES;
    const int x = bx * G::LINES + li;
    const bool live = kz < planes && x < n0;
    C* col = spec + ((size_t)kz * L + a) * L0 + (live ? x : 0);
    const unsigned step = (unsigned)(G::TL * L0);
    C v[M];
#pragma unroll
    for (int m = 0; m < M; ++m)
        v[m] = (live && (INV || m < M / 2)) ? col[(unsigned)m * step] : C{(T)0, (T)0};
    line_fft<T, INV, !INV, L, true, G::TL>(v, a, xbuf[li], twy);
    if (!live) return;
    constexpr int MO = INV ? M / 2 : M;  // D keeps y < L/2
#pragma unroll
    for (int m = 0; m < MO; ++m) col[(unsigned)m * step] = v[m];
}

template <typename T, bool INV, int L>
__global__ void __launch_bounds__(YGeo<T, L>::NT, kYBlocks<T, L>) k_fft_y_lines(Cx<T>* __restrict__ spec, int n0, int L0, int planes,
                                                              const Cx<T>* __restrict__ twy) {
    fft_y_lines_body<T, INV, L>(spec, n0, L0, planes, twy, blockIdx.x, blockIdx.y);
}

// Pass A on z lines of L = 2 n2 points: two real columns (x, x + 1) of one y
// per complex line, TL threads per line with the lanes along x (consecutive
// column pairs, so a warp reads and writes whole rows) and block-level
// exchanges.  The two half spectra need Z[k] and Z[L - k], which sit in
// different threads: the transformed line goes through its buffer once more.
//
// ACC: the charge density is formed here from the deposit's accumulators
// (k_assemble_rho: the same values, rho stored, the accumulators cleared), which
// saves a launch of the small meshes where launches are what the step waits
// for (fft_assembles).
struct AccIn {
    ulonglong2* acc;
    const StepState* st;
    double dT, rdT;
    int weights;
};
template <typename T, int L, bool ACC = false>
__global__ void __launch_bounds__(LineGeo<L>::NT) k_fft_z_r2c_lines(T* __restrict__ rho, Cx<T>* __restrict__ spec,
                                                                  int n0, int n1, int L0, int L1,
                                                                  const Cx<T>* __restrict__ twz, AccIn in) {
    using C = Cx<T>;
    using G = LineGeo<L>;
    constexpr int M = G::M, K = L / 2;
    __shared__ __align__(16) C xbuf[G::LINES][G::BUF + 1];
    const int li = threadIdx.x % G::LINES, a = threadIdx.x / G::LINES;
    const int np = (n0 + 1) / 2;
    const int line = blockIdx.x * G::LINES + li;
    const int y = line / np, x = 2 * (line - y * np);
    const bool live = y < n1;
    const bool odd = live && x + 1 < n0;
    C v[M];
    double unit = 0.0, tmp2 = 0.0;
    if constexpr (ACC) {
        unit = in.weights ? in.st->qdt * 0x1p-26 : in.st->dep_unit;
        tmp2 = in.st->tmp2;
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        v[m] = C{(T)0, (T)0};
        if (live && m < M / 2) {
            const size_t c = ((size_t)(a + G::TL * m) * n1 + y) * n0 + x;
            if constexpr (ACC) {
                v[m].x = (T)node_density(in.acc[c], unit, in.dT, in.rdT, tmp2);
                rho[c] = v[m].x;
                in.acc[c] = make_ulonglong2(0ull, 0ull);
                if (odd) {
                    v[m].y = (T)node_density(in.acc[c + 1], unit, in.dT, in.rdT, tmp2);
                    rho[c + 1] = v[m].y;
                    in.acc[c + 1] = make_ulonglong2(0ull, 0ull);
                }
            } else {
                v[m].x = rho[c];
                if (odd) v[m].y = rho[c + 1];
            }
        }
    }
    C* xs = xbuf[li];
    line_fft<T, false, true, L, true>(v, a, xs, twz);
#pragma unroll
    for (int m = 0; m < M; ++m) xs[xidx<L>(a + G::TL * m)] = v[m];
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int m = 0; m <= M / 2; ++m) {
        const int k = a + G::TL * m;
        if (k > K) break;
        const C Z = xs[xidx<L>(k)];
        const C Zm = xs[xidx<L>(k == 0 ? 0 : L - k)];
        C* dst = spec + ((size_t)k * L1 + y) * L0 + x;
        dst[0] = C{(T)0.5 * (Z.x + Zm.x), (T)0.5 * (Z.y - Zm.y)};
        if (odd) dst[1] = C{(T)0.5 * (Z.y + Zm.y), (T)-0.5 * (Z.x - Zm.x)};
    }
}

// ---------------------------------------------------------------- pass E
// FLIP: the image potential is read back with z flipped,
// rho[i][j][k] = rho2[i][j][n2 - k - 1] (FFTPoissonSolver.cpp:322-326).
// FULL: all L2 = n2 outputs of an unpadded (periodic) z transform.
template <typename T, bool SELF, int LT, int NC, int NT, bool FLIP = false, bool FULL = false>
__device__ __forceinline__ void fft_z_c2r_body(const Cx<T>* __restrict__ spec, double* __restrict__ phi, int n0, int n1,
                                               int n2, int L0, int L1, const FftPlan& pz, const Cx<T>* __restrict__ twz,
                                               const StepState* __restrict__ st, double normFact, double coupling, int bx,
                                               int by) {
    using C = Cx<T>;
    constexpr int RC = 2 * NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L2 = LT > 0 ? LT : pz.L;
    const int CS = col_stride(L2);
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* buf = tw + L2;
    C* tmp = buf + NC * CS + RC;
    stage_twiddles<C, NT>(tw, twz, L2);
    const int y = by;
    const int x0 = bx * RC;
    // the half spectra of the 2 NC columns in tmp: [xi][k], k <= K = L2 / 2
    const int K = L2 / 2;
    for (int e = threadIdx.x; e < RC * (K + 1); e += NT) {
        const int xi = e % RC, k = e / RC;
        const int x = x0 + xi;
        C* slot = &tmp[xi * (K + 1) + k];
        if (x < n0)
            cp_elem(slot, &spec[((size_t)k * L1 + y) * L0 + x]);
        else
            *slot = C{(T)0, (T)0};
    }
    cp_async_wait_all();
    __syncthreads();
    for (int e = threadIdx.x; e < NC * L2; e += NT) {
        const int q = e / L2, k = e - q * L2;
        const C* A = tmp + (2 * q) * (K + 1);
        const C* B = tmp + (2 * q + 1) * (K + 1);
        C z;
        if (k <= K) {
            C a = A[k], b = B[k];
            if (k == 0 || k == K) {  // the half-complex format holds no imaginary part there
                a.y = (T)0;
                b.y = (T)0;
            }
            z = C{a.x - b.y, a.y + b.x};
        } else {
            const C a = A[L2 - k], b = B[L2 - k];
            z = C{a.x + b.y, b.x - a.y};
        }
        buf[q * CS + sk(k)] = z;
    }
    __syncthreads();
    const C* out = block_fft<T, true, LT, NC, NT, FULL ? kPruneNone : kPruneOut>(buf, tmp, pz, tw);
    const double hvol = SELF ? st->hvol : 1.0;
    for (int e = threadIdx.x; e < RC * n2; e += NT) {
        const int xi = e % RC, zz = e / RC;
        const int x = x0 + xi;
        if (x >= n0) continue;
        const C v = out[(xi >> 1) * CS + sk(zz)];
        double r = (double)((xi & 1) ? v.y : v.x);
        r = r * normFact;
        if (SELF) {
            r = r * hvol;
            r = r * coupling;
        }
        phi[((size_t)(FLIP ? n2 - 1 - zz : zz) * n1 + y) * n0 + x] = r;
    }
}
template <typename T, bool SELF, int LT, int NC, int NT, bool FLIP = false, bool FULL = false>
__global__ void __launch_bounds__(NT, 1024 / NT) k_fft_z_c2r(const Cx<T>* __restrict__ spec, double* __restrict__ phi, int n0, int n1,
                                                  int n2, int L0, int L1, FftPlan pz, const Cx<T>* __restrict__ twz,
                                                  const StepState* __restrict__ st, double normFact, double coupling) {
    fft_z_c2r_body<T, SELF, LT, NC, NT, FLIP, FULL>(spec, phi, n0, n1, n2, L0, L1, pz, twz, st, normFact, coupling,
                                                    blockIdx.x, blockIdx.y);
}

// Pass E on z lines of L = 2 n2 points (as k_fft_z_r2c_lines backwards): two
// half spectra (x, x + 1) of one y per complex line, lanes along x; thread a
// packs the elements k = a + TL m <= L/2 and their mirrors through the line's
// buffer, so each spectrum entry is read once.  The staged form moves the tile
// through shared memory at every stage (75 % of the L1 throughput at 256
// points).  Convolution phase, staged -> this: 128^3 152.3 -> 143.0 us (mixed
// 133.6 -> 122.9), 64^3 32.8 -> 31.8 (29.8 -> 28.7).  At 32 and 64 points the
// step does not move and the staged form stays.
template <int L>
using ZLine = LineGeo<L, L == 256 ? 16 : 8>;
template <bool SELF, int L, bool FLIP>
__global__ void __launch_bounds__(ZLine<L>::NT, L == 256 ? 4 : 1)
    k_fft_z_c2r_lines(const double2* __restrict__ spec, double* __restrict__ phi, int n0, int n1, int L0, int L1,
                      const double2* __restrict__ twz, const StepState* __restrict__ st, double normFact,
                      double coupling) {
    using G = ZLine<L>;
    constexpr int M = G::M, TL = G::TL, K = L / 2, LINES = G::LINES;
    __shared__ __align__(16) double2 xbuf[LINES][G::BUF + 1];
    const int li = threadIdx.x % LINES, a = threadIdx.x / LINES;
    const int np = (n0 + 1) / 2;
    const int line = blockIdx.x * LINES + li;
    const int y = line / np, x = 2 * (line - y * np);
    const bool live = y < n1;
    const bool odd = live && x + 1 < n0;
    double2* xs = xbuf[li];
    const double2* src = spec + (live ? (size_t)y * L0 + x : 0);
    const size_t plane = (size_t)L1 * L0;
#pragma unroll
    for (int m = 0; m <= M / 2; ++m) {
        const int k = a + TL * m;
        if (m < M / 2 || a == 0) {
            double2 A = live ? src[k * plane] : double2{0.0, 0.0};
            double2 B = odd ? src[k * plane + 1] : double2{0.0, 0.0};
            if (k == 0 || k == K) A.y = B.y = 0.0;  // the half-complex format holds no imaginary part there
            xs[xidx<L, TL>(k)] = double2{A.x - B.y, A.y + B.x};
            if (k > 0 && k < K) xs[xidx<L, TL>(L - k)] = double2{A.x + B.y, B.x - A.y};
        }
    }
    __syncthreads();
    double2 v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = xs[xidx<L, TL>(a + TL * m)];
    __syncthreads();
    line_fft<double, true, false, L, 1, TL>(v, a, xs, twz);
    if (!live) return;
    const double hvol = SELF ? st->hvol : 1.0;
#pragma unroll
    for (int m = 0; m < M / 2; ++m) {
        const int zz = a + TL * m;
        double re = v[m].x * normFact, im = v[m].y * normFact;
        if (SELF) {
            re = re * hvol * coupling;
            im = im * hvol * coupling;
        }
        double* o = phi + ((size_t)(FLIP ? K - 1 - zz : zz) * n1 + y) * n0 + x;
        o[0] = re;
        if (odd) o[1] = im;
    }
}

// ---------------------------------------------------------------- G spectrum
// Cosine transform of every line along one axis: Y[m] = sum over the even
// extension (length L = 2(len-1)) of g, m in [0, len-1].  Lines are addressed
// as in[b * sb + o * so + e * se]; 2 NC lines per block (two per complex FFT).
// FROM_TMP (the z lines, b = x, o = y, e = z): in is the IGF antiderivative
// on the (t0 = n0+2) x (t1 = n1+2) grid and each element of G is formed from
// it as it is staged (igf_G_at), so G itself is never stored.
template <typename TO, int LT, int NC, int NT, bool FROM_TMP = false>
__device__ __forceinline__ void dct_lines_body(const double* __restrict__ in, TO* __restrict__ out, int len, int nb,
                                               long long sb, long long so, long long se, const FftPlan& pl,
                                               const double2* __restrict__ twd, int bx, int by, int t0 = 0,
                                               int t1 = 0) {
    constexpr int RC = 2 * NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = LT > 0 ? LT : pl.L;
    const int CS = col_stride(L);
    double2* tw = reinterpret_cast<double2*>(smem_raw);
    double2* buf = tw + L;
    double2* tmp = buf + NC * CS + RC;
    stage_twiddles<double2, NT>(tw, twd, L);
    const int b0 = bx * RC;
    const long long obase = (long long)by * so;
    for (int e = threadIdx.x; e < RC * len; e += NT) {
        const int li = e % RC, m = e / RC;
        const int b = b0 + li;
        double* slot = reinterpret_cast<double*>(&buf[(li >> 1) * CS + sk(m)]) + (li & 1);
        const bool inner = m >= 1 && m <= len - 2;
        double* mir = reinterpret_cast<double*>(&buf[(li >> 1) * CS + sk(inner ? L - m : m)]) + (li & 1);
        if (b < nb) {
            if constexpr (FROM_TMP) {
                const double v = igf_G_at(in, t0, t1, b, by, m);
                *slot = v;
                if (inner) *mir = v;
            } else {
                const double* src = in + (long long)b * sb + obase + (long long)m * se;
                cp_elem(slot, src);
                if (inner) cp_elem(mir, src);
            }
        } else {
            *slot = 0.0;
            if (inner) *mir = 0.0;
        }
    }
    cp_async_wait_all();
    __syncthreads();
    const double2* o = block_fft<double, false, LT, NC, NT>(buf, tmp, pl, tw);
    for (int e = threadIdx.x; e < RC * len; e += NT) {
        const int li = e % RC, m = e / RC;
        const int b = b0 + li;
        if (b >= nb) continue;
        const double2 v = o[(li >> 1) * CS + sk(m)];
        out[(long long)b * sb + obase + (long long)m * se] = (TO)((li & 1) ? v.y : v.x);
    }
}
template <typename TO, int LT, int NC, int NT, bool FROM_TMP = false>
__global__ void __launch_bounds__(NT, 1024 / NT) k_dct_lines(const double* __restrict__ in, TO* __restrict__ out, int len, int nb,
                                                  long long sb, long long so, long long se, FftPlan pl,
                                                  const double2* __restrict__ twd, int t0, int t1) {
    dct_lines_body<TO, LT, NC, NT, FROM_TMP>(in, out, len, nb, sb, so, se, pl, twd, blockIdx.x, blockIdx.y, t0, t1);
}

// The same cosine transforms for 256-point extensions with the
// register-resident line transform: two real lines per complex line (lines
// 2p and 2p + 1 as its real and imaginary parts, as in dct_lines_body), 16
// threads per complex line with the lanes along p, so one access reads
// consecutive lines; thread a holds the extension's elements a + TL m.  The
// butterflies, twiddles and operation order are block_fft's, so Ĝ has the
// same bits.
template <typename TO, int L>
__global__ void __launch_bounds__(LineGeo<L, 16>::NT, 4) k_dct_lines_reg(const double* __restrict__ in, TO* __restrict__ out,
                                                                 int len, int nb, long long sb, long long so,
                                                                 long long se, const double2* __restrict__ twd) {
    using C = Cx<double>;
    using G = LineGeo<L, 16>;
    constexpr int M = G::M;
    __shared__ __align__(16) C xbuf[G::LINES][G::BUF + 1];
    const int li = threadIdx.x % G::LINES, a = threadIdx.x / G::LINES;
    const int p = blockIdx.x * G::LINES + li;
    const int b0 = 2 * p, b1 = 2 * p + 1;
    const long long obase = (long long)blockIdx.y * so;
    C v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int e = a + G::TL * m;
        const long long src = e <= L / 2 ? e : L - e;  // the even extension
        const double re = b0 < nb ? in[(long long)b0 * sb + obase + src * se] : 0.0;
        const double im = b1 < nb ? in[(long long)b1 * sb + obase + src * se] : 0.0;
        v[m] = C{re, im};
    }
    line_fft<double, false, false, L, true, 16>(v, a, xbuf[li], reinterpret_cast<const C*>(twd));
    if (b0 >= nb) return;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int e = a + G::TL * m;
        if (e < len) {
            out[(long long)b0 * sb + obase + (long long)e * se] = (TO)v[m].x;
            if (b1 < nb) out[(long long)b1 * sb + obase + (long long)e * se] = (TO)v[m].y;
        }
    }
}

// The first cosine transform (z lines of one y) with G formed in registers:
// TL threads per pair of lines (b0 = 2p, b0 + 1), lanes along p.  Thread a
// forms the L/(2 TL) consecutive elements of its part of both lines, so one
// plane of the antiderivative (3 x by 2 y values) serves two elements in z and
// the shared column two in x: 3.4 loads per element in place of igf_G_at's 8,
// in whole rows; the elements and their mirrors then go through the line's
// buffer to the transform's order.  Same operation order as igf_G_at.  The
// staged form (dct_lines_body<FROM_TMP>) reads 32-byte pieces of eight planes
// per access, 83 % of the L1 throughput at 256 points.  Green's-function phase,
// staged -> this: 128^3 128.7 -> 114.8 us (mixed 120.4 -> 106.7), 64^3 36.0 ->
// 33.8 (31.9 -> 29.8).  At 32 and 64 points the branch gains 1 us at most, the
// step nothing (32^3 slower: 49.7 -> 56 us), and the staged form stays.
template <int L>
struct ZGeo {
    using G = ZLine<L>;
    static constexpr int TL = G::TL, LINES = 8, NT = TL * LINES;
};
template <int L>
__global__ void __launch_bounds__(ZGeo<L>::NT, 512 / ZGeo<L>::NT) k_dct_z_lines(const double* __restrict__ tmp,
                                                                                double* __restrict__ out, int nb,
                                                                                long long so, long long se,
                                                                                const double2* __restrict__ twd, int t0,
                                                                                int t1) {
    using G = typename ZGeo<L>::G;
    constexpr int N = L / 2, M = G::M, TL = G::TL, LINES = ZGeo<L>::LINES, CH = N / TL;
    __shared__ __align__(16) double2 xbuf[LINES][G::BUF + 1];
    const int li = threadIdx.x % LINES, a = threadIdx.x / LINES;
    const int b0 = 2 * (blockIdx.x * LINES + li), j = blockIdx.y;
    const bool one = b0 < nb, two = b0 + 1 < nb;
    double2* xs = xbuf[li];
    const long long plane = (long long)t0 * t1;
    const double* q = tmp + (one ? b0 : 0) + (long long)j * t0 + (long long)(a * CH) * plane;
    // c: the values at (b0 .. b0 + 2, j) and (.., j + 1) of plane k, d: of plane k + 1
    double c[6], d[6];
    auto load = [&](double* v, const double* r) {
        v[0] = r[0];
        v[1] = r[1];
        v[2] = two ? r[2] : 0.0;
        v[3] = r[t0];
        v[4] = r[t0 + 1];
        v[5] = two ? r[t0 + 2] : 0.0;
    };
    auto corner = [&](int i) {
        double g = d[i + 4];
        g += c[i + 1];
        g += c[i + 3];
        g += d[i];
        g -= c[i + 4];
        g -= d[i + 1];
        g -= d[i + 3];
        g -= c[i];
        return g;
    };
    load(c, q);
    double2 first{0.0, 0.0};
    const int cnt = a == TL - 1 ? CH + 1 : CH;  // the last thread also forms element N
#pragma unroll
    for (int m = 0; m <= CH; ++m) {
        if (m < cnt) {
            load(d, q + (long long)(m + 1) * plane);
            double2 g{one ? corner(0) : 0.0, two ? corner(1) : 0.0};
            if (m == 0) first = g;
            // G[0,0,0] <- G[0,0,1]
            if (m == 1 && a == 0) xs[xidx<L, TL>(0)] = double2{b0 == 0 && j == 0 ? g.x : first.x, first.y};
            const int e = a * CH + m;
            if (e > 0) {
                xs[xidx<L, TL>(e)] = g;
                if (e < N) xs[xidx<L, TL>(L - e)] = g;
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) c[k] = d[k];
        }
    }
    __syncthreads();
    double2 v[M];
#pragma unroll
    for (int m = 0; m < M; ++m) v[m] = xs[xidx<L, TL>(a + TL * m)];
    __syncthreads();
    line_fft<double, false, false, L, 1, TL>(v, a, xs, twd);
    if (!one) return;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int e = a + TL * m;
        if (e <= N) {
            double* o = out + b0 + (long long)j * so + (long long)e * se;
            o[0] = v[m].x;
            if (two) o[1] = v[m].y;
        }
    }
}

// Full real transform of lines of length L along z (stride se), 2 NC lines
// per block packed two per complex FFT and split by the Hermitian symmetry,
// as pass A; the half spectrum k in [0, L/2] of line b goes to
// out[k * nb + b], negated with NEG (imgrho2tr = -rho2tr * grntr,
// FFTPoissonSolver.cpp:316).
template <typename TO, int LT, int NC, int NT, bool NEG = true>
__device__ __forceinline__ void rfft_lines_neg_body(const double* __restrict__ in, Cx<TO>* __restrict__ out, int nb,
                                                    long long se, const FftPlan& pl, const double2* __restrict__ twd,
                                                    int bx) {
    constexpr int RC = 2 * NC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = LT > 0 ? LT : pl.L;
    const int CS = col_stride(L);
    double2* tw = reinterpret_cast<double2*>(smem_raw);
    double2* buf = tw + L;
    double2* tmp = buf + NC * CS + RC;
    stage_twiddles<double2, NT>(tw, twd, L);
    const int b0 = bx * RC;
    for (int e = threadIdx.x; e < RC * L; e += NT) {
        const int li = e % RC, m = e / RC;
        const int b = b0 + li;
        double* slot = reinterpret_cast<double*>(&buf[(li >> 1) * CS + sk(m)]) + (li & 1);
        if (b < nb)
            cp_elem(slot, in + b + (long long)m * se);
        else
            *slot = 0.0;
    }
    cp_async_wait_all();
    __syncthreads();
    const double2* o = block_fft<double, false, LT, NC, NT>(buf, tmp, pl, tw);
    const int half = L / 2;
    for (int e = threadIdx.x; e < RC * (half + 1); e += NT) {
        const int li = e % RC, k = e / RC;
        const int b = b0 + li;
        if (b >= nb) continue;
        const int q = li >> 1;
        const double2 Z = o[q * CS + sk(k)];
        const double2 Zm = o[q * CS + sk(k == 0 ? 0 : L - k)];
        double re, im;
        if ((li & 1) == 0) {
            re = 0.5 * (Z.x + Zm.x);
            im = 0.5 * (Z.y - Zm.y);
        } else {
            re = 0.5 * (Z.y + Zm.y);
            im = -0.5 * (Z.x - Zm.x);
        }
        out[(long long)k * nb + b] = NEG ? Cx<TO>{(TO)(-re), (TO)(-im)} : Cx<TO>{(TO)re, (TO)im};
    }
}
template <typename TO, int LT, int NC, int NT, bool NEG = true>
__global__ void __launch_bounds__(NT, 1024 / NT) k_rfft_lines_neg(const double* __restrict__ in, Cx<TO>* __restrict__ out, int nb,
                                                       long long se, FftPlan pl, const double2* __restrict__ twd) {
    rfft_lines_neg_body<TO, LT, NC, NT, NEG>(in, out, nb, se, pl, twd, blockIdx.x);
}

// Tile-shape variants of a length: V = 0 is the widest shape (cols_for
// columns, up to 256 threads), each further variant halves the columns per
// block (more, smaller blocks, down to a single warp for the long
// transforms), which shortens each block's chain of barriers.  The batched
// autotuner picks per length; single-bunch launches use single_variant().
__host__ __device__ constexpr int cols_v(int LT, int V) {
    const int c = cols_for(LT) >> V;
    return c > 1 ? c : 1;
}
__host__ __device__ constexpr int threads_v(int LT, int V) {
    if (LT == 0) return 256;
    const int t = cols_v(LT, V) * (LT / min_radix(LT));
    return t < 32 ? 32 : t;
}

// ---------------------------------------------------------------- dispatch
template <int LT, int V = 0>
struct Geo {
    static constexpr int NC = cols_v(LT, V);
    static constexpr int NT = threads_v(LT, V);
};

// Tile-shape variant of single-bunch launches for a transform length (0 for
// lengths without a template instance): SCGPU_FFT_VARIANT=v forces one for
// every length, otherwise the measured default of the length.
int single_variant(int LT) {
    static const int forced = [] {
        const char* e = std::getenv("SCGPU_FFT_VARIANT");
        const int v = e ? std::atoi(e) : -1;
        return (v >= 0 && v < kFftLinesVariant) ? v : -1;
    }();
    if (LT == 0) return 0;
    if (forced >= 0) return forced;
    return LT >= 64 ? 1 : 0;  // half-width tiles measured faster from 64 points up (the cosine transforms most)
}

// Passes A (open z; from 32 points), B, C and D of 64-, 128- and 256-point
// lines, E and G's z transform of 128- and 256-point lines take the
// register-resident kernels (k_*_lines, the same bits as the staged ones).
// SCGPU_FFT_LINES=0 selects the staged kernels everywhere.
bool register_lines() {
    static const bool on = [] {
        const char* e = std::getenv("SCGPU_FFT_LINES");
        return !(e && std::string(e) == "0");
    }();
    return on;
}

// Calls f.template go<LT, V>() with V = single_variant(LT).
template <int LT, typename F>
void with_variant(F& f) {
    switch (single_variant(LT)) {
        case 1: f.template go<LT, 1>(); break;
        case 2: f.template go<LT, 2>(); break;
        case 3: f.template go<LT, 3>(); break;
        default: f.template go<LT, 0>(); break;
    }
}

template <typename C>
size_t smem_of(int L, int nc) {
    return sizeof(C) * tile_elems(L, nc);
}

template <typename TI>
size_t smem_conv(int L, int nc) {
    return (sizeof(double2) + sizeof(Cx<TI>)) * (size_t)L + 2 * sizeof(double2) * (size_t)nc * col_stride(L);
}

// Calls f.template run<LT>() with LT the template length for L, or 0.
template <typename F>
void with_length(int L, F&& f) {
    switch (L) {
        case 32: f.template run<32>(); break;
        case 64: f.template run<64>(); break;
        case 96: f.template run<96>(); break;
        case 128: f.template run<128>(); break;
        case 256: f.template run<256>(); break;
        default: f.template run<0>(); break;
    }
}

// The longest z transform whose pass A can form rho itself (fft_assembles).
constexpr int kAssembleMax = 64;

template <typename T, bool FULL = false>
struct LaunchA {
    T* rho;
    Cx<T>* spec;
    int n0, n1, n2, L0, L1;
    FftPlan pz;
    const Cx<T>* twz;
    cudaStream_t s;
    const AccIn* in = nullptr;  // form rho from the accumulators (fft_assembles)
    template <int LT>
    void run() {
        if constexpr (!FULL && (LT == 32 || LT == 64 || LT == 128 || LT == 256)) {
            if (register_lines() && 2 * n2 == LT) {
                using G = LineGeo<LT>;
                const long long lines = (long long)n1 * ((n0 + 1) / 2);
                const unsigned g = (unsigned)((lines + G::LINES - 1) / G::LINES);
                if constexpr (LT <= kAssembleMax) {
                    if (in) {
                        k_fft_z_r2c_lines<T, LT, true><<<g, G::NT, 0, s>>>(rho, spec, n0, n1, L0, L1, twz, *in);
                        return;
                    }
                }
                k_fft_z_r2c_lines<T, LT><<<g, G::NT, 0, s>>>(rho, spec, n0, n1, L0, L1, twz, AccIn{});
                return;
            }
        }
        with_variant<LT>(*this);
    }
    template <int LT, int V>
    void go() {
        constexpr int NC = Geo<LT, V>::NC, NT = Geo<LT, V>::NT;
        dim3 g((unsigned)((n0 + 2 * NC - 1) / (2 * NC)), (unsigned)n1);
        k_fft_z_r2c<T, LT, NC, NT, FULL><<<g, NT, smem_of<Cx<T>>(pz.L, NC), s>>>(rho, spec, n0, n1, n2, L0, L1, pz, twz);
    }
};

template <typename T, bool INV>
struct LaunchY {
    Cx<T>* spec;
    int n0, L0, n_in, n_out, planes;
    FftPlan py;
    const Cx<T>* twy;
    cudaStream_t s;
    template <int LT>
    void run() {
        if constexpr (LT == 64 || LT == 128 || LT == 256) {
            if (register_lines() && 2 * (INV ? n_out : n_in) == LT) {
                using G = YGeo<T, LT>;
                const dim3 g((unsigned)((n0 + G::LINES - 1) / G::LINES), (unsigned)planes);
                k_fft_y_lines<T, INV, LT><<<g, G::NT, 0, s>>>(spec, n0, L0, planes, twy);
                return;
            }
        }
        with_variant<LT>(*this);
    }
    template <int LT, int V>
    void go() {
        constexpr int NC = Geo<LT, V>::NC, NT = Geo<LT, V>::NT;
        dim3 g((unsigned)((n0 + NC - 1) / NC), (unsigned)planes);
        k_fft_y<T, INV, LT, NC, NT><<<g, NT, smem_of<Cx<T>>(py.L, NC), s>>>(spec, n0, L0, n_in, n_out, py, twy);
    }
};

template <typename TI, bool CG = false>
struct LaunchC {
    const Cx<TI>* in;
    double2* out;
    const TI* ghat;
    int n0, n1, L1, rows;
    FftPlan px;
    const Cx<TI>* twi;
    const double2* two;
    cudaStream_t s;
    template <int LT>
    void run() {
        if constexpr (LT == 64 || LT == 128 || LT == 256) {
            if (register_lines() && 2 * n0 == LT) {
                using G = LineGeo<LT>;
                k_fft_x_conv_lines<TI, double, CG, LT><<<(unsigned)((rows + G::LINES - 1) / G::LINES), G::NT, 0, s>>>(
                    in, out, ghat, n0, n1, L1, rows, twi, two);
                return;
            }
        }
        with_variant<LT>(*this);
    }
    template <int LT, int V>
    void go() {
        constexpr int NC = Geo<LT, V>::NC, NT = Geo<LT, V>::NT;
        k_fft_x_conv<TI, double, LT, NC, NT, CG><<<(unsigned)((rows + NC - 1) / NC), NT, smem_conv<TI>(px.L, NC), s>>>(
            in, out, ghat, n0, n1, L1, rows, px, twi, two);
    }
};

template <typename TO, bool NEG = true>
struct LaunchRfftNeg {
    const double* in;
    Cx<TO>* out;
    int nb;
    long long se;
    FftPlan pl;
    const double2* tw;
    cudaStream_t s;
    template <int LT>
    void run() {
        with_variant<LT>(*this);
    }
    template <int LT, int V>
    void go() {
        constexpr int NC = Geo<LT, V>::NC, NT = Geo<LT, V>::NT;
        k_rfft_lines_neg<TO, LT, NC, NT, NEG>
            <<<(unsigned)((nb + 2 * NC - 1) / (2 * NC)), NT, smem_of<double2>(pl.L, NC), s>>>(in, out, nb, se, pl, tw);
    }
};

// Threads of the staged pass E: staging, packing and scaling its tile take more
// of them than its butterflies need, so no fewer than 256 up to 128 points
// (48^3 step 78.6 -> 76.8 us).  At 256 points fewer blocks fit and it loses.
__host__ __device__ constexpr int threads_e(int lt, int nt) { return lt > 0 && lt <= 128 && nt < 256 ? 256 : nt; }
template <bool SELF, bool FLIP = false, bool FULL = false>
struct LaunchE {
    const double2* spec;
    double* phi;
    int n0, n1, n2, L0, L1;
    FftPlan pz;
    const double2* twz;
    const StepState* st;
    double normFact, coupling;
    cudaStream_t s;
    template <int LT>
    void run() {
        if constexpr (!FULL && (LT == 128 || LT == 256)) {
            if (register_lines() && 2 * n2 == LT) {
                using G = ZLine<LT>;
                const int lines = n1 * ((n0 + 1) / 2);
                k_fft_z_c2r_lines<SELF, LT, FLIP><<<(unsigned)((lines + G::LINES - 1) / G::LINES), G::NT, 0, s>>>(
                    spec, phi, n0, n1, L0, L1, twz, st, normFact, coupling);
                return;
            }
        }
        with_variant<LT>(*this);
    }
    template <int LT, int V>
    void go() {
        constexpr int NC = Geo<LT, V>::NC, NT = threads_e(LT, Geo<LT, V>::NT);
        dim3 g((unsigned)((n0 + 2 * NC - 1) / (2 * NC)), (unsigned)n1);
        k_fft_z_c2r<double, SELF, LT, NC, NT, FLIP, FULL><<<g, NT, smem_of<double2>(pz.L, NC), s>>>(
            spec, phi, n0, n1, n2, L0, L1, pz, twz, st, normFact, coupling);
    }
};

template <typename TO, bool FROM_TMP = false>
struct LaunchDct {
    const double* in;
    TO* out;
    int len, nb, outer;
    long long sb, so, se;
    FftPlan pl;
    const double2* tw;
    cudaStream_t s;
    int t0 = 0, t1 = 0;
    template <int LT>
    void run() {
        // 256-point lines only: at 128 points the staged tiles measured faster
        // (Green's-function phase 41.6 against 45.6 us at 64^3), at 256 points
        // the line form (185 against 175 us at 128^3).  16 threads per line
        // with 16 elements each, 16 warps per SM, took it from 138 to 128 us
        // (phase profile; mixed 129 to 120); 8 threads held 32 in some 200 registers, 8 warps.
        // The convolution's passes keep 8: with 16 their transforms of both
        // types spill at 4 blocks and lose at 3 (156 -> 167 us at 128^3).
        if constexpr (!FROM_TMP && LT == 256) {
            if (register_lines() && pl.L == LT && len == LT / 2 + 1) {
                using G = LineGeo<LT, 16>;
                const int pairs = (nb + 1) / 2;
                dim3 g((unsigned)((pairs + G::LINES - 1) / G::LINES), (unsigned)outer);
                k_dct_lines_reg<TO, LT><<<g, G::NT, 0, s>>>(in, out, len, nb, sb, so, se, tw);
                return;
            }
        }
        if constexpr (FROM_TMP && (LT == 128 || LT == 256)) {
            if (register_lines() && pl.L == LT && len == LT / 2 + 1 && sb == 1) {
                using Z = ZGeo<LT>;
                dim3 g((unsigned)(((nb + 1) / 2 + Z::LINES - 1) / Z::LINES), (unsigned)outer);
                k_dct_z_lines<LT><<<g, Z::NT, 0, s>>>(in, out, nb, so, se, tw, t0, t1);
                return;
            }
        }
        with_variant<LT>(*this);
    }
    template <int LT, int V>
    void go() {
        // forming G reads eight values per element, so the z pass takes 256
        // threads to stage its tile, however few its butterflies need
        constexpr int NC = Geo<LT, V>::NC, NT = FROM_TMP ? 256 : Geo<LT, V>::NT;
        dim3 g((unsigned)((nb + 2 * NC - 1) / (2 * NC)), (unsigned)outer);
        k_dct_lines<TO, LT, NC, NT, FROM_TMP><<<g, NT, smem_of<double2>(pl.L, NC), s>>>(in, out, len, nb, sb, so, se, pl,
                                                                                     tw, t0, t1);
    }
};

// Raises the dynamic shared-memory limit of every instance of one length.
struct SetLimits {
    template <typename K>
    static void allow(K kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    }
    template <int LT>
    void run() {
        go<LT, 0>();
        if constexpr (LT > 0) {
            go<LT, 1>();
            go<LT, 2>();
            go<LT, 3>();
        }
    }
    template <int LT, int V>
    void go() {
        constexpr int NC = Geo<LT, V>::NC, NT = Geo<LT, V>::NT;
        allow(k_fft_z_r2c<double, LT, NC, NT>);
        allow(k_fft_z_r2c<float, LT, NC, NT>);
        allow(k_fft_y<double, false, LT, NC, NT>);
        allow(k_fft_y<float, false, LT, NC, NT>);
        allow(k_fft_y<double, true, LT, NC, NT>);
        allow(k_fft_x_conv<double, double, LT, NC, NT>);
        allow(k_fft_x_conv<float, double, LT, NC, NT>);
        allow(k_fft_z_c2r<double, true, LT, NC, threads_e(LT, NT)>);
        allow(k_fft_z_c2r<double, false, LT, NC, threads_e(LT, NT)>);
        allow(k_dct_lines<double, LT, NC, NT>);
        allow(k_dct_lines<float, LT, NC, NT>);
        allow(k_dct_lines<double, LT, NC, 256, true>);
        allow(k_fft_x_conv<double, double, LT, NC, NT, true>);
        allow(k_fft_x_conv<float, double, LT, NC, NT, true>);
        allow(k_fft_z_c2r<double, true, LT, NC, threads_e(LT, NT), true>);
        allow(k_fft_z_c2r<double, false, LT, NC, threads_e(LT, NT), true>);
        allow(k_rfft_lines_neg<double, LT, NC, NT>);
        allow(k_rfft_lines_neg<float, LT, NC, NT>);
        allow(k_rfft_lines_neg<double, LT, NC, NT, false>);
        allow(k_rfft_lines_neg<float, LT, NC, NT, false>);
        allow(k_fft_z_r2c<double, LT, NC, NT, true>);
        allow(k_fft_z_r2c<float, LT, NC, NT, true>);
        allow(k_fft_z_c2r<double, true, LT, NC, threads_e(LT, NT), false, true>);
        allow(k_fft_z_c2r<double, false, LT, NC, threads_e(LT, NT), false, true>);
    }
};

// ---------------------------------------------------------------- batches
__device__ __forceinline__ FftPlan plan_dev(int L) {
    const RadixPlan r = radix_plan(L);
    FftPlan p;
    p.L = L;
    p.nst = r.nst;
#pragma unroll
    for (int i = 0; i < 12; ++i) p.r[i] = r.r[i];
    return p;
}

// twiddles of axis a as complex T (the float table follows the double one)
template <typename T>
__device__ __forceinline__ const Cx<T>* tw_dev(const DevBunch& d, int a) {
    const double2* p = reinterpret_cast<const double2*>(d.tw[a]);
    if constexpr (sizeof(T) == sizeof(double))
        return reinterpret_cast<const Cx<T>*>(p);
    else
        return reinterpret_cast<const Cx<T>*>(p + 2 * d.bc.n[a]);
}

// One kernel per pass: block i runs the single-bunch body for bunch work[i].x
// at block coordinates (work[i].y, work[i].z), with that bunch's sizes and
// buffers (T: the forward-half type, as in convolution_t).
template <typename T, int PASS, int LT, int NC, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_fft_pass_batch(const DevBunch* __restrict__ tab, const int4* __restrict__ work,
                                                        int nitems) {
    const int4 w = resolve_block(work, nitems);
    const DevBunch& d = tab[w.x];
    const int n0 = d.bc.n[0], n1 = d.bc.n[1], n2 = d.bc.n[2];
    const int L0 = 2 * n0, L1 = 2 * n1, L2 = 2 * n2;
    Cx<T>* fwd = reinterpret_cast<Cx<T>*>(d.precision == 0 ? d.spec : d.spec_lo);
    double2* inv = reinterpret_cast<double2*>(d.spec);
    if constexpr (PASS == kPassZR2C) {
        fft_z_r2c_body<T, LT, NC, NT>((const T*)d.rho, fwd, n0, n1, n2, L0, L1, plan_dev(L2), tw_dev<T>(d, 2), w.y, w.z);
    } else if constexpr (PASS == kPassYFwd) {
        fft_y_body<T, false, LT, NC, NT>(fwd, n0, L0, n1, L1, plan_dev(L1), tw_dev<T>(d, 1), w.y, w.z);
    } else if constexpr (PASS == kPassXConv) {
        fft_x_conv_body<T, double, LT, NC, NT>(fwd, inv, (const T*)d.ghat, n0, n1, L1, (n2 + 1) * L1, plan_dev(L0),
                                               tw_dev<T>(d, 0), tw_dev<double>(d, 0), w.y);
    } else if constexpr (PASS == kPassYInv) {
        fft_y_body<double, true, LT, NC, NT>(inv, n0, L0, L1, n1, plan_dev(L1), tw_dev<double>(d, 1), w.y, w.z);
    } else if constexpr (PASS == kPassZC2R) {
        double normFact = 1.0;
        normFact /= L0;
        normFact /= L1;
        normFact /= L2;
        fft_z_c2r_body<double, true, LT, NC, NT>(inv, d.phi, n0, n1, n2, L0, L1, plan_dev(L2), tw_dev<double>(d, 2), d.st,
                                                 normFact, d.bc.coupling, w.y, w.z);
    } else {
        const long long g0 = n0 + 1, g1 = n1 + 1, g2 = n2 + 1;
        // G formed from the antiderivative in the z pass (gtmp -> gline ->
        // gtmp -> ghat), as launch_green_transform_from_tmp
        if constexpr (PASS == kPassDctZ)
            dct_lines_body<double, LT, NC, NT, true>(d.gtmp, d.gline, (int)g2, (int)g0, 1, g0, g0 * g1, plan_dev(L2),
                                                     tw_dev<double>(d, 2), w.y, w.z, n0 + 2, n1 + 2);
        else if constexpr (PASS == kPassDctY)
            dct_lines_body<double, LT, NC, NT>(d.gline, d.gtmp, (int)g1, (int)g0, 1, g0 * g1, g0, plan_dev(L1),
                                               tw_dev<double>(d, 1), w.y, w.z);
        else
            dct_lines_body<T, LT, NC, NT>(d.gtmp, (T*)d.ghat, (int)g0, (int)g1, g0, g0 * g1, 1, plan_dev(L0),
                                          tw_dev<double>(d, 0), w.y, w.z);
    }
}

inline bool line_length(int L) { return L == 64 || L == 128 || L == 256; }

// Variant kFftLinesVariant: passes B, C and D of 64-, 128- and 256-point
// lines run the register-resident line transforms (the same bits), block
// (x, y) of a bunch as in the single-bunch launch.
template <typename T, int PASS, int L>
struct BatchLines {
    using TY = typename std::conditional<PASS == kPassYInv, double, T>::type;
    static constexpr int NT = PASS == kPassXConv ? LineGeo<L>::NT : YGeo<TY, L>::NT;
    static constexpr int MINB = PASS == kPassXConv ? 1 : kYBlocks<TY, L>;
};
template <typename T, int PASS, int L>
__global__ void __launch_bounds__(BatchLines<T, PASS, L>::NT, BatchLines<T, PASS, L>::MINB) k_fft_lines_batch(const DevBunch* __restrict__ tab,
                                                                  const int4* __restrict__ work, int nitems) {
    const int4 w = resolve_block(work, nitems);
    const DevBunch& d = tab[w.x];
    const int n0 = d.bc.n[0], n1 = d.bc.n[1], n2 = d.bc.n[2];
    const int L0 = 2 * n0, L1 = 2 * n1;
    Cx<T>* fwd = reinterpret_cast<Cx<T>*>(d.precision == 0 ? d.spec : d.spec_lo);
    double2* inv = reinterpret_cast<double2*>(d.spec);
    if constexpr (PASS == kPassYFwd)
        fft_y_lines_body<T, false, L>(fwd, n0, L0, n2 + 1, tw_dev<T>(d, 1), w.y, w.z);
    else if constexpr (PASS == kPassXConv)
        fft_x_conv_lines_body<T, double, false, L>(fwd, inv, (const T*)d.ghat, n0, n1, L1, (n2 + 1) * L1, tw_dev<T>(d, 0),
                                                   tw_dev<double>(d, 0), w.y);
    else
        fft_y_lines_body<double, true, L>(inv, n0, L0, n2 + 1, tw_dev<double>(d, 1), w.y, w.z);
}

template <typename T, int PASS>
struct LaunchLinesBatch {
    const DevBunch* tab;
    const int4* work;
    int nitems, n;
    cudaStream_t s;
    template <int LT>
    void run() {
        if constexpr (LT == 64 || LT == 128 || LT == 256)
            k_fft_lines_batch<T, PASS, LT><<<n, BatchLines<T, PASS, LT>::NT, 0, s>>>(tab, work, nitems);
    }
};

template <typename T, int PASS>
size_t pass_smem(int L, int nc) {
    if constexpr (PASS == kPassXConv) return smem_conv<T>(L, nc);
    if constexpr (PASS == kPassZR2C || PASS == kPassYFwd) return smem_of<Cx<T>>(L, nc);
    return smem_of<double2>(L, nc);
}

template <typename T, int PASS, int V>
struct LaunchPassBatch {
    const DevBunch* tab;
    const int4* work;
    int nitems, n, L;
    cudaStream_t s;
    template <int LT>
    void run() {
        constexpr int NC = cols_v(LT, V), NT = threads_v(LT, V);
        auto k = k_fft_pass_batch<T, PASS, LT, NC, NT>;
        const size_t sm = pass_smem<T, PASS>(L, NC);
        static bool limits = [&] {
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            return true;
        }();
        (void)limits;
        k<<<n, NT, sm, s>>>(tab, work, nitems);
    }
};

template <typename T, int PASS>
void pass_batch_t(int L, int variant, const DevBunch* tab, const int4* work, int nitems, int n, cudaStream_t s) {
    if (variant == kFftLinesVariant) {
        if constexpr (PASS == kPassYFwd || PASS == kPassXConv || PASS == kPassYInv) {
            if (line_length(L)) {
                with_length(L, LaunchLinesBatch<T, PASS>{tab, work, nitems, n, s});
                return;
            }
        }
        variant = 0;  // the other passes with the widest tiles
    }
    switch (variant) {
        case 1: with_length(L, LaunchPassBatch<T, PASS, 1>{tab, work, nitems, n, L, s}); break;
        case 2: with_length(L, LaunchPassBatch<T, PASS, 2>{tab, work, nitems, n, L, s}); break;
        case 3: with_length(L, LaunchPassBatch<T, PASS, 3>{tab, work, nitems, n, L, s}); break;
        default: with_length(L, LaunchPassBatch<T, PASS, 0>{tab, work, nitems, n, L, s}); break;
    }
}

template <typename T>
void pass_batch(int pass, int L, int variant, const DevBunch* tab, const int4* work, int nitems, int n, cudaStream_t s) {
    switch (pass) {
        case kPassZR2C: pass_batch_t<T, kPassZR2C>(L, variant, tab, work, nitems, n, s); break;
        case kPassYFwd: pass_batch_t<T, kPassYFwd>(L, variant, tab, work, nitems, n, s); break;
        case kPassXConv: pass_batch_t<T, kPassXConv>(L, variant, tab, work, nitems, n, s); break;
        case kPassYInv: pass_batch_t<T, kPassYInv>(L, variant, tab, work, nitems, n, s); break;
        case kPassZC2R: pass_batch_t<T, kPassZC2R>(L, variant, tab, work, nitems, n, s); break;
        case kPassDctZ: pass_batch_t<T, kPassDctZ>(L, variant, tab, work, nitems, n, s); break;
        case kPassDctY: pass_batch_t<T, kPassDctY>(L, variant, tab, work, nitems, n, s); break;
        default: pass_batch_t<T, kPassDctX>(L, variant, tab, work, nitems, n, s); break;
    }
}

inline bool special_length(int L) { return L == 32 || L == 64 || L == 96 || L == 128 || L == 256; }

}  // namespace

bool fft_register_lines() { return register_lines(); }

// Open z, n2 = 16 or 32 (pass A's line kernel of 32 or 64 points) and at most
// 64000 cells: there the step waits on its launches, and the separate assembly
// is one (32^3, 1e5 particles: 51.0 -> 48.0 us a step, mixed 47.7 -> 45.5); at
// 64^3 the assembly fills the GPU and does its divisions faster than the
// transform's threads between their loads (mixed 107.5 against 109.2 us).
bool fft_assembles(const DevBunch& b) {
    const int L2 = 2 * b.bc.n[2];
    return register_lines() && !b.periodic_z && (L2 == 32 || L2 == kAssembleMax) &&
           (long long)b.bc.n[0] * b.bc.n[1] * b.bc.n[2] <= 64000;
}

bool fft_pass_plane(const DevBunch& b, int variant) {
    return variant == kFftLinesVariant && fft_plane_length(2 * b.bc.n[0], 2 * b.bc.n[1]);
}

int fft_pass_length(int pass, const DevBunch& b) {
    switch (pass) {
        case kPassZR2C:
        case kPassZC2R:
        case kPassDctZ: return 2 * b.bc.n[2];
        case kPassYFwd:
        case kPassYInv:
        case kPassDctY: return 2 * b.bc.n[1];
        default: return 2 * b.bc.n[0];
    }
}

void fft_pass_grid(int pass, const DevBunch& b, int variant, int* gx, int* gy) {
    const int L = fft_pass_length(pass, b);
    const int n0 = b.bc.n[0], n1 = b.bc.n[1], n2 = b.bc.n[2];
    if (pass == kPassPlane) {  // block (rank in the cluster, plane)
        *gx = fft_plane_cluster(L);
        *gy = n2 + 1;
        return;
    }
    if (pass == kPassDctPlane) {
        *gx = n2 + 1;
        *gy = 1;
        return;
    }
    if (variant == kFftLinesVariant) {
        const int lines = L >= 256 ? LineGeo<256>::LINES : LineGeo<128>::LINES;
        if (line_length(L) && (pass == kPassYFwd || pass == kPassYInv)) {
            *gx = (n0 + lines - 1) / lines;
            *gy = n2 + 1;
            return;
        }
        if (line_length(L) && pass == kPassXConv) {
            *gx = ((n2 + 1) * 2 * n1 + lines - 1) / lines;
            *gy = 1;
            return;
        }
        variant = 0;
    }
    const int nc = cols_v(special_length(L) ? L : 0, variant);
    switch (pass) {
        case kPassZR2C:
        case kPassZC2R:
            *gx = (n0 + 2 * nc - 1) / (2 * nc);
            *gy = n1;
            break;
        case kPassYFwd:
        case kPassYInv:
            *gx = (n0 + nc - 1) / nc;
            *gy = n2 + 1;
            break;
        case kPassXConv:
            *gx = ((n2 + 1) * 2 * n1 + nc - 1) / nc;
            *gy = 1;
            break;
        case kPassDctZ:
            *gx = (n0 + 1 + 2 * nc - 1) / (2 * nc);
            *gy = n1 + 1;
            break;
        case kPassDctY:
            *gx = (n0 + 1 + 2 * nc - 1) / (2 * nc);
            *gy = n2 + 1;
            break;
        default:
            *gx = (n1 + 1 + 2 * nc - 1) / (2 * nc);
            *gy = n2 + 1;
            break;
    }
}

void launch_fft_pass_batch(int pass, int L, int precision, int variant, const DevBunch* tab, const int4* work, int nitems,
                           int n, cudaStream_t s) {
    if (n <= 0 || nitems <= 0) return;
    if (pass == kPassPlane) {
        launch_plane_conv_batch(L, precision, tab, work, nitems, n, s);
        return;
    }
    if (pass == kPassDctPlane) {
        launch_dct_plane_batch(L, precision, tab, work, nitems, n, s);
        return;
    }
    if (precision == 0)
        pass_batch<double>(pass, L, variant, tab, work, nitems, n, s);
    else
        pass_batch<float>(pass, L, variant, tab, work, nitems, n, s);
}

FftPlan make_plan(int L) {
    const RadixPlan r = radix_plan(L);
    FftPlan p{};
    p.L = L;
    p.nst = r.nst;
    for (int i = 0; i < 12; ++i) p.r[i] = r.r[i];
    return p;
}

size_t fft_smem_bytes(const DevBunch& b) {
    size_t m = 0;
    for (int d = 0; d < 3; ++d) {
        const int L = 2 * b.bc.n[d];
        m = std::max(m, smem_of<double2>(L, cols_for(0)));
        m = std::max(m, smem_conv<double>(L, cols_for(0)));
    }
    return m;
}

// Axis d's transform length: the doubled grid, except z with periodic z.
static inline int axis_length(const DevBunch& b, int d) {
    return (d == 2 && b.periodic_z) ? b.bc.n[2] : 2 * b.bc.n[d];
}

// twiddles exp(-2 pi i e / L), e in [0, L), from long double arithmetic
// rounded once to the table's type (tf may be null)
void twiddle_values(int L, double2* td, float2* tf) {
    for (int e = 0; e < L; ++e) {
        const long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double)e / (long double)L;
        td[e] = double2{(double)cosl(a), (double)sinl(a)};
        if (tf) tf[e] = float2{(float)cosl(a), (float)sinl(a)};
    }
}

void upload_twiddles(DevBunch& b, cudaStream_t s) {
    for (int d = 0; d < 3; ++d) {
        const int L = axis_length(b, d);
        std::vector<double2> td(L);
        std::vector<float2> tf(L);
        twiddle_values(L, td.data(), tf.data());
        // the double table always (the G spectrum is built in FP64); the float one in the mixed form
        double2* dptr = reinterpret_cast<double2*>(b.tw[d]);
        cudaMemcpyAsync(dptr, td.data(), L * sizeof(double2), cudaMemcpyHostToDevice, s);
        if (b.precision != 0) {
            float2* fptr = reinterpret_cast<float2*>(dptr + L);
            cudaMemcpyAsync(fptr, tf.data(), L * sizeof(float2), cudaMemcpyHostToDevice, s);
        }
    }
    cudaStreamSynchronize(s);
}

static inline const void* tw_for(const DevBunch& b, int d) {
    const int L = axis_length(b, d);
    const double2* dptr = reinterpret_cast<const double2*>(b.tw[d]);
    return b.precision == 0 ? (const void*)dptr : (const void*)(dptr + L);
}

// Cosine transforms of `planes` planes of (n0+1)(n1+1) reals along y (in to
// tmp) and x (tmp to out), or both in one kernel per plane (in to out).
template <typename TO>
static void dct_yx(const DevBunch& b, const double* in, double* tmp, TO* out, int planes, cudaStream_t s) {
    const int n0 = b.bc.n[0], n1 = b.bc.n[1];
    const long long g0 = n0 + 1, g1 = n1 + 1;
    if (fft_plane_length(2 * n0, 2 * n1)) {
        launch_dct_plane(2 * n0, in, out, sizeof(TO) == sizeof(double), planes, b.tw[1], b.tw[0], s);
        return;
    }
    const FftPlan p0 = make_plan(2 * n0), p1 = make_plan(2 * n1);
    const double2* tw0 = reinterpret_cast<const double2*>(b.tw[0]);
    const double2* tw1 = reinterpret_cast<const double2*>(b.tw[1]);
    // y lines: batch x, outer z
    with_length(2 * n1, LaunchDct<double>{in, tmp, (int)g1, (int)g0, planes, 1, g0 * g1, g0, p1, tw1, s});
    // x lines: batch y (stride g0), outer z
    with_length(2 * n0, LaunchDct<TO>{tmp, out, (int)g0, (int)g1, planes, g0, g0 * g1, 1, p0, tw0, s});
}

// Spectrum of the mirrored G from b.gline ((n0+1)(n1+1)(n2+1), FP64), into b.ghat.
void launch_green_transform(const DevBunch& b, cudaStream_t s) {
    const long long g0 = b.bc.n[0] + 1, g1 = b.bc.n[1] + 1, g2 = b.bc.n[2] + 1;
    const FftPlan p2 = make_plan(2 * b.bc.n[2]);
    const double2* tw2 = reinterpret_cast<const double2*>(b.tw[2]);
    // z lines: batch x (stride 1), outer y
    with_length(p2.L, LaunchDct<double>{b.gline, b.gtmp, (int)g2, (int)g0, (int)g1, 1, g0, g0 * g1, p2, tw2, s});
    if (b.precision == 0)
        dct_yx(b, b.gtmp, b.gline, (double*)b.ghat, (int)g2, s);
    else
        dct_yx(b, b.gtmp, b.gline, (float*)b.ghat, (int)g2, s);
}

// The same spectrum from the antiderivative (b.gtmp, launch_igf_tmp): the
// z transforms form G as they stage it and write gline, the y transforms
// gline -> gtmp, the x transforms gtmp -> ghat (or both gline -> ghat).  G's
// values and every transform are those of launch_igf +
// launch_green_transform, so Ĝ has the same bits; G is never stored.
void launch_green_transform_from_tmp(const DevBunch& b, cudaStream_t s) {
    const int n0 = b.bc.n[0], n1 = b.bc.n[1];
    const long long g0 = n0 + 1, g1 = n1 + 1, g2 = b.bc.n[2] + 1;
    const FftPlan p2 = make_plan(2 * b.bc.n[2]);
    const double2* tw2 = reinterpret_cast<const double2*>(b.tw[2]);
    LaunchDct<double, true> z{b.gtmp, b.gline, (int)g2, (int)g0, (int)g1, 1, g0, g0 * g1, p2, tw2, s};
    z.t0 = n0 + 2;
    z.t1 = n1 + 2;
    with_length(p2.L, z);
    if (b.precision == 0)
        dct_yx(b, b.gline, b.gtmp, (double*)b.ghat, (int)g2, s);
    else
        dct_yx(b, b.gline, b.gtmp, (float*)b.ghat, (int)g2, s);
}

// Spectrum of the image's shifted G (b.gimg, (n0+1)(n1+1)(2 n2), FP64):
// cosine transforms along y and x on every z plane (G is even in x and y),
// then a full real transform along z (it is not even in z), negated, into
// b.ghat_img (n2+1)(n1+1)(n0+1) complex T.
void launch_green_transform_image(const DevBunch& b, cudaStream_t s) {
    const int n0 = b.bc.n[0], n1 = b.bc.n[1], n2 = b.bc.n[2];
    const long long g0 = n0 + 1, g1 = n1 + 1, L2 = 2 * n2;
    const long long GI = g0 * g1 * L2;
    const FftPlan p2 = make_plan(2 * n2);
    const double2* tw2 = reinterpret_cast<const double2*>(b.tw[2]);
    double* ga = b.gimg;
    double* gb = b.gimg + GI;
    const bool plane = fft_plane_length(2 * n0, 2 * n1);
    double* go = plane ? gb : ga;  // the plane kernel does not work in place
    dct_yx(b, ga, gb, go, (int)L2, s);
    // z lines of length 2 n2: batch (x, y), element stride g0 g1
    if (b.precision == 0)
        with_length(2 * n2, LaunchRfftNeg<double>{go, (double2*)b.ghat_img, (int)(g0 * g1), g0 * g1, p2, tw2, s});
    else
        with_length(2 * n2, LaunchRfftNeg<float>{go, (float2*)b.ghat_img, (int)(g0 * g1), g0 * g1, p2, tw2, s});
}

// Periodic z (FFTPoissonSolver with bcz, :130-155, :661-662): G on its first
// n2 z planes (the unshifted G of b.gline, not mirrored in z), cosine
// transforms along y and x, then a full real transform of length n2 along z
// into b.ghat_img (complex T).
void launch_green_transform_periodic(const DevBunch& b, cudaStream_t s) {
    const int n0 = b.bc.n[0], n1 = b.bc.n[1], n2 = b.bc.n[2];
    const long long g0 = n0 + 1, g1 = n1 + 1;
    const FftPlan pz = make_plan(n2);
    const double2* tw2 = reinterpret_cast<const double2*>(b.tw[2]);
    const bool plane = fft_plane_length(2 * n0, 2 * n1);
    double* go = plane ? b.gtmp : b.gline;
    dct_yx(b, b.gline, b.gtmp, go, n2, s);
    if (b.precision == 0)
        with_length(n2, LaunchRfftNeg<double, false>{go, (double2*)b.ghat_img, (int)(g0 * g1), g0 * g1, pz, tw2, s});
    else
        with_length(n2, LaunchRfftNeg<float, false>{go, (float2*)b.ghat_img, (int)(g0 * g1), g0 * g1, pz, tw2, s});
}

// T is the type of the forward half (A, B and the forward x transform of C);
// the inverse half (C's inverse, D, E) is FP64 in both forms.  With energy
// bins the plain form keeps the forward spectrum in b.spec_fwd, so the bin's
// own and its image's convolutions (C, D, E twice) start from one A, B.
// parts: kConvForwardPart (A, B: need only rho) and/or kConvRestPart (C, D,
// E: need the spectrum of G as well).
template <typename T>
static void convolution_t(const DevBunch& b, int mode, int parts, cudaStream_t s) {
    using C = Cx<T>;
    const int n0 = b.bc.n[0], n1 = b.bc.n[1], n2 = b.bc.n[2];
    const int L0 = 2 * n0, L1 = 2 * n1, L2 = axis_length(b, 2);
    const int K = L2 / 2;  // half-spectrum planes 0..K along z
    const bool plane = fft_plane_length(L0, L1);
    const FftPlan px = make_plan(L0), py = make_plan(L1), pz = make_plan(L2);
    const C* twx = reinterpret_cast<const C*>(tw_for(b, 0));
    const C* twy = reinterpret_cast<const C*>(tw_for(b, 1));
    const C* twz = reinterpret_cast<const C*>(tw_for(b, 2));
    const double2* twx_d = reinterpret_cast<const double2*>(b.tw[0]);
    const double2* twy_d = reinterpret_cast<const double2*>(b.tw[1]);
    const double2* twz_d = reinterpret_cast<const double2*>(b.tw[2]);
    C* fwd = reinterpret_cast<C*>(b.precision == 0 ? (b.spec_fwd ? b.spec_fwd : b.spec) : b.spec_lo);
    double2* inv = reinterpret_cast<double2*>(b.spec);
    double normFact = 1.0;
    normFact /= L0;
    normFact /= L1;
    normFact /= L2;
    if (parts & kConvForwardPart) {
        const AccIn acc{reinterpret_cast<ulonglong2*>(b.nacc), b.st, b.bc.dT, b.bc.rdT, b.dep_weights};
        if (b.periodic_z)
            with_length(L2, LaunchA<T, true>{(T*)b.rho, fwd, n0, n1, n2, L0, L1, pz, twz, s});
        else
            with_length(L2, LaunchA<T>{(T*)b.rho, fwd, n0, n1, n2, L0, L1, pz, twz, s,
                                       (parts & kConvAssemble) ? &acc : nullptr});
        if (!plane) with_length(L1, LaunchY<T, false>{fwd, n0, L0, n1, L1, K + 1, py, twy, s});
    }
    // passes C and D, or B, C and D of a plane in one kernel
    auto conv_cd = [&](const void* ghat, bool complex_g) {
        if (plane) {
            launch_plane_conv(L0, PlaneConv{fwd, inv, ghat, b.tw[0], b.tw[1], K + 1, b.precision == 0, complex_g}, s);
            return;
        }
        if (complex_g)
            with_length(L0, LaunchC<T, true>{fwd, inv, (const T*)ghat, n0, n1, L1, (K + 1) * L1, px, twx, twx_d, s});
        else
            with_length(L0, LaunchC<T>{fwd, inv, (const T*)ghat, n0, n1, L1, (K + 1) * L1, px, twx, twx_d, s});
        with_length(L1, LaunchY<double, true>{inv, n0, L0, L1, n1, K + 1, py, twy_d, s});
    };
    if ((parts & kConvRestPart) && b.periodic_z) {
        conv_cd(b.ghat_img, true);
        if (mode == kConvSelfField)
            with_length(L2, LaunchE<true, false, true>{inv, b.phi, n0, n1, n2, L0, L1, pz, twz_d, b.st, normFact,
                                                       b.bc.coupling, s});
        else
            with_length(L2, LaunchE<false, false, true>{inv, b.phi, n0, n1, n2, L0, L1, pz, twz_d, b.st, normFact,
                                                        b.bc.coupling, s});
        return;
    }
    if (parts & kConvRestPart) {
        conv_cd(b.ghat, false);
        if (mode == kConvSelfField)
            with_length(L2, LaunchE<true>{inv, b.phi, n0, n1, n2, L0, L1, pz, twz_d, b.st, normFact, b.bc.coupling, s});
        else
            with_length(L2, LaunchE<false>{inv, b.phi, n0, n1, n2, L0, L1, pz, twz_d, b.st, normFact, b.bc.coupling, s});
    }
    if (parts & kConvImagePart) {
        conv_cd(b.ghat_img, true);
        if (mode == kConvSelfField)
            with_length(L2, LaunchE<true, true>{inv, b.phi, n0, n1, n2, L0, L1, pz, twz_d, b.st, normFact, b.bc.coupling, s});
        else
            with_length(L2,
                        LaunchE<false, true>{inv, b.phi, n0, n1, n2, L0, L1, pz, twz_d, b.st, normFact, b.bc.coupling, s});
    }
}

void launch_convolution(const DevBunch& b, int mode, cudaStream_t s) {
    launch_convolution_part(b, mode, kConvForwardPart | kConvRestPart, s);
}

void launch_convolution_part(const DevBunch& b, int mode, int parts, cudaStream_t s) {
    if (b.precision == 0)
        convolution_t<double>(b, mode, parts, s);
    else
        convolution_t<float>(b, mode, parts, s);
}

void fft_set_smem_limits() {
    SetLimits sl;
    sl.run<32>();
    sl.run<64>();
    sl.run<96>();
    sl.run<128>();
    sl.run<256>();
    sl.run<0>();
    fft_plane_set_limits();
}

}  // namespace sc
