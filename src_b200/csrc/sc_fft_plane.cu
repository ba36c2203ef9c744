// sc_fft_plane.cu -- the transforms of a whole kz plane in one kernel, for
// meshes with n0 = n1 (16, 32 or 64 cells across: lines of 32, 64 or 128
// points).
//
//   k_fft_plane_conv  passes B, C and D: a cluster of blocks holds the plane's
//                     doubled rows in its shared memory, so the spectrum goes
//                     through L2 once in and once out (three times each for
//                     the separate passes) and two kernel boundaries are gone
//   k_dct_plane       the cosine transforms of G along y and x
//
// Both run the register-resident line transform (sc_fft_lines.cuh): the same
// butterflies, twiddles and operation order as the separate passes, so the
// same bits.  Compiled without FMA contraction, as sc_fft.cu.
#include "sc_fft_lines.cuh"

namespace sc {
namespace {

// ---------------------------------------------------------------- clusters
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// shared::cluster address of this block's shared address `a` in block `rank`
__device__ __forceinline__ unsigned map_rank(unsigned a, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster(unsigned a, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned a, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ double2 ld_cluster(unsigned a) {
    double2 v;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}

// ---------------------------------------------------------------- passes B, C, D
// A plane of L x L points (n = L/2 columns of L rows in, n x n out) on CL
// blocks: block `rank` transforms the columns x in [rank COLS, ...) along y
// and the rows ky in [rank ROWS, ...) along x.
//   1  forward y transform of the own columns (rows y < n in); row ky of the
//      result goes to the block that owns it (distributed shared memory)
//   2  own rows: forward x transform, times the spectrum of G, inverse x
//      transform, x < n kept in place
//   3  own columns back from their rows, inverse y transform, rows y < n out
// The y transforms use the first half of the block's threads (COLS = ROWS/2
// lines of TL threads, lanes along x).
//
// Bound by latency (64^3: FP64 pipe 29 %, 16 warps per SM at 128 registers).
// Convolution phase, separate passes -> this kernel: 64^3 38.9 -> 32.8 us
// (mixed 38.7 -> 29.8), 32^3 24.6 -> 18.4, 16^3 25.5 -> 17.4.  256-point
// lines stay with the separate passes: a plane is 512 KB, eight blocks of one
// per SM.
template <int L>
struct PlaneGeo {
    using G = LineGeo<L>;
    static constexpr int N = L / 2;
    // blocks per plane: enough that the n + 1 planes fill the SMs
    static constexpr int CL = L == 32 ? 2 : 4;
    static constexpr int ROWS = L / CL, COLS = N / CL;
    static constexpr int NT = G::TL * ROWS, NY = G::TL * COLS;
    static constexpr int PITCH = L + 9;  // exchange buffer of a line; odd, so the lines of one access fall in distinct banks
    static constexpr size_t SMEM = (size_t)ROWS * N * sizeof(double2) + (size_t)ROWS * PITCH * sizeof(double2);
    static_assert(NY % 32 == 0, "whole warps in the y transforms");
};

template <typename TI, bool CG, int L>
__device__ __forceinline__ void plane_conv_body(const Cx<TI>* in, double2* out, const TI* __restrict__ ghat,
                                                const Cx<TI>* __restrict__ twx, const double2* __restrict__ twxo,
                                                const Cx<TI>* __restrict__ twy, const double2* __restrict__ twyo, int kz,
                                                int rank) {
    using CI = Cx<TI>;
    using P = PlaneGeo<L>;
    using G = LineGeo<L>;
    constexpr int N = P::N, M = G::M, TL = G::TL;
    extern __shared__ __align__(16) unsigned char plane_smem[];
    // rows of N complex doubles; the mixed form's forward rows use the first half of each row
    double2* rows = reinterpret_cast<double2*>(plane_smem);
    double2* xb = rows + P::ROWS * N;
    const unsigned rows_s = (unsigned)__cvta_generic_to_shared(rows);
    const int t = threadIdx.x;
    const bool ycol = t < P::NY;
    const int li = t % P::COLS, ay = t / P::COLS;  // y transforms: column li, part ay
    const int x = rank * P::COLS + li;
    cluster_arrive();  // every block of the cluster has started before its rows are written
    CI v[M];
    if (ycol) {
        const CI* col = in + (size_t)kz * L * L + x;
#pragma unroll
        for (int m = 0; m < M; ++m) v[m] = m < M / 2 ? col[(size_t)(ay + TL * m) * L] : CI{(TI)0, (TI)0};
        line_fft<TI, false, true, L, P::NY>(v, ay, reinterpret_cast<CI*>(xb + li * P::PITCH), twy);
    }
    cluster_wait();
    if (ycol) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int ky = ay + TL * m;
            st_cluster(map_rank(rows_s + (unsigned)(((ky % P::ROWS) * N) * sizeof(double2) + x * sizeof(CI)),
                                (unsigned)(ky / P::ROWS)),
                       v[m]);
        }
    }
    cluster_arrive();
    // row r of this block: ky = rank ROWS + r, 8 (4) threads of one warp
    const int r = t / TL, a = t % TL;
    const int ky = rank * P::ROWS + r;
    const int gy = ky <= N ? ky : L - ky;
    const size_t grow = ((size_t)kz * (N + 1) + gy) * (N + 1);
    double2* row = rows + r * N;
    double2 w[M];
    {
        // the row of G's spectrum is on its way while the cluster gathers
        using GV = typename std::conditional<CG, CI, TI>::type;
        GV g[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int kx = a + TL * m;
            g[m] = reinterpret_cast<const GV*>(ghat)[grow + (kx <= N ? kx : L - kx)];
        }
        cluster_wait();
        CI f[M];
#pragma unroll
        for (int m = 0; m < M; ++m)
            f[m] = m < M / 2 ? reinterpret_cast<const CI*>(row)[a + TL * m] : CI{(TI)0, (TI)0};
        line_fft<TI, false, true, L>(f, a, reinterpret_cast<CI*>(xb + r * P::PITCH), twx);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            if constexpr (CG)
                w[m] = double2{(double)(f[m].x * g[m].x - f[m].y * g[m].y), (double)(f[m].x * g[m].y + f[m].y * g[m].x)};
            else
                w[m] = double2{(double)(f[m].x * g[m]), (double)(f[m].y * g[m])};
        }
    }
    line_fft<double, true, false, L>(w, a, xb + r * P::PITCH, twxo);
#pragma unroll
    for (int m = 0; m < M / 2; ++m) row[a + TL * m] = w[m];
    cluster_arrive();
    cluster_wait();
    if (ycol) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int k = ay + TL * m;
            w[m] = ld_cluster(map_rank(rows_s + (unsigned)(((k % P::ROWS) * N + x) * sizeof(double2)),
                                       (unsigned)(k / P::ROWS)));
        }
        line_fft<double, true, false, L, P::NY>(w, ay, xb + li * P::PITCH, twyo);
    }
    cluster_arrive();  // this block has read its columns
    if (ycol) {
        double2* col = out + (size_t)kz * L * L + x;
#pragma unroll
        for (int m = 0; m < M / 2; ++m) col[(size_t)(ay + TL * m) * L] = w[m];
    }
    cluster_wait();  // the rows stay until every block has
}

template <typename TI, bool CG, int L>
__global__ void __cluster_dims__(PlaneGeo<L>::CL, 1, 1) __launch_bounds__(PlaneGeo<L>::NT, L == 128 ? 2 : 4)
    k_fft_plane_conv(const Cx<TI>* in, double2* out, const TI* __restrict__ ghat, const Cx<TI>* __restrict__ twx,
                     const double2* __restrict__ twxo, const Cx<TI>* __restrict__ twy,
                     const double2* __restrict__ twyo) {
    constexpr int CL = PlaneGeo<L>::CL;
    plane_conv_body<TI, CG, L>(in, out, ghat, twx, twxo, twy, twyo, blockIdx.x / CL, blockIdx.x % CL);
}

// Batched: a bunch's blocks start at a multiple of the cluster size (every
// item of the launch has CL blocks per plane).
template <typename T, int L>
__global__ void __cluster_dims__(PlaneGeo<L>::CL, 1, 1) __launch_bounds__(PlaneGeo<L>::NT, L == 128 ? 2 : 4)
    k_fft_plane_conv_batch(const DevBunch* __restrict__ tab, const int4* __restrict__ work, int nitems) {
    const int4 w = resolve_block(work, nitems);
    const DevBunch& d = tab[w.x];
    const double2* tx = reinterpret_cast<const double2*>(d.tw[0]);
    const double2* ty = reinterpret_cast<const double2*>(d.tw[1]);
    const Cx<T>*txi, *tyi;
    const Cx<T>* fwd;
    if constexpr (sizeof(T) == sizeof(double)) {
        txi = tx;
        tyi = ty;
        fwd = reinterpret_cast<const Cx<T>*>(d.spec);
    } else {  // the float table follows the double one
        txi = reinterpret_cast<const Cx<T>*>(tx + L);
        tyi = reinterpret_cast<const Cx<T>*>(ty + L);
        fwd = reinterpret_cast<const Cx<T>*>(d.spec_lo);
    }
    plane_conv_body<T, false, L>(fwd, reinterpret_cast<double2*>(d.spec), (const T*)d.ghat, txi, tx, tyi, ty, w.z, w.y);
}

// ---------------------------------------------------------------- G, y and x
// The cosine transforms of one z plane of G ((n+1) x (n+1) reals, x fastest)
// along y, then x, one block per plane: two real lines per complex line (lines
// 2p and 2p + 1 as its real and imaginary parts), even extensions of L points.
// The plane between the transforms stays in shared memory (the separate
// passes write it to global memory and launch a second kernel).  One block
// per plane leaves SMs to the deposit that runs beside it.  With the z pass
// on 256 threads, Green's-function phase 22.4 -> 16.4 us at 16^3, 25.0 -> 19.6
// at 32^3, unchanged at 64^3 (36 us; 33.8 since k_dct_z_lines), where the step
// gains the launch.  At 256 points a plane and its lines do not fit one block's shared memory.
template <int L>
struct DctGeo {
    using G = LineGeo<L>;
    static constexpr int N = L / 2;
    static constexpr int PAIRS = N / 2 + 1;                       // pairs of the n + 1 lines
    static constexpr int LB = (PAIRS * G::TL + 31) / 32 * 32 / G::TL;  // with the idle lines of the last warp
    static constexpr int NT = LB * G::TL;
    static constexpr int PP = N + 2;       // plane row: even, so a pair is one 16-byte access
    static constexpr int PITCH = L + 9;
    static constexpr size_t SMEM = ((size_t)(N + 1) * PP + 2 * (size_t)LB * PITCH) * sizeof(double);
};

template <typename TO, int L>
__device__ __forceinline__ void dct_plane_body(const double* __restrict__ in, TO* __restrict__ out,
                                               const double2* __restrict__ twy, const double2* __restrict__ twx,
                                               int plane) {
    using D = DctGeo<L>;
    using G = LineGeo<L>;
    constexpr int N = D::N, M = G::M, TL = G::TL, PP = D::PP;
    extern __shared__ __align__(16) unsigned char plane_smem[];
    double* S = reinterpret_cast<double*>(plane_smem);
    double2* xb = reinterpret_cast<double2*>(S + (N + 1) * PP);
    const int t = threadIdx.x;
    const double* src = in + (size_t)plane * (N + 1) * (N + 1);
    double2 v[M];
    {  // along y, lanes along the pairs of columns
        const int p = t % D::LB, a = t / D::LB;
        const bool one = p < D::PAIRS, two = 2 * p + 1 <= N;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int e = a + TL * m;
            const double* q = src + (size_t)(e <= N ? e : L - e) * (N + 1) + 2 * p;
            v[m] = double2{one ? q[0] : 0.0, two ? q[1] : 0.0};
        }
        line_fft<double, false, false, L, 1>(v, a, xb + p * D::PITCH, twy);
        if (one) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int e = a + TL * m;
                if (e <= N) *reinterpret_cast<double2*>(S + e * PP + 2 * p) = v[m];  // the pad column takes the odd end
            }
        }
    }
    __syncthreads();
    // along x, the threads of a line beside each other
    const int p = t / TL, a = t % TL;
    const bool one = p < D::PAIRS, two = 2 * p + 1 <= N;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int e = a + TL * m;
        const double* q = S + (2 * p) * PP + (e <= N ? e : L - e);
        v[m] = double2{one ? q[0] : 0.0, two ? q[PP] : 0.0};
    }
    line_fft<double, false, false, L>(v, a, xb + p * D::PITCH, twx);
    TO* dst = out + (size_t)plane * (N + 1) * (N + 1);
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const int e = a + TL * m;
        if (e > N) continue;
        if (one) dst[(size_t)(2 * p) * (N + 1) + e] = (TO)v[m].x;
        if (two) dst[(size_t)(2 * p + 1) * (N + 1) + e] = (TO)v[m].y;
    }
}

template <typename TO, int L>
__global__ void __launch_bounds__(DctGeo<L>::NT) k_dct_plane(const double* __restrict__ in, TO* __restrict__ out,
                                                             const double2* __restrict__ twy,
                                                             const double2* __restrict__ twx) {
    dct_plane_body<TO, L>(in, out, twy, twx, blockIdx.x);
}

template <typename T, int L>
__global__ void __launch_bounds__(DctGeo<L>::NT) k_dct_plane_batch(const DevBunch* __restrict__ tab,
                                                                   const int4* __restrict__ work, int nitems) {
    const int4 w = resolve_block(work, nitems);
    const DevBunch& d = tab[w.x];
    dct_plane_body<T, L>(d.gline, (T*)d.ghat, reinterpret_cast<const double2*>(d.tw[1]),
                         reinterpret_cast<const double2*>(d.tw[0]), w.y);
}

// f.run<L>() for the plane kernels' line lengths
template <typename F>
void with_plane_length(int L, F&& f) {
    switch (L) {
        case 32: f.template run<32>(); break;
        case 64: f.template run<64>(); break;
        default: f.template run<128>(); break;
    }
}

struct LaunchDctPlane {
    const double* in;
    void* out;
    bool out_f64;
    int planes;
    const double2 *twy, *twx;
    cudaStream_t s;
    template <int L>
    void run() {
        using D = DctGeo<L>;
        if (out_f64)
            k_dct_plane<double, L><<<planes, D::NT, D::SMEM, s>>>(in, (double*)out, twy, twx);
        else
            k_dct_plane<float, L><<<planes, D::NT, D::SMEM, s>>>(in, (float*)out, twy, twx);
    }
};

struct LaunchDctPlaneBatch {
    bool f64;
    const DevBunch* tab;
    const int4* items;
    int nitems, nblocks;
    cudaStream_t s;
    template <int L>
    void run() {
        using D = DctGeo<L>;
        if (f64)
            k_dct_plane_batch<double, L><<<nblocks, D::NT, D::SMEM, s>>>(tab, items, nitems);
        else
            k_dct_plane_batch<float, L><<<nblocks, D::NT, D::SMEM, s>>>(tab, items, nitems);
    }
};

struct AllowDctPlane {
    template <int L>
    void run() {
        const int sm = (int)DctGeo<L>::SMEM;
        cudaFuncSetAttribute(k_dct_plane<double, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        cudaFuncSetAttribute(k_dct_plane<float, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        cudaFuncSetAttribute(k_dct_plane_batch<double, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        cudaFuncSetAttribute(k_dct_plane_batch<float, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    }
};

template <int L>
void conv_plane_l(const PlaneConv& c, cudaStream_t s) {
    constexpr size_t SM = PlaneGeo<L>::SMEM;
    const int blocks = c.planes * PlaneGeo<L>::CL, nt = PlaneGeo<L>::NT;
    const double2* tx = reinterpret_cast<const double2*>(c.tw0);
    const double2* ty = reinterpret_cast<const double2*>(c.tw1);
    if (c.f64) {
        auto k = c.complex_g ? k_fft_plane_conv<double, true, L> : k_fft_plane_conv<double, false, L>;
        k<<<blocks, nt, SM, s>>>((const double2*)c.in, c.out, (const double*)c.ghat, tx, tx, ty, ty);
    } else {
        auto k = c.complex_g ? k_fft_plane_conv<float, true, L> : k_fft_plane_conv<float, false, L>;
        k<<<blocks, nt, SM, s>>>((const float2*)c.in, c.out, (const float*)c.ghat, (const float2*)(tx + L), tx,
                                 (const float2*)(ty + L), ty);
    }
}

template <int L>
void allow_l() {
    const int sm = (int)PlaneGeo<L>::SMEM;
    cudaFuncSetAttribute(k_fft_plane_conv<double, true, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fft_plane_conv<double, false, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fft_plane_conv<float, true, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fft_plane_conv<float, false, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fft_plane_conv_batch<double, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_fft_plane_conv_batch<float, L>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
}

}  // namespace

bool fft_plane_length(int L0, int L1) { return fft_register_lines() && L0 == L1 && (L0 == 32 || L0 == 64 || L0 == 128); }

int fft_plane_cluster(int L) { return L == 32 ? PlaneGeo<32>::CL : L == 64 ? PlaneGeo<64>::CL : PlaneGeo<128>::CL; }

void launch_plane_conv(int L, const PlaneConv& c, cudaStream_t s) {
    if (L == 32)
        conv_plane_l<32>(c, s);
    else if (L == 64)
        conv_plane_l<64>(c, s);
    else
        conv_plane_l<128>(c, s);
}

void launch_plane_conv_batch(int L, int precision, const DevBunch* tab, const int4* items, int nitems, int nblocks,
                             cudaStream_t s) {
    const bool f64 = precision == 0;
    if (L == 32) {
        auto k = f64 ? k_fft_plane_conv_batch<double, 32> : k_fft_plane_conv_batch<float, 32>;
        k<<<nblocks, PlaneGeo<32>::NT, PlaneGeo<32>::SMEM, s>>>(tab, items, nitems);
    } else if (L == 64) {
        auto k = f64 ? k_fft_plane_conv_batch<double, 64> : k_fft_plane_conv_batch<float, 64>;
        k<<<nblocks, PlaneGeo<64>::NT, PlaneGeo<64>::SMEM, s>>>(tab, items, nitems);
    } else {
        auto k = f64 ? k_fft_plane_conv_batch<double, 128> : k_fft_plane_conv_batch<float, 128>;
        k<<<nblocks, PlaneGeo<128>::NT, PlaneGeo<128>::SMEM, s>>>(tab, items, nitems);
    }
}

void launch_dct_plane(int L, const double* in, void* out, bool out_f64, int planes, const void* tw1, const void* tw0,
                      cudaStream_t s) {
    with_plane_length(L, LaunchDctPlane{in, out, out_f64, planes, (const double2*)tw1, (const double2*)tw0, s});
}

void launch_dct_plane_batch(int L, int precision, const DevBunch* tab, const int4* items, int nitems, int nblocks,
                            cudaStream_t s) {
    with_plane_length(L, LaunchDctPlaneBatch{precision == 0, tab, items, nitems, nblocks, s});
}

void fft_plane_set_limits() {
    allow_l<32>();
    allow_l<64>();
    allow_l<128>();
    AllowDctPlane a;
    a.run<32>();
    a.run<64>();
    a.run<128>();
}

}  // namespace sc
