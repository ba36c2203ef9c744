// log and atan of sc_ddmath.cuh on the device, whose quick atan takes another
// reciprocal and another first quotient than the host's.  Prints
//   <n> <log_dd != log_dd_full> <atan_dd != atan_dd_full> <log_dd != host> <atan_dd != host>
//   <log_fast != host> <atan_fast further than one double from atan_dd> <atan_fast != atan_dd>
//   <largest |1 - d rcp_approx(d)|>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "sc_ddmath.cuh"

using namespace sc::ddm;

// log_dd, atan_dd and log_fast of the host build (ddmath_host_eval.cpp)
extern "C" void host_eval(double x, double y, double* log_cr, double* atan_cr, double* log_quick);

struct Out {
    double log_cr, log_full, log_quick, atan_cr, atan_full, atan_quick, rcp;
};

__global__ void k_eval(const double* x, const double* y, const double* d, Out* o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = Out{log_dd(x[i]), log_dd_full(x[i]), log_fast(x[i]), atan_dd(y[i]), atan_dd_full(y[i]), atan_fast(y[i]),
               rcp_approx(d[i])};
}

int main(int argc, char** argv) {
    const int n = argc > 1 ? std::atoi(argv[1]) : 1000000;
    std::mt19937_64 g(777);
    std::uniform_real_distribution<double> mant(1.0, 2.0), w(-1.0 / 128, 1.0 / 128);
    std::uniform_int_distribution<int> xl(-43, 43), xa(-32, 31), xd(0, 30);
    std::vector<double> x(n), y(n), d(n);
    for (int i = 0; i < n; ++i) {
        const bool table = i % 4 == 3;  // every table interval, edges included
        x[i] = table ? (90 + (i / 4) % 93) / 128.0 + w(g) : std::ldexp(mant(g), xl(g));
        const double t = ((i / 4) % 129) / 128.0 + w(g) / 2;
        y[i] = table ? ((i & 4) && t != 0.0 ? 1.0 / t : t) : ((i & 1) ? -1.0 : 1.0) * std::ldexp(mant(g), xa(g));
        d[i] = std::ldexp(mant(g), xd(g));
    }
    const size_t bytes = sizeof(double) * (size_t)n;
    double *dx = nullptr, *dy = nullptr, *dd = nullptr;
    Out* dout = nullptr;
    std::vector<Out> o(n);
    if (cudaMalloc(&dx, bytes) || cudaMalloc(&dy, bytes) || cudaMalloc(&dd, bytes) || cudaMalloc(&dout, sizeof(Out) * (size_t)n))
        return 2;
    cudaMemcpy(dx, x.data(), bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(dy, y.data(), bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(dd, d.data(), bytes, cudaMemcpyHostToDevice);
    k_eval<<<(n + 255) / 256, 256>>>(dx, dy, dd, dout, n);
    if (cudaMemcpy(o.data(), dout, sizeof(Out) * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    long lf = 0, af = 0, lh = 0, ah = 0, lq = 0, far = 0, off = 0;
    double rcp = 0.0;
    for (int i = 0; i < n; ++i) {
        lf += o[i].log_cr != o[i].log_full;
        af += o[i].atan_cr != o[i].atan_full;
        double l, a0, q;
        host_eval(x[i], y[i], &l, &a0, &q);
        lh += o[i].log_cr != l;
        ah += o[i].atan_cr != a0;
        lq += o[i].log_quick != q;
        if (atan_range(y[i])) {
            const double a = o[i].atan_cr, v = o[i].atan_quick;
            off += v != a;
            far += v < std::nextafter(a, -INFINITY) || v > std::nextafter(a, INFINITY);
        }
        rcp = std::fmax(rcp, std::fabs(std::fma(-d[i], o[i].rcp, 1.0)));
    }
    std::printf("%d %ld %ld %ld %ld %ld %ld %ld %.3e\n", n, lf, af, lh, ah, lq, far, off, rcp);
    return 0;
}
