// Checks inv_roots_in of csrc/p3t_exact.cuh: y, y^3, y^4 and y^5 of y = 1 / sqrt(x)
// within 0.6 units of the last place of long double references (64 bits; the
// bound is one rounding, 0.5, and 2^-57 relative of fixed-point truncation, with
// the references' own few 2^-64), over argv[1] operands of the accepted exponents,
// the FP32 seed perturbed by up to three units.  Compiled by nvcc it also
// compares the device's results, with the GPU's seeds.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "p3t_exact.cuh"
using namespace p3t;

static std::mt19937_64 g(11);
static double operand(long i) {
    uint64_t m = g() & (EX_ONE - 1);
    if (i % 4 == 1) m = g() % 64;
    if (i % 4 == 2) m = EX_ONE - 1 - g() % 64;
    const uint32_t e = i % 16 == 3 ? 643 : i % 16 == 7 ? 1402 : i % 16 == 11 ? 1022 + g() % 3 : 643 + g() % 760;
    return ex_double(((uint64_t)e << 52) | m);
}
static bool near(double v, long double p) {
    return std::fabs((long double)v - p) <= 0.6L * std::ldexp(1.0L, std::ilogb(p) - 52);
}
static long wrong(double x, const InvRoots &r) {
    const long double y2 = 1.0L / (long double)x, y = std::sqrt(y2);
    return !near(r.y1, y) + !near(r.y3, y2 * y) + !near(r.y4, y2 * y2) + !near(r.y5, y2 * y2 * y);
}
#ifdef __CUDACC__
__global__ void on_device(const double *x, int n, InvRoots *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = inv_roots_in<true>(x[i]);
}
#endif

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    long bad = 0;
#ifndef __CUDACC__
    for (long i = 0; i < n; i++) {
        const double x = operand(i);
        bad += wrong(x, inv_roots_in<true>(x));
        const uint64_t X = (g() >> 2) + (g() & 1 ? 1ULL << 62 : 2ULL << 62);  // the root alone, seeds perturbed
        const float f = (float)std::ldexp((double)X, -62);
        uint32_t fb;
        std::memcpy(&fb, &f, 4);
        if (f >= 4.f) continue;
        const long double want = 1.0L / std::sqrt(std::ldexp((long double)X, -62));
        const long double got = std::ldexp((long double)ex_rsqrt63(X, ex_rsqrt32(fb) + (uint32_t)(g() % 7) - 3u), -63);
        bad += !(std::fabs(got - want) <= 0x1p-59L);
    }
    for (const double x : {0., 1. / 0., 0. / 0., 5e-324, std::ldexp(1., -381), std::ldexp(1., 380), -1.})
        bad += ex_inv_roots_range(x);
    bad += !ex_inv_roots_range(std::ldexp(1., -380)) + !ex_inv_roots_range(std::ldexp(1., 379));
#else
    // the host's long double may be wider or narrower than 64 bits on other machines: compare with the
    // host's results of the same function, which the CPU test checks; seeds differ, so one unit is allowed
    const int m = 1 << 18;
    double *h = (double *)std::malloc(m * sizeof(double)), *dx;
    InvRoots *o = (InvRoots *)std::malloc(m * sizeof(InvRoots)), *dv;
    for (int i = 0; i < m; i++) h[i] = operand(i);
    if (cudaMalloc(&dx, m * sizeof(double)) != cudaSuccess || cudaMalloc(&dv, m * sizeof(InvRoots)) != cudaSuccess)
        return 2;
    cudaMemcpy(dx, h, m * sizeof(double), cudaMemcpyHostToDevice);
    on_device<<<m / 256, 256>>>(dx, m, dv);
    if (cudaMemcpy(o, dv, m * sizeof(InvRoots), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    auto apart = [](double a, double b) { return std::llabs((long long)(ex_bits(a) - ex_bits(b))) > 1; };
    for (int i = 0; i < m; i++) {
        const InvRoots w = inv_roots_in<true>(h[i]);
        bad += apart(o[i].y1, w.y1) + apart(o[i].y3, w.y3) + apart(o[i].y4, w.y4) + apart(o[i].y5, w.y5);
    }
    (void)wrong;
#endif
    std::printf("%ld operands, %ld wrong\n", n, bad);
    return bad != 0;
}
