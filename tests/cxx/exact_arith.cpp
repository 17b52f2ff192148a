// Checks csrc/p3t_exact.cuh bit for bit against the compiler's own sqrt and
// division: argv[1] random operands of every kind (plain, few mantissa bits,
// all ones, near powers of two, near squares and near reciprocals), the FP32
// seeds perturbed by up to three units in the last place, and the special
// values.  Compiled by g++ (the host's IEEE operations) and by nvcc, where it
// also runs the device functions with the GPU's own seeds.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "p3t_exact.cuh"
using namespace p3t;

static std::mt19937_64 g(7);
static uint64_t mantissa(int kind) {
    uint64_t m = g() & (EX_ONE - 1);
    switch (kind % 6) {
        case 1: m = g() % 64; break;
        case 2: m = EX_ONE - 1 - g() % 64; break;
        case 3: m = (EX_ONE >> (1 + g() % 51)) + g() % 3 - 1; break;
        case 4: { const double r = 1 + (double)(g() >> 11) * 0x1p-53; m = ex_bits(r * r); break; }
        case 5: { const double r = 1 + (double)(g() >> 11) * 0x1p-53; m = ex_bits(1 / r); break; }
    }
    return m & (EX_ONE - 1);
}
static double make(uint32_t e, uint64_t m, bool neg) {
    return ex_double(((uint64_t)neg << 63) | ((uint64_t)e << 52) | m);
}
static bool same(double a, double b) { return (a != a && b != b) || ex_bits(a) == ex_bits(b); }

#ifdef __CUDACC__
__global__ void on_device(const double *a, const double *b, int n, double *s, double *r, double *q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    s[i] = sqrt_rn(a[i]);
    r[i] = rcp_rn(a[i]);
    q[i] = div_rn(a[i], b[i]);
}
#endif

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const int pert = (int)(g() % 7) - 3;
        const double x = make(1 + g() % 2046, mantissa((int)i), false);
        const uint64_t bx = ex_bits(x);
        const uint32_t e = (uint32_t)(bx >> 52), odd = (e & 1u) ^ 1u, fx = (uint32_t)(bx >> 29) & 0x7fffffu;
        bad += !same(sqrt_rn(x), std::sqrt(x));
        bad += !same(ex_double(ex_sqrt_core(((bx & (EX_ONE - 1)) | EX_ONE) << (10 + odd),
                                            ex_rsqrt32(((127u + odd) << 23) | fx) + pert, e)), std::sqrt(x));
        const double y = make(1 + g() % 2043, mantissa((int)i / 3), g() & 1);
        const uint32_t fy = 0x3f800000u | ((uint32_t)(ex_bits(y) >> 29) & 0x7fffffu);
        bad += !same(rcp_rn(y), 1. / y);
        bad += !same(ex_double(ex_rcp_core(ex_bits(y), ex_rcp32(fy) + pert)), 1. / y);
        const double d = make(600 + g() % 800, mantissa((int)i / 5), g() & 1);
        const uint32_t fd = 0x3f800000u | ((uint32_t)(ex_bits(d) >> 29) & 0x7fffffu);
        double c = make(600 + g() % 800, mantissa((int)i / 7), g() & 1);
        if (i % 4 == 0) c = d * make(1023, mantissa((int)i / 7), false);  // a quotient near a double
        bad += !same(div_rn(c, d), c / d);
        bad += !same(ex_double(ex_div_core(ex_bits(c), ex_bits(d), ex_rcp32(fd) + pert)), c / d);
    }
    const double sp[] = {0., -0., 1. / 0., -1. / 0., 0. / 0., 5e-324, 2.2250738585072014e-308, 4.4501477170144023e-308,
                         1.7976931348623157e308, 8.9884656743115795e307, -1., 1., 2., 4., 0.25, -2., 3.};
    for (double u : sp) {
        bad += !same(sqrt_rn(u), std::sqrt(u));
        bad += !same(rcp_rn(u), 1. / u);
        for (double v : sp) bad += !same(div_rn(u, v), u / v);
    }
#ifdef __CUDACC__
    const int m = 1 << 20;
    double *h[2], *dv, *out = (double *)std::malloc(3 * m * sizeof(double));
    for (auto &p : h) p = (double *)std::malloc(m * sizeof(double));
    for (int i = 0; i < m; i++) {
        h[0][i] = make(1 + g() % 2046, mantissa(i), false);
        h[1][i] = make(1 + g() % 2046, mantissa(i / 6), g() & 1);
    }
    for (int i = 0; i < (int)(sizeof sp / sizeof *sp); i++) h[0][i] = sp[i];
    if (cudaMalloc(&dv, 5 * m * sizeof(double)) != cudaSuccess) return 2;
    for (int k = 0; k < 2; k++) cudaMemcpy(dv + k * m, h[k], m * sizeof(double), cudaMemcpyHostToDevice);
    on_device<<<m / 256, 256>>>(dv, dv + m, m, dv + 2 * m, dv + 3 * m, dv + 4 * m);
    if (cudaMemcpy(out, dv + 2 * m, 3 * m * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    for (int i = 0; i < m; i++) {
        bad += !same(out[i], std::sqrt(h[0][i]));
        bad += !same(out[m + i], 1. / h[0][i]);
        bad += !same(out[2 * m + i], h[0][i] / h[1][i]);
    }
#endif
    std::printf("%ld operands, %ld differ\n", n, bad);
    return bad != 0;
}
