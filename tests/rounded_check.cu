// Device check of rounded.cuh for tests/test_gpu_rounded.py: n operands of
// one kind against CUDA's IEEE operations; bad[0..3] count the reciprocals,
// quotients, roots that are sure but differ, and the roots that are not sure.
// kind 0: random mantissas; 1: mantissas of ones, or nearly, and powers of two;
// 2: quotients and roots next to a midpoint of two doubles; 3: squares of
// 26-bit numbers and their neighbours, divisors of few bits.
#include <cmath>
#include <cstdint>
#include <random>
#include <vector>

#include "rounded.cuh"

__global__ void check(long n, const double* a, const double* b, const double* x,
                      unsigned long long* bad) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n;
         i += (long)gridDim.x * blockDim.x) {
        const double rh = __drcp_rn(b[i]);
        if (!sa::low_ones(b[i]) && sa::rcp_rn(b[i]) != rh) atomicAdd(bad, 1ull);
        const double q = sa::quot(a[i], b[i], rh, sa::recip_lo(b[i], rh));
        if (q != __ddiv_rn(a[i], b[i])) atomicAdd(bad + 1, 1ull);
        bool sure;
        const double s = sa::sqrt_rn(x[i], &sure);
        if (!sure) atomicAdd(bad + 3, 1ull);
        else if (s != __dsqrt_rn(x[i])) atomicAdd(bad + 2, 1ull);
    }
}

// the 53 leading bits of v, rounded up or down, as a double in [1, 2)
static double lead(unsigned __int128 v, bool up) {
    int sh = 0;
    while ((v >> sh) >> 53) sh++;
    return std::ldexp((double)((uint64_t)(v >> sh) + (up ? 1 : 0)), -52);
}

extern "C" int rounded_check(int kind, long n, unsigned long seed, unsigned long long* bad) {
    std::mt19937_64 g(seed);
    std::vector<double> a(n), b(n), x(n);
    auto mant = [&]() { return (g() >> 12) | (1ull << 52); };
    auto scale = [&](double m, int range) { return std::ldexp(m, (int)(g() % (2 * range)) - range); };
    for (long i = 0; i < n; i++) {
        uint64_t mb = mant(), ma = mant();
        const uint64_t all = (1ull << 53) - 1;
        if (kind == 1) {
            const uint64_t low = g() % 3 == 0 ? 0 : (1ull << (g() % 53)) - 1;
            mb = (g() & 1) ? all ^ (g() % 4 * (g() & 1)) : (1ull << 52) | low;
            ma = (g() & 1) ? all - g() % 4 : ma;
        } else if (kind == 3) {
            mb = (1ull << 52) | (mb & ~((1ull << 40) - 1));
        }
        b[i] = std::ldexp((double)mb, -52);
        a[i] = std::ldexp((double)ma, -52);
        x[i] = std::ldexp((double)ma, -52 + (int)(g() & 1));
        if (kind == 2) {   // a / b and sqrt(x) half an ulp from a double
            const uint64_t q = 2 * mant() + 1;
            a[i] = lead((unsigned __int128)mb * q, g() & 1);
            // (a 54-bit odd square has 107 or 108 bits: keep its parity)
            unsigned __int128 s = (unsigned __int128)q * q;
            const bool odd = (s >> 107) != 0;
            x[i] = std::ldexp(lead(s, g() & 1), odd ? 1 : 0);
        } else if (kind == 3) {
            const double r = (double)((g() >> 38) | 1);
            x[i] = r * r;
            const int k = (int)(g() % 3);
            if (k) x[i] = std::nextafter(x[i], k == 1 ? 0.0 : 1e300);
        }
        b[i] = scale(b[i], 100) * ((g() & 1) ? 1 : -1);
        a[i] = scale(a[i], 100) * ((g() & 1) ? 1 : -1);
        x[i] = std::ldexp(x[i], 2 * ((int)(g() % 200) - 100));
    }
    double *da, *db, *dx;
    unsigned long long* dn;
    if (cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&dx, n * 8) ||
        cudaMalloc(&dn, 32))
        return 1;
    cudaMemcpy(da, a.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemset(dn, 0, 32);
    check<<<592, 256>>>(n, da, db, dx, dn);
    const int rc = cudaMemcpy(bad, dn, 32, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(da);
    cudaFree(db);
    cudaFree(dx);
    cudaFree(dn);
    return rc;
}
