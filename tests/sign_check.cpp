// Host build of the dispersion search's approximate secular functions
// (surfker_search.cuh: dltar4_near, dltar1_near) for tests/test_sign_check.py:
// the largest |near - exact| over `n` evaluations that the search would trust
// (not NaN), exact being dltar4 / dltar1 (normalised likewise), and how many
// were not trusted.  `where`: 0 any trial velocity, 1 next to the half-space's
// shear velocity, 2 next to a layer's, 3 next to the half-space's compressional.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

#include <cuda_runtime.h>
static inline double __longlong_as_double(long long v) {
    double d;
    std::memcpy(&d, &v, 8);
    return d;
}
using std::fabs;
using std::max;
using std::min;
using std::signbit;
#define __syncthreads()
#define __noinline__
#include "surfker_search.cuh"

using namespace sa::sk;

extern "C" double sign_check(int love, int tables, int where, double pmin, double pmax, double dmin,
                             double dmax, long n, unsigned long seed, long* untrusted) {
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    auto logu = [&](double a, double b) { return a * std::pow(b / a, U(g)); };
    double worst = 0.0;
    *untrusted = 0;
    for (long i = 0; i < n; i++) {
        SDModel M;
        M.mmax = 3 + (int)(U(g) * (MMAX - 2));
        M.llw = 1;
        const double thick = logu(dmin, dmax);
        double xka[MMAX], xkb[MMAX], gk[MMAX], rr[MMAX], r2[MMAX];
        for (int m = 0; m < M.mmax; m++) {
            const double vs = 2.0 + 2.8 * m / M.mmax + 0.3 * (U(g) - 0.5);
            M.b[m] = (float)vs;
            M.a[m] = (float)(1.75 * vs);
            M.rho[m] = (float)(2.3 + 0.2 * vs);
            M.d[m] = m + 1 < M.mmax ? (float)(thick * (0.7 + 0.6 * U(g))) : 0.0f;
        }
        const double omega = 2.0 * 3.141592653589793 / logu(pmin, pmax);
        const int k = (int)(U(g) * (M.mmax - 1));
        const double at = where == 1 ? (double)M.b[M.mmax - 1] : where == 2 ? (double)M.b[k]
                        : where == 3 ? (double)M.a[M.mmax - 1] : 1.6 + 3.2 * U(g);
        const double c = where ? at * (1.0 + (U(g) < 0.5 ? -1.0 : 1.0) * logu(1e-16, 1e-3)) : at;
        const double wvno = omega / c;
        Layers Y{M.mmax, M.llw, M.d, M.a, M.b, M.rho, nullptr, nullptr, nullptr, nullptr, nullptr};
        double near;
        if (tables) {   // as the groups' kernel fills them
            const double w = omega < 1.0e-4 ? 1.0e-4 : omega;
            for (int m = 0; m < M.mmax; m++) {
                const double t = (double)M.b[m] / w, r = (double)M.rho[m], b = (double)M.b[m];
                xka[m] = w / (double)M.a[m];
                xkb[m] = (love ? omega : w) / b;
                gk[m] = 2.0 * t * t;
                r2[m] = love ? r * b * b : 1.0 / (r * r);
                rr[m] = love ? 1.0 / r2[m] : 1.0 / r;
            }
            Y.xka = xka;
            Y.xkb = xkb;
            Y.gk = gk;
            Y.rr = rr;
            Y.r2 = r2;
            near = love ? dltar1_near<true>(Y, wvno, omega) : dltar4_near<true>(Y, wvno, omega);
        } else {
            near = love ? dltar1_near<false>(Y, wvno, omega) : dltar4_near<false>(Y, wvno, omega);
        }
        if (near != near) {
            ++*untrusted;
            continue;
        }
        const double exact = love ? dltar1(M, wvno, omega) : dltar4(M, wvno, omega);
        worst = std::max(worst, fabs(near - exact));
    }
    return worst;
}
