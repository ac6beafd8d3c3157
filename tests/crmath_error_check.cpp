// Host build of crmath.cuh's short evaluations for tests/test_crmath_error.py:
// the largest error of s + lo, as a share of the eps that the rounding test
// allows it, over n arguments, against quad-precision values; *at is the
// argument.  f: 0 exp, 1 log, 2 sin and cos.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <quadmath.h>

static double g_s[2], g_lo[2], g_eps;
static int g_n;
#define CR_PROBE(s, lo, eps) (g_s[g_n & 1] = s, g_lo[g_n & 1] = lo, g_eps = eps, ++g_n)
#include "crmath.cuh"

namespace cr = sa::cr;

extern "C" double cr_short_error(int f, const double* x, long n, double* at) {
    double worst = 0.0;
    for (long i = 0; i < n; i++) {
        double y, c;
        g_n = 0;
        if (f == 0) cr::exp_short(x[i], &y);
        else if (f == 1) cr::log_short(x[i], &y);
        else cr::sincos_short(x[i], &y, &c);
        for (int k = 0; k < g_n; k++) {
            const __float128 v = (__float128)g_s[k] + g_lo[k], a = x[i];
            __float128 e;
            if (f == 0) {   // up to a power of two
                e = expq(a);
                e = scalbnq(e, ilogbq(v) - ilogbq(e));
                if (e > v * 1.5Q) e *= 0.5Q;
                if (e < v * 0.75Q) e *= 2.0Q;
            } else if (f == 1) {
                e = logq(a);
            } else {
                const __float128 s = fabsq(sinq(a)), q = fabsq(cosq(a));
                if (s < 0x1p-20Q || q < 0x1p-20Q) continue;   // (not accepted)
                e = fabsq(s - v) < fabsq(q - v) ? s : q;
            }
            const double share = (double)(fabsq(v - e) / fabsq(e) / (__float128)g_eps);
            if (share > worst) {
                worst = share;
                *at = x[i];
            }
        }
    }
    return worst;
}
