// Host build of crmath.cuh's short evaluations for tests/test_crmath_short.py:
// on n arguments, how many pass the rounding test (*taken) and how many of
// those differ in any bit from the full evaluation (returned).
#include <cmath>
#include <cstdint>
#include <cstring>

#include "crmath.cuh"

namespace cr = sa::cr;

static bool differ(double a, double b) { return std::memcmp(&a, &b, 8) != 0; }

extern "C" long cr_short_check(int f, const double* x, long n, long* taken) {
    long bad = 0;
    *taken = 0;
    for (long i = 0; i < n; i++) {
        double y = 0, s = 0, c = 0, fs = 0, fc = 0;
        bool ok;
        if (f == 0) ok = cr::exp_short(x[i], &y);
        else if (f == 1) ok = cr::log_short(x[i], &y);
        else ok = cr::sincos_short(x[i], &s, &c);
        if (!ok) continue;
        ++*taken;
        if (f == 0) bad += differ(y, cr::exp_full(x[i]));
        else if (f == 1) bad += differ(y, cr::log_full(x[i]));
        else {
            cr::sincos_full(x[i], &fs, &fc);
            bad += differ(s, fs) || differ(c, fc);
        }
    }
    return bad;
}
