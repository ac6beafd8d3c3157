// surfdisp96's fundamental-mode root searches on the device: one column per
// thread or per group of G lanes.
//
// A search (getsol, surfdisp96.f:403-498) marches trial velocities c1 +- dc
// until the secular function dltar changes sign and then refines the bracket
// (nevill, :578-711).  Of about 31 evaluations per period only the
// refinement's and the bracket ends' values are used; the march asks for
// signs alone.  So the march evaluates dltar approximately (dltar_near: FP64
// with short table functions, fused multiply-adds and no normalising
// divisions, about a third of the work): its value is within 1e-7 of the
// normalised vector's largest component of dltar's (2e-8 the most seen at
// periods from 1 s, next to a layer's velocity, where dltar itself cancels;
// 3e-11 elsewhere), and a sign is taken from it only where it stands above
// 1e-6 of that; anything smaller, or not a number, is evaluated exactly.
// Trial velocities, brackets and Neville tables are those of the Fortran, so
// the phase velocities are too, bit for bit.
#pragma once
#include "surfker_dev.cuh"

namespace sa {
namespace sk {

// ---------------------------------------------------------------------------
// The secular function's sign: an approximate dltar
// ---------------------------------------------------------------------------
// exp and sin / cos to about 2^-50 from crmath's tables (no second words),
// 1/x and 1/sqrt(x) to about 2^-44 (hardware FP32 value, one Newton step).
__device__ __forceinline__ double exp_near(double x) {   // -700 <= x <= 0
    const double kd = rint(x * CR_EXP_INVL);
    const int k = (int)kd;
    const double h = fma(-kd, CR_EXP_L2, fma(-kd, CR_EXP_L1, x));
    const double p = fma(h * h, fma(h, CR_IFACT3, 0.5), h);
    const double P = cr::CR_TAB(kExpT1)[2 * (k & 63)] * cr::CR_TAB(kExpT2)[2 * ((k >> 6) & 63)];
    return fma(P, p, P) * cr::bits_to_double((uint64_t)(1023 + (k >> 12)) << 52);
}
__device__ __forceinline__ void sincos_near(double x, double* sn, double* cs) {   // 0 <= x < 1e5
    const double kd = rint(x * CR_2OPI);
    const double h = fma(-kd, CR_PIO2_2, fma(-kd, CR_PIO2_1, x));
    const double aj = rint(fabs(h) * 256.0);
    const int j = min((int)aj, CR_SC_N - 1);
    const double t = fma(aj, -1.0 / 256.0, fabs(h));
    const double z = t * t;
    const double st = fma(t * z, fma(z, CR_IFACT5, -CR_IFACT3), t);
    const double ct = z * fma(z, CR_IFACT4, -0.5);   // cos t - 1
    const double S = cr::CR_TAB(kSinT)[2 * j], C = cr::CR_TAB(kCosT)[2 * j];
    double s = S + fma(C, st, S * ct);
    const double c = C + fma(C, ct, -(S * st));
    s = copysign(s, h);
    const int q = (int)kd & 3;
    const double a = (q & 1) ? c : s, b = (q & 1) ? s : c;
    *sn = (q & 2) ? -a : a;
    *cs = (q == 1 || q == 2) ? -b : b;
}
__device__ __forceinline__ double rcp_near(double x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((float)x));
#else
    const float r = 1.0f / (float)x;
#endif
    const double y = (double)r;
    return fma(y, fma(-x, y, 1.0), y);
}
__device__ __forceinline__ double rsqrt_near(double x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((float)x));
#else
    const float r = 1.0f / sqrtf((float)x);
#endif
    const double y = (double)r;
    return fma(y, fma(-0.5 * x * y, y, 0.5), y);
}
// a power of two near 1/x (x > 0, normal)
__device__ __forceinline__ double pow2_rcp(double x) {
    return cr::bits_to_double((uint64_t)(2046 - (int)(cr::double_to_bits(x) >> 52)) << 52);
}

// One vertical wavenumber's functions over a layer: cos and sin / r, r sin
// (trigonometric below the layer's wavenumber, scaled hyperbolic above) and
// the hyperbolic scale e = exp(-r d), or 1; NaN where they are not accurate
// enough to be trusted.  xk from rcp_near is off by 2^-46, which moves cos and
// sin by up to (xk d)^2 2^-46 (below 1e-9 for xk d < 256); rsqrt_near moves
// the phase p by up to p 2^-43 (1e-10 at 1e3).
template <bool TAB>
__device__ __forceinline__ void wave_near(double wvno, double xk, double d, double& co,
                                          double& sr, double& rs, double& e) {
    const double s = (wvno + xk) * (wvno - xk);
    const double r2 = fabs(s);
    const double ir = rsqrt_near(r2);
    const double r = r2 * ir;
    const double p = r * d;
    const bool in = TAB ? s >= 0.0 || p < 1e3 : xk * d < 256.0;
    if (s < 0.0) {
        double sn;
        sincos_near(in ? p : 0.0, &sn, &co);
        sr = sn * ir;
        rs = -(r * sn);
        e = 1.0;
    } else {
        e = exp_near(-fmin(p, 700.0));
        const double f = e * e;
        co = fma(0.5, f, 0.5);
        const double sn = fma(-0.5, f, 0.5);
        sr = sn * ir;
        rs = r * sn;
    }
    if (!in) e = __longlong_as_double(0x7ff8000000000000ll);
}

// The layers of one column as the evaluations read them: flattened REAL*4
// thickness, velocities and density, and for a group of lanes (tables in
// shared memory) omega / a, omega / b, gammk of the period and the rounded
// reciprocals of the density (Love: of the rigidity) and its square.
struct Layers {
    int mmax, llw;
    const float *d, *a, *b, *rho;
    const double *xka, *xkb, *gk, *rr, *r2;
};

// e(1) of dltar4 over the largest component, or NaN where it is not to be
// trusted (models with a water layer, phases beyond 1e5).
template <bool TAB>
__device__ __forceinline__ double dltar4_near(const Layers& M, double wvno, double omega) {
    const int n = M.mmax - 1;
    if (omega < 1.0e-4) omega = 1.0e-4;   // (as dltar4 has it)
    const double w2 = wvno * wvno;
    const double io = 1.0 / omega;
    double e0, e1, e2, e3, e4;
    {
        // (quotients: ra and rb are roots of what is left of wvno next to a
        // velocity of the half-space's, 3e-7 of it with rcp_near)
        const double xka = TAB ? M.xka[n] : omega / (double)M.a[n];
        const double xkb = TAB ? M.xkb[n] : omega / (double)M.b[n];
        const double ra = sqrt((wvno + xka) * fabs(wvno - xka));
        const double rb = sqrt((wvno + xkb) * fabs(wvno - xkb));
        const double t = (double)M.b[n] * io;
        const double gk = 2.0 * t * t, gam = gk * w2, g1 = gam - 1.0;
        const double rho = (double)M.rho[n];
        e0 = rho * rho * (g1 * g1 - gam * gk * ra * rb);
        e1 = -(rho * ra);
        e2 = rho * (g1 - gk * ra * rb);
        e3 = rho * rb;
        e4 = w2 - ra * rb;
    }
#pragma unroll 1
    for (int m = n - 1; m >= 0; m--) {
        const double rho = (double)M.rho[m], d = (double)M.d[m];
        const double xka = TAB ? M.xka[m] : omega * rcp_near(M.a[m]);
        const double xkb = TAB ? M.xkb[m] : omega * rcp_near(M.b[m]);
        const double ir = TAB ? M.rr[m] : rcp_near(M.rho[m]);
        double gk;
        if (TAB) {
            gk = M.gk[m];
        } else {
            const double t = (double)M.b[m] * io;
            gk = 2.0 * t * t;
        }
        double cp, w, x, ea, cq, y, z, eb;
        wave_near<TAB>(wvno, xka, d, cp, w, x, ea);
        wave_near<TAB>(wvno, xkb, d, cq, y, z, eb);
        const double gam = gk * w2, g1 = gam - 1.0, tg = gam + g1;
        const double gmk = gam * gk, gm1 = gam * g1, g1s = g1 * g1;
        const double cpcq = cp * cq, cpy = cp * y, cpz = cp * z, cqw = cq * w, cqx = cq * x;
        const double xy = x * y, xz = x * z, wy = w * y, wz = w * z;
        const double a0 = ea * eb, a0pq = a0 - cpcq;
        const double wwy = w2 * wy;
        const double m00 = cpcq - fma(2.0 * gm1, a0pq, fma(gmk, xz, g1s * wwy));
        const double m01 = fma(w2, cpy, -cqx) * ir;
        const double m02 = -(fma(tg, a0pq, fma(gk, xz, g1 * wwy)) * ir);
        const double m03 = fma(-w2, cqw, cpz) * ir;
        const double m04 = -(fma(2.0 * w2, a0pq, fma(w2, wwy, xz)) * (ir * ir));
        const double m10 = fma(gmk, cpz, -(g1s * cqw)) * rho;
        const double m12 = fma(gk, cpz, -(g1 * cqw));
        const double m30 = fma(g1s, cpy, -(gmk * cqx)) * rho;
        const double m32 = fma(g1, cpy, -(gk * cqx));
        const double m40 = -(fma(2.0 * gmk * g1s, a0pq, fma(gmk * gmk, xz, g1s * g1s * wy))
                             * (rho * rho));
        const double m42 = -(fma(gk * g1 * tg, a0pq, fma(gmk * gk, xz, g1 * g1s * wy)) * rho);
        const double m22 = a0 + 2.0 * (cpcq - m00);
        const double te = -2.0 * w2 * e2;
        const double f0 = fma(e0, m00, fma(e1, m10, fma(te, m42, fma(e3, m30, e4 * m40))));
        const double f1 = fma(e0, m01, fma(e1, cpcq, fma(te, m32, fma(-e3, xy, e4 * m30))));
        const double f2 = fma(e0, m02, fma(e1, m12, fma(e2, m22, fma(e3, m32, e4 * m42))));
        const double f3 = fma(e0, m03, fma(-e1, wz, fma(te, m12, fma(e3, cpcq, e4 * m10))));
        const double f4 = fma(e0, m04, fma(e1, m03, fma(te, m02, fma(e3, m01, e4 * m00))));
        e0 = f0;
        e1 = f1;
        e2 = f2;
        e3 = f3;
        e4 = f4;
        if ((m & 3) == 0) {
            const double t1 = fmax(fmax(fmax(fabs(e0), fabs(e1)), fmax(fabs(e2), fabs(e3))),
                                   fabs(e4));
            if (m == 0) return M.llw == 1 ? e0 / t1 : t1 * __longlong_as_double(0x7ff8000000000000ll);
            const double s = pow2_rcp(t1);
            e0 *= s;
            e1 *= s;
            e2 *= s;
            e3 *= s;
            e4 *= s;
        }
    }
    return __longlong_as_double(0x7ff8000000000000ll);   // no layer over the half-space
}

// dltar1 (Love) likewise: e1 over the larger of |e1|, |e2|.
template <bool TAB>
__device__ __forceinline__ double dltar1_near(const Layers& M, double wvno, double omega) {
    const int n = M.mmax - 1;
    double e1, e2;
    {
        const double b = (double)M.b[n], ib = rcp_near(b), xkb = TAB ? M.xkb[n] : omega / b;
        e1 = (double)M.rho[n] * sqrt((wvno + xkb) * fabs(wvno - xkb));
        e2 = ib * ib;
    }
#pragma unroll 1
    for (int m = n - 1; m >= 0; m--) {
        const double b = (double)M.b[m], mu = (double)M.rho[m] * b * b;
        const double xkb = TAB ? M.xkb[m] : omega * rcp_near(M.b[m]);
        double co, y, z, e;
        wave_near<TAB>(wvno, xkb, (double)M.d[m], co, y, z, e);
        const double im = TAB ? M.rr[m] : rcp_near(mu);
        const double a = fma(e1, co, e2 * mu * z), c = fma(e1 * y, im, e2 * co);
        const double t1 = fmax(fabs(a), fabs(c));
        if (!(e == e) || (m == 0 && M.llw != 1)) return __longlong_as_double(0x7ff8000000000000ll);
        if (m == 0) return a / t1;
        const double s = pow2_rcp(t1);
        e1 = a * s;
        e2 = c * s;
    }
    return __longlong_as_double(0x7ff8000000000000ll);
}

constexpr double kSignSure = 1e-6;   // smallest normalised |dltar_near| whose sign is taken

// ---------------------------------------------------------------------------
// The search as a state machine: what it wants next is a sign (kEntry: of
// dltar at c1, kMarch: at the trial c2) or a value (the kX phases: at wvno).
// ---------------------------------------------------------------------------
struct Search {
    enum : int { kEntry = 0, kMarch = 1, kXEntry, kXTrial, kXLow, kXHigh, kNvFirst, kNvTopEval,
                 kNvEnd, kDone };
    // per column
    double cc, dc, cm;
    float betmx;
    int igr, kmax;
    // progress
    int ph, k, stage, status;
    float t1a, t1b;
    double cprev;                  // c(k-1) of the period before
    double ck;                     // this period's phase velocity
    // getsol: del1 belongs to cdel (its value known or only its sign)
    double omega, c1, clow, c2, cdel, del1, del2;
    int idir, guard, ifirst, sgn1, sgn0;
    bool known1;
    // nevill
    double n1, n2, nd1, nd2, c3, del3;
    int nev, nctrl, m;
    double x[11], y[11];
    double wvno;                   // the requested evaluation's wavenumber
    // the results: velocity k at out[(k - 1) * pitch]
    double* out;
    size_t pitch;

    __device__ bool wants_sign() const { return ph <= kMarch; }
    __device__ bool wants_value() const { return ph > kMarch && ph != kDone; }
};

__device__ __forceinline__ int sgn_(double x) { return signbit(x) ? -1 : 1; }

__device__ inline void search_request(Search& S, int ph, double c) {
    S.ph = ph;
    S.wvno = S.omega / c;
}
__device__ inline void search_getsol(Search& S, double t1) {   // surfdisp96.f:413
    S.omega = 2.0 * 3.141592653589793 / t1;
    S.ph = Search::kEntry;
}
// the next period's search (surfdisp96.f:121-160)
__device__ inline void search_period(Search& S, const double* t) {
    const float h = 0.005f;
    S.k++;
    if (S.k > S.kmax) {
        S.ph = Search::kDone;
        S.status = 0;
        return;
    }
    double t1 = t[S.k - 1];
    S.t1b = 0.0f;
    if (S.igr > 0) {
        S.t1a = (float)(t1 / (double)(1.0f + h));
        S.t1b = (float)(t1 / (double)(1.0f - h));
        t1 = (double)S.t1a;
    } else {
        S.t1a = (float)t1;
    }
    if (S.k == 1) {
        S.c1 = S.cc;
        S.clow = S.cc;
        S.ifirst = 1;
    } else {
        S.ifirst = 0;
        S.c1 = S.cprev - (double)1.500f * S.dc;
        S.clow = S.cm;
    }
    S.stage = 0;
    search_getsol(S, t1);
}
__device__ inline float group_velocity(const Search& S, float cc0, float ccg) {
    return (1.0f / S.t1a - 1.0f / S.t1b) / (1.0f / (S.t1a * cc0) - 1.0f / (S.t1b * ccg));
}
// getsol without a root (surfdisp96.f:463-498, :194-232)
__device__ inline void search_fail(Search& S, const double* t) {
    if (S.stage == 0) {   // the fundamental mode fails from this period on
        for (int i = S.k; i <= S.kmax; i++) S.out[(i - 1) * S.pitch] = 0.0;
        S.ph = Search::kDone;
        S.status = 1;
        return;
    }
    // the second search failed: the group velocity uses c itself
    S.out[(S.k - 1) * S.pitch] = group_velocity(S, (float)S.ck, (float)S.ck);
    S.cprev = S.ck;
    search_period(S, t);
}
// the sign of dltar at c1 is known (surfdisp96.f:417-430)
__device__ inline void search_entered(Search& S, int sg, bool known) {
    S.sgn1 = sg;
    S.known1 = known;
    S.cdel = S.c1;
    if (S.ifirst == 1) S.sgn0 = sg;
    S.idir = (S.ifirst == 1 || S.sgn0 * sg >= 0) ? +1 : -1;
    S.guard = 0;
    S.ph = Search::kMarch;
}
// the next trial velocity c2 from c1 (surfdisp96.f:431-446), false when the
// march gives up
__device__ inline bool march_trial(double& c1, int& idir, int& guard, double dc, double clow,
                                   double& c2) {
    for (;;) {
        if (guard >= 100000) return false;
        c2 = idir > 0 ? c1 + dc : c1 - dc;
        if (!(c2 <= clow)) return true;
        idir = +1;
        c1 = clow;
        guard++;
    }
}
// a trial without a sign change is accepted, false when it ends the march
__device__ inline bool march_accept(double& c1, int& guard, double c2, double cm, double cend) {
    c1 = c2;
    if (c1 < cm || c1 >= cend) return false;
    guard++;
    return true;
}
// the bracket's ends (surfdisp96.f:447-455): their values, then nevill
__device__ inline void search_refine(Search& S) {
    S.n1 = S.c1;
    S.n2 = S.c2;
    S.nd1 = S.del1;
    S.nd2 = S.del2;
    S.c3 = 0.5 * (S.n1 + S.n2);
    search_request(S, Search::kNvFirst, S.c3);
}
__device__ inline void search_bracket(Search& S, bool high_known) {
    if (!S.known1) {
        search_request(S, Search::kXLow, S.cdel);
        S.nev = high_known;
    } else if (!high_known) {
        search_request(S, Search::kXHigh, S.c2);
    } else {
        search_refine(S);
    }
}

// The requested value has arrived: the search runs on to its next request.
__device__ inline void search_value(Search& S, double del, const double* t) {
    switch (S.ph) {
        case Search::kXEntry:
            S.del1 = del;
            search_entered(S, sgn_(del), true);
            return;
        case Search::kXTrial:
            if (sgn_(del) != S.sgn1) {
                S.del2 = del;
                search_bracket(S, true);
                return;
            }
            S.del1 = del;
            S.known1 = true;
            S.cdel = S.c2;
            if (!march_accept(S.c1, S.guard, S.c2, S.cm, (double)S.betmx + S.dc)) search_fail(S, t);
            else S.ph = Search::kMarch;
            return;
        case Search::kXLow:
            S.del1 = del;
            S.known1 = true;
            search_bracket(S, S.nev != 0);
            return;
        case Search::kXHigh:
            S.del2 = del;
            search_refine(S);
            return;
        case Search::kNvFirst:
            S.nev = 1;
            S.nctrl = 1;
            S.m = 1;
            break;
        default:
            break;
    }
    S.del3 = del;
    bool done = false;
    if (S.ph != Search::kNvTopEval) {   // surfdisp96.f:593-600
        S.nctrl = S.nctrl + 1;
        if (S.nctrl >= 100) {
            done = true;
        } else if (S.c3 < fmin(S.n1, S.n2) || S.c3 > fmax(S.n1, S.n2)) {
            S.nev = 0;
            S.c3 = 0.5 * (S.n1 + S.n2);
            search_request(S, Search::kNvTopEval, S.c3);
            return;
        }
    }
    if (!done) {   // surfdisp96.f:601-696
        const double s13 = S.nd1 - S.del3;
        const double s32 = S.del3 - S.nd2;
        if (dsign1(S.del3) * dsign1(S.nd1) < 0.0) {
            S.n2 = S.c3;
            S.nd2 = S.del3;
        } else {
            S.n1 = S.c3;
            S.nd1 = S.del3;
        }
        if (fabs(S.n1 - S.n2) <= 1.e-6 * S.n1) {
            done = true;
        } else {
            if (dsign1(s13) != dsign1(s32)) S.nev = 0;
            const double p01 = (double)0.01f;
            const double ss1 = fabs(S.nd1);
            const double s1 = p01 * ss1;
            const double ss2 = fabs(S.nd2);
            const double s2 = p01 * ss2;
            bool halve = s1 > ss2 || s2 > ss1 || S.nev == 0;
            if (!halve) {
                int m = S.m;
                if (S.nev == 2) {
                    S.x[m] = S.c3;
                    S.y[m] = S.del3;
                } else {
                    S.x[0] = S.n1;
                    S.y[0] = S.nd1;
                    S.x[1] = S.n2;
                    S.y[1] = S.nd2;
                    m = 1;
                }
                for (int kk = 1; kk <= m; kk++) {
                    const int j = m - kk + 1;
                    const double denom = S.y[m] - S.y[j - 1];
                    if (fabs(denom) < 1.0e-10 * fabs(S.y[m])) {
                        halve = true;
                        break;
                    }
                    S.x[j - 1] = (-(S.y[j - 1] * S.x[j]) + S.y[m] * S.x[j - 1]) / denom;
                }
                if (!halve) {
                    S.c3 = S.x[0];
                    S.nev = 2;
                    m = m + 1;
                    if (m > 10) m = 10;
                    S.m = m;
                }
            }
            if (halve) {
                S.c3 = 0.5 * (S.n1 + S.n2);
                S.nev = 1;
                S.m = 1;
            }
            search_request(S, Search::kNvEnd, S.c3);
            return;
        }
    }
    // getsol after nevill (surfdisp96.f:455-459)
    S.c1 = S.c3;
    if (S.c1 > (double)S.betmx) {
        search_fail(S, t);
        return;
    }
    if (S.stage == 0) {
        S.ck = S.c1;
        if (S.igr > 0) {   // the group velocity's second search (:181-192)
            S.stage = 1;
            S.ifirst = 0;
            S.clow = 0.0 + 1.0e-2 * S.dc;   // cb(k) is still 0 in mode 1
            S.c1 = S.c1 - (double)1.500f * S.dc;
            search_getsol(S, (double)S.t1b);
            return;
        }
        S.out[(S.k - 1) * S.pitch] = (float)S.ck;
    } else {
        S.out[(S.k - 1) * S.pitch] = group_velocity(S, (float)S.ck, (float)S.c1);
    }
    S.cprev = S.ck;
    search_period(S, t);
}

// A sign evaluation by one lane: v = dltar_near at c1 (entry) or c2.
__device__ inline void search_sign(Search& S, double v, const double* t) {
    const bool sure = fabs(v) > kSignSure;
    if (S.ph == Search::kEntry) {
        if (!sure) search_request(S, Search::kXEntry, S.c1);
        else search_entered(S, sgn_(v), false);
    } else if (!sure) {
        search_request(S, Search::kXTrial, S.c2);
    } else if (sgn_(v) != S.sgn1) {
        search_bracket(S, false);
    } else {
        S.known1 = false;
        S.cdel = S.c2;
        if (!march_accept(S.c1, S.guard, S.c2, S.cm, (double)S.betmx + S.dc)) search_fail(S, t);
    }
}

}  // namespace sk
}  // namespace sa
