// SurfGrid::fwdsurf (src/surf_grid.cpp:194-245): surfdisp96 of every surface
// column, by the searches of surfker_search.cuh.  Compiled with -fmad=false
// (see surfker_dev.cuh).
#ifndef SK_ATTR_DLTAR4
#define SK_ATTR_DLTAR4 __noinline__
#endif
#include "surfker_search.cuh"

namespace sa {

using sk::LayerConst;
using sk::Layers;
using sk::Search;

namespace {

__device__ __forceinline__ void search_init(Search& S, int igr, int nper, double* out,
                                            size_t pitch) {
    S.cm = S.cc;
    S.igr = igr;
    S.kmax = nper;
    S.k = 0;
    S.status = 0;
    S.cprev = 0.0;
    S.ck = 0.0;
    S.sgn0 = 1;
    S.known1 = false;
    S.out = out;
    S.pitch = pitch;
}

// ---------------------------------------------------------------------------
// One column per thread (grids of more than about 35,000 columns).  The
// lanes of a warp alternate between two loops: signs until every lane has
// its bracket, then values until every lane has its root.  The marches and
// refinements of neighbouring columns are nearly equally long, so a warp
// runs two evaluations' code one after the other instead of side by side
// (301x301x40, 20 periods: 61 ms; switching as soon as half the lanes wait
// for the other kind 111 ms, four lanes 75 ms).  Bound by FP64 issue: 13.8
// values and 18.9 signs a period where every evaluation was a value before
// (30.7: 113 -> 61 ms; Love 42 -> 24 ms; 601x601x50 with 10 periods 333 ->
// 160 ms).  10 blocks of 64 threads an SM (96 registers): 8 blocks 73
// ms, 12 61 ms, 16 65 ms.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(64, 10)
surfdisp_columns_kernel(int nx, int ny, int nz, const double* __restrict__ vs3d, int nper,
                        const double* __restrict__ periods, int iflsph, int iwave, int igr,
                        const LayerConst* __restrict__ Lp, double* svel, int* status) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = col < nx * ny;
    const LayerConst& L = *Lp;
    periods += (size_t)blockIdx.y * nper;   // blockIdx.y: the run
    svel += (size_t)blockIdx.y * nx * ny * nper;
    if (status) status += (size_t)blockIdx.y * nx * ny;
    const size_t pos = live ? (size_t)(col / ny) + (size_t)nx * (col % ny) : 0;
    const int ifunc = iwave == 1 ? 1 : 2;
    sk::SDModel M;
    Search S;
    S.ph = Search::kDone;
    if (live) {
        sk::sd_setup(L, vs3d + (size_t)col * nz, nz, iflsph, iwave, M, S.betmx, S.cc, S.dc);
        search_init(S, igr, nper, svel + pos, (size_t)nx * ny);
        sk::search_period(S, periods);
    }
    const Layers Y{M.mmax, M.llw, M.d, M.a, M.b, M.rho, nullptr, nullptr, nullptr, nullptr,
                   nullptr};
    bool signs = true;
    for (;;) {
        const unsigned ms = __ballot_sync(0xffffffffu, S.wants_sign());
        const unsigned mv = __ballot_sync(0xffffffffu, S.wants_value());
        if (!(ms | mv)) break;
        if (!(signs ? ms : mv)) signs = !signs;
        if (signs) {
            if (S.wants_sign()) {
                if (S.ph == Search::kMarch &&
                    !sk::march_trial(S.c1, S.idir, S.guard, S.dc, S.clow, S.c2)) {
                    sk::search_fail(S, periods);
                } else {
                    const double c = S.ph == Search::kEntry ? S.c1 : S.c2;
                    const double w = S.omega / c;
                    const double v = ifunc == 1 ? sk::dltar1_near<false>(Y, w, S.omega)
                                                : sk::dltar4_near<false>(Y, w, S.omega);
                    sk::search_sign(S, v, periods);
                }
            }
        } else if (S.wants_value()) {
            sk::search_value(S, sk::dltar(M, S.wvno, S.omega, ifunc), periods);
        }
    }
    if (live && status) status[pos] = S.status;
}

// ---------------------------------------------------------------------------
// One column per group of G lanes: G trial velocities of a march at a time,
// a lane each; a value by all lanes together, the layer matrices G at a time
// (a layer per lane) into shared memory, then the row-vector product down
// the layers with a component per lane.  The layers, the period's omega / a,
// omega / b and gammk and the densities' reciprocals lie in shared memory.
// Bound by the latency of the row-vector products (five products and sums,
// three exchanges, a division a layer).  41x41x30 with 10 periods (1681
// columns) 39.4 ms with a thread per column -> 2.4 ms with 32 lanes.
// ---------------------------------------------------------------------------
constexpr int kGroupThreads = 128;
constexpr int kMatPitch = 15;   // distinct entries of a compound layer matrix

__host__ __device__ constexpr size_t group_bytes(int mmax, int G) {
    return ((size_t)mmax * 56 + 15) / 16 * 16 + (size_t)(G * kMatPitch + 1) * 8;
}

// The compound layer matrix's distinct entries in the order ca00 ca01 ca02
// ca03 ca04 ca10 ca11 ca12 ca13 ca30 ca31 ca32 ca40 ca42 ca22, and the places
// of ca[0..4][i] (row 2: times -2 wvno^2 unless i = 2) for each component i.
__device__ __forceinline__ unsigned mat_places(int i) {
    switch (i) {
        case 0: return 0u | 5u << 4 | 13u << 8 | 9u << 12 | 12u << 16;
        case 1: return 1u | 6u << 4 | 11u << 8 | 10u << 12 | 9u << 16;
        case 2: return 2u | 7u << 4 | 14u << 8 | 11u << 12 | 13u << 16;
        case 3: return 3u | 8u << 4 | 7u << 8 | 6u << 12 | 5u << 16;
        default: return 4u | 3u << 4 | 2u << 8 | 1u << 12 | 0u << 16;
    }
}

// dltar4 (surfdisp96.f:801-901) by a group; every lane returns the value.
// All lanes of the warp call it; groups with `on` false take part in the
// exchanges only.
template <int G>
__device__ __forceinline__ double group_dltar4(const Layers& M, double* mat, int gl, bool on,
                                               double wvno) {
    const int n = M.mmax - 1;
    const double wvno2 = wvno * wvno;
    double e0, e1, e2, e3, e4;
    {
        const double xka = M.xka[n], xkb = M.xkb[n], gammk = M.gk[n];
        const double ra = sqrt((wvno + xka) * fabs(wvno - xka));
        const double rb = sqrt((wvno + xkb) * fabs(wvno - xkb));
        const double gam = gammk * wvno2;
        const double gamm1 = gam - 1.0;
        const double rho1 = (double)M.rho[n];
        e0 = rho1 * rho1 * (gamm1 * gamm1 - gam * gammk * ra * rb);
        e1 = -(rho1 * ra);
        e2 = rho1 * (gamm1 - gammk * ra * rb);
        e3 = rho1 * rb;
        e4 = wvno2 - ra * rb;
    }
    const int comp = min(gl & 7, 4);
    const unsigned at = mat_places(comp);
    const double f2 = comp == 2 ? 1.0 : -2.0 * wvno2;
    const int base = (threadIdx.x & 31) & ~7;
    const int last = on ? M.llw - 1 : n;   // the topmost solid layer
    for (int top = n - 1; top >= 0; top -= G) {
        const int m = top - gl;
        if (m >= last) {
            const double xka = M.xka[m], xkb = M.xkb[m], gammk = M.gk[m];
            const double gam = gammk * wvno2;
            const double ra = sqrt((wvno + xka) * fabs(wvno - xka));
            const double rb = sqrt((wvno + xkb) * fabs(wvno - xkb));
            const double dpth = (double)M.d[m], rho1 = (double)M.rho[m];
            const sk::VarOut v = sk::var(ra * dpth, rb * dpth, ra, rb, wvno, xka, xkb, dpth);
            double ca[5][5];
            sk::dnka_matrix(ca, wvno2, gam, gammk, rho1, v, M.rr[m], M.r2[m]);
            double* q = mat + gl * kMatPitch;
            q[0] = ca[0][0];
            q[1] = ca[0][1];
            q[2] = ca[0][2];
            q[3] = ca[0][3];
            q[4] = ca[0][4];
            q[5] = ca[1][0];
            q[6] = ca[1][1];
            q[7] = ca[1][2];
            q[8] = ca[1][3];
            q[9] = ca[3][0];
            q[10] = ca[3][1];
            q[11] = ca[3][2];
            q[12] = ca[4][0];
            q[13] = ca[4][2];
            q[14] = ca[2][2];
        }
        __syncwarp();
        const int cnt = min(G, top + 1);
        for (int l = 0; l < cnt; l++) {
            const double* q = mat + l * kMatPitch;
            double cr = 0.0;
            cr = cr + e0 * q[at & 15u];
            cr = cr + e1 * q[(at >> 4) & 15u];
            cr = cr + e2 * (f2 * q[(at >> 8) & 15u]);
            cr = cr + e3 * q[(at >> 12) & 15u];
            cr = cr + e4 * q[(at >> 16) & 15u];
            double t1 = fabs(cr);
            t1 = fmax(t1, __shfl_xor_sync(0xffffffffu, t1, 1));
            t1 = fmax(t1, __shfl_xor_sync(0xffffffffu, t1, 2));
            t1 = fmax(t1, __shfl_xor_sync(0xffffffffu, t1, 4));
            if (t1 < 1.e-40) t1 = 1.0;
            const double rh = 1.0 / t1;
            cr = quot(cr, t1, rh, recip_lo(t1, rh));
            const double g0 = __shfl_sync(0xffffffffu, cr, base);
            const double g1 = __shfl_sync(0xffffffffu, cr, base + 1);
            const double g2 = __shfl_sync(0xffffffffu, cr, base + 2);
            const double g3 = __shfl_sync(0xffffffffu, cr, base + 3);
            const double g4 = __shfl_sync(0xffffffffu, cr, base + 4);
            if (top - l >= last) {
                e0 = g0;
                e1 = g1;
                e2 = g2;
                e3 = g3;
                e4 = g4;
            }
        }
        __syncwarp();
    }
    if (on && M.llw != 1) {
        const double xka = M.xka[0];
        const double ra = sqrt((wvno + xka) * fabs(wvno - xka));
        const double dpth = (double)M.d[0], rho1 = (double)M.rho[0];
        const double znul = 1.0e-05;
        const sk::VarOut v = sk::var(ra * dpth, znul, ra, znul, wvno, xka, znul, dpth);
        return v.cosp * e0 + -(rho1 * v.w) * e1;
    }
    return e0;
}

// dltar1 (surfdisp96.f:737-797) likewise: cos q, sin q / rb and rb sin q of
// G layers at a time, the two-vector's recursion by every lane.
template <int G>
__device__ __forceinline__ double group_dltar1(const Layers& M, double* mat, int gl, bool on,
                                               double wvno) {
    const int n = M.mmax - 1;
    double e1, e2;
    {
        const double xkb = M.xkb[n], beta1 = (double)M.b[n];
        e1 = (double)M.rho[n] * sqrt((wvno + xkb) * fabs(wvno - xkb));
        e2 = 1.0 / (beta1 * beta1);
    }
    const int last = on ? M.llw - 1 : n;
    for (int top = n - 1; top >= 0; top -= G) {
        const int m = top - gl;
        if (m >= last) {
            const double xkb = M.xkb[m], d = (double)M.d[m];
            const double rb = sqrt((wvno + xkb) * fabs(wvno - xkb));
            const double q = d * rb;
            double sinq, y, z, cosq;
            if (wvno < xkb) {
                sk::sk_sincos(q, &sinq, &cosq);
                y = sinq / rb;
                z = -(rb * sinq);
            } else if (wvno == xkb) {
                cosq = 1.0;
                y = d;
                z = 0.0;
            } else {
                double fac = 0.0;
                if (q < 16) fac = sk::sk_exp(-2.0 * q);
                cosq = (1.0 + fac) * 0.5;
                sinq = (1.0 - fac) * 0.5;
                y = sinq / rb;
                z = rb * sinq;
            }
            double* o = mat + gl * kMatPitch;
            o[0] = cosq;
            o[1] = y;
            o[2] = z;
        }
        __syncwarp();
        const int cnt = min(G, top + 1);
        for (int l = 0; l < cnt; l++) {
            const int ml = top - l;
            if (ml < last) break;
            const double* o = mat + l * kMatPitch;
            const double cosq = o[0], xmu = M.r2[ml], rh = M.rr[ml];
            const double e10 = e1 * cosq + e2 * xmu * o[2];
            const double e20 = quot(e1 * o[1], xmu, rh, recip_lo(xmu, rh)) + e2 * cosq;
            double xnor = fabs(e10);
            const double ynor = fabs(e20);
            if (ynor > xnor) xnor = ynor;
            if (xnor < 1.e-40) xnor = 1.0;
            e1 = e10 / xnor;
            e2 = e20 / xnor;
        }
        __syncwarp();
    }
    return e1;
}

template <int G>
__global__ void __launch_bounds__(kGroupThreads, 4)
surfdisp_groups_kernel(int nx, int ny, int nz, const double* __restrict__ vs3d, int nper,
                       const double* __restrict__ periods, int iflsph, int iwave, int igr,
                       const LayerConst* __restrict__ Lp, double* svel, int* status) {
    extern __shared__ double4 smem4[];
    const LayerConst& L = *Lp;
    const int mmax = L.mmax;
    const int gl = threadIdx.x % G, grp = threadIdx.x / G;
    const int lane = threadIdx.x & 31, gbase = lane & ~(G - 1);
    const unsigned gmask = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    const int col = blockIdx.x * (kGroupThreads / G) + grp;
    const bool live = col < nx * ny;
    periods += (size_t)blockIdx.y * nper;   // blockIdx.y: the run
    svel += (size_t)blockIdx.y * nx * ny * nper;
    if (status) status += (size_t)blockIdx.y * nx * ny;
    const size_t pos = live ? (size_t)(col / ny) + (size_t)nx * (col % ny) : 0;
    const bool love = iwave == 1;
    double* dp = reinterpret_cast<double*>(reinterpret_cast<char*>(smem4) +
                                           grp * group_bytes(mmax, G));
    double *xka = dp, *xkb = xka + mmax, *gk = xkb + mmax, *rr = gk + mmax, *r2 = rr + mmax;
    float* fd = reinterpret_cast<float*>(r2 + mmax);
    float *fa = fd + mmax, *fb = fa + mmax, *fr = fb + mmax;
    double* mat = dp + ((size_t)mmax * 56 + 15) / 16 * 2;
    // the column's layers, the bracket step and the first velocity (sd_setup)
    Search S;
    S.ph = Search::kDone;
    Layers Y{mmax, 1, fd, fa, fb, fr, xka, xkb, gk, rr, r2};
    const double* v1 = vs3d + (size_t)(live ? col : 0) * nz;
    float vmin = 1e30f;
    for (int i = gl; i < mmax; i += G) {
        float vp, vs, rho;
        sk::layer_model(v1[min(i, nz - 1)], vp, vs, rho);
        vmin = fminf(vmin, vs);
        if (i == 0) vmin = vs;
        sk::flatten_layer(L, i, iflsph, love, vp, vs, rho, fd[i], fa[i], fb[i], fr[i]);
        const double r = (double)fr[i], b = (double)fb[i];
        if (love) {
            const double mu = r * b * b;
            r2[i] = mu;
            rr[i] = 1.0 / mu;
        } else {
            rr[i] = 1.0 / r;
            r2[i] = 1.0 / (r * r);
        }
    }
    for (int o = G / 2; o > 0; o >>= 1) vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
    __syncwarp();
    if (live) {
        Y.llw = (float)v1[0] <= 0.0f ? 2 : 1;
        sk::first_velocity(mmax, vmin, fa, fb, S.betmx, S.cc, S.dc);
        search_init(S, igr, nper, svel + pos, (size_t)nx * ny);
        sk::search_period(S, periods);
    }
    bool signs = true;
    for (;;) {
        const bool ws = S.wants_sign();
        const unsigned ms = __ballot_sync(0xffffffffu, ws);
        const unsigned mv = __ballot_sync(0xffffffffu, S.wants_value());
        if (!(ms | mv)) break;
        if (!(signs ? ms : mv)) signs = !signs;
        if (signs) {
            if (ws && S.ph == Search::kEntry) {   // the period's tables
                const double omega = S.omega < 1.0e-4 ? 1.0e-4 : S.omega;
                for (int i = gl; i < mmax; i += G) {
                    const double t = (double)fb[i] / omega;
                    xka[i] = omega / (double)fa[i];
                    xkb[i] = (love ? S.omega : omega) / (double)fb[i];
                    gk[i] = 2.0 * t * t;
                }
            }
            __syncwarp();
            // the trial of this lane: the march's next G steps as they follow
            // while no sign changes, or at a search's entry c1 itself and the
            // G - 1 steps after it (upwards, the usual direction)
            const bool entry = S.ph == Search::kEntry;
            double c1 = S.c1, c2 = S.c1, cdel = entry ? S.c1 : S.cdel;
            int idir = entry ? +1 : S.idir, guard = entry ? 0 : S.guard;
            const double cend = (double)S.betmx + S.dc;
            int code = 0;   // the sign, 0 not sure, 2 the march ends before
            if (ws) {
                bool ok = true;
                const int steps = gl + (entry ? 0 : 1);
                for (int s = 0; s < steps && ok; s++) {
                    if (s > 0) {
                        cdel = c2;
                        ok = sk::march_accept(c1, guard, c2, S.cm, cend);
                    }
                    if (ok) ok = sk::march_trial(c1, idir, guard, S.dc, S.clow, c2);
                }
                code = 2;
                if (ok) {
                    const double w = S.omega / c2;
                    const double v = love ? sk::dltar1_near<true>(Y, w, S.omega)
                                          : sk::dltar4_near<true>(Y, w, S.omega);
                    code = fabs(v) > sk::kSignSure ? sk::sgn_(v) : 0;
                }
            }
            const int code0 = __shfl_sync(0xffffffffu, code, gbase);
            int first = 0;
            bool go = ws;
            if (ws && entry) {
                first = 1;
                if (code0 == 0) sk::search_request(S, Search::kXEntry, S.c1);
                else sk::search_entered(S, code0, false);
                go = code0 != 0 && S.idir > 0;
            }
            const unsigned diff = __ballot_sync(0xffffffffu, code != S.sgn1);
            unsigned d = (diff >> gbase) & gmask;
            if (first) d &= ~1u;
            const int f = d ? __ffs(d) - 1 : G;
            const int src = gbase + min(f, G - 1);
            const double sc1 = __shfl_sync(0xffffffffu, c1, src);
            const double sc2 = __shfl_sync(0xffffffffu, c2, src);
            const double scd = __shfl_sync(0xffffffffu, cdel, src);
            const int sdir = __shfl_sync(0xffffffffu, idir, src);
            const int sgd = __shfl_sync(0xffffffffu, guard, src);
            const int scode = __shfl_sync(0xffffffffu, code, src);
            if (go) {
                if (f > first) S.known1 = false;   // steps were accepted
                S.c1 = sc1;
                S.c2 = sc2;
                S.cdel = scd;
                S.idir = sdir;
                S.guard = sgd;
                if (f == G) {
                    S.known1 = false;
                    S.cdel = sc2;
                    if (!sk::march_accept(S.c1, S.guard, sc2, S.cm, cend))
                        sk::search_fail(S, periods);
                } else if (scode == 2) {
                    sk::search_fail(S, periods);
                } else if (scode == 0) {
                    sk::search_request(S, Search::kXTrial, S.c2);
                } else {
                    sk::search_bracket(S, false);
                }
            }
        } else {
            const bool wv = S.wants_value();
            const double del = love ? group_dltar1<G>(Y, mat, gl, wv, S.wvno)
                                    : group_dltar4<G>(Y, mat, gl, wv, S.wvno);
            if (wv) sk::search_value(S, del, periods);
        }
        __syncwarp();
    }
    if (live && gl == 0 && status) status[pos] = S.status;
}

template <int G>
cudaError_t launch_groups(int nx, int ny, int nz, const double* vs3d, int nper, int runs,
                          const double* periods, int iflsph, int iwave, int igr,
                          const LayerConst* Lp, double* svel, int* status, cudaStream_t st) {
    constexpr int per = kGroupThreads / G;
    const int n = nx * ny;
    const size_t bytes = per * group_bytes(nz + 1, G);
    // (the limit belongs to the device and threads launch at the same time: the
    // largest that any call needs, not this one's)
    constexpr int most = (int)(per * group_bytes(sk::MMAX, G));
    cudaError_t e = cudaFuncSetAttribute(surfdisp_groups_kernel<G>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
    surfdisp_groups_kernel<G><<<dim3((n + per - 1) / per, runs), kGroupThreads, bytes, st>>>(
        nx, ny, nz, vs3d, nper, periods, iflsph, iwave, igr, Lp, svel, status);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_surfdisp_columns(int nx, int ny, int nz, const double* vs3d, int nper,
                                    const double* periods, int iflsph, int iwave, int igr,
                                    const void* layer_const, double* svel, int* status,
                                    cudaStream_t st, int runs) {
    const int n = nx * ny;
    const long long all = (long long)n * runs;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const LayerConst* Lp = reinterpret_cast<const LayerConst*>(layer_const);
    // Lanes per column by the number of columns.  A thread per column leaves
    // most of the GPU idle below some 240 columns an SM, each column a serial
    // chain of about 30 evaluations a period; a group of lanes shortens that
    // chain at the price of idle lanes in the row-vector products, so the
    // widest group that still fits one wave (4 blocks of 128 threads an SM)
    // is the fastest, and the 8-lane group stays ahead of a thread per column
    // for several waves.  Rayleigh phase velocities, ms with 32 / 16 / 8 / 1
    // lanes: 1681 columns x 10 periods 2.37 / 2.50 / 3.15 / 15.8; 3233 x 8
    // 3.80 / 2.30 / 2.69 / 12.4; 8787 x 12 14.6 / 9.3 / 6.6 / 19.0; 20,687 x
    // 12 36 / 23 / 17.8 / 26.1; 40,401 x 15 85 / 52 / 36.7 / 34.8.
    // Several runs (the three period lists of the group kernels) count as
    // that many columns: in one launch they fill the SMs that one run leaves
    // idle (group kernels with their runs, Rayleigh / Love: 41x41x30 with 10
    // periods 10.0 -> 7.5 / 5.2 -> 3.1 ms, 101x87x33 with 12 31.1 -> 30.4 /
    // 12.3 -> 11.9, 151x151x30 with 8 50.5 -> 38.5 / 20.5 -> 12.9).
    auto groups = all <= 16 * nsm    ? launch_groups<32>
                  : all <= 32 * nsm  ? launch_groups<16>
                  : all <= 240 * nsm ? launch_groups<8>
                                     : nullptr;
    if (groups)
        return groups(nx, ny, nz, vs3d, nper, runs, periods, iflsph, iwave, igr, Lp, svel, status,
                      st);
    surfdisp_columns_kernel<<<dim3((n + 63) / 64, runs), 64, 0, st>>>(
        nx, ny, nz, vs3d, nper, periods, iflsph, iwave, igr, Lp, svel, status);
    return cudaGetLastError();
}

}  // namespace sa
