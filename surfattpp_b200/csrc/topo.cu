// Media matrices from topography (SurfGrid::build_media_matrix_with_topo,
// reference src/surf_grid.cpp:80-166) and the kernel-depth correction
// (SurfGrid::correct_depth_with_topo, :307-354), on device.
//   gauss_rows_kernel  gaussian_smooth_geo_2 (include/utils.h:505-571) on an
//                      evenly spaced longitude grid: a block per row and
//                      period, the haversine-distance Gaussian weights of the
//                      row once per (latitude, longitude distance) in shared
//                      memory for all its cells.
//   gauss_geo_kernel   the same on any grid: one thread per output cell, a
//                      weight per window point; the window's latitude terms
//                      are shared by the block.
//   media_kernel       gradient_2_geo (:593-649), dip angle (src/topo.cpp:97-114)
//                      and m11 = a, m12 = -c, m22 = b per cell.
//   depth_topo_kernel  per (column, period): depth nodes stretched by
//                      1/cos(dip), clamped, linear interpolation (utils.h:451-485).
//   grid_kernel        interp2d onto the model grid (Topography::grid).
// Compiled with -fmad=false; sin/cos/atan/exp are CUDA's (ulp-level
// differences from the C library), so parity is to a stated tolerance.
#include <algorithm>

#include "event_common.cuh"
#include "launch.h"

namespace sa {

namespace {
constexpr double PI_T = 3.14159265358979323846264338327950288;
constexpr double DEG2RAD_T = PI_T / 180.0;
constexpr double RAD2DEG_T = 180.0 / PI_T;
constexpr double R_EARTH_T = 6371.0;

// Squared great-circle distance in degrees^2 from a = sin^2(d/2):
// (2 atan sqrt(a / (1 - a)))^2 = (2 asin sqrt a)^2, by its series
// 4 (a + a^2/3 + 8 a^3/45 + ...) where the next term is below 2^-56 of it.
__device__ __forceinline__ double dist2_deg(double a) {
    constexpr double k = 4.0 * RAD2DEG_T * RAD2DEG_T;
    if (a < 1e-3) {
        double p = fma(a, 128.0 / 2079.0, 128.0 / 1575.0);
        p = fma(a, p, 4.0 / 35.0);
        p = fma(a, p, 8.0 / 45.0);
        p = fma(a, p, 1.0 / 3.0);
        return k * fma(a * a, p, a);
    }
    a = fmin(a, 1.0);
    const double t = 2.0 * RAD2DEG_T * atan(sqrt(a / (1.0 - a)));
    return t * t;
}

// The smoothing of all periods on an evenly spaced longitude grid: block (row
// j, period ip).  The weight of a window point depends on the row, the
// point's latitude and the longitude distance, which for cell i and point m
// is (m - i) h up to the rounding of the grid values: with off[m] = lon[m] -
// lon[0] - m h and W' the weight's derivative, w = W + W' (off[m] - off[i]).
// The host checks that off is below 1e-9 of sigma, so that what this leaves
// out is below rounding.  The window's sum is then sum W z + sum W' off z -
// off[i] sum W' z, three products a point.
// The block fills W, W' and the rows z, off z of `rows` latitudes into shared
// memory; four groups of 64 threads take a latitude each, a thread four
// neighbouring cells, whose points slide through its registers, so that a
// point costs a quarter of a weight's load and half a value's.  Rows lie in
// quarters (m mod 4 first), so that the lanes' points are consecutive words.
// Bound by FP64 issue (six cycles a point and scheduler, 7.5 G points):
// 201x201, 15 periods, 113 ms with a weight (sine, root, quotient, arc
// tangent, exponential) per point and cell, 9.5 ms with shared weights and a
// cell a thread, 4.5 ms so.
constexpr int kGaussThreads = 256;
constexpr int kGaussCells = 256;   // cells of a row at a time
constexpr int kGaussShared = 200 * 1024;   // bytes of a block at most
__host__ __device__ constexpr int gauss_pitch(int hx) { return (hx + 3) / 4 * 4 + 4; }
__host__ __device__ constexpr int gauss_quarter(int nx) { return (nx + 3) / 4; }

__global__ void __launch_bounds__(kGaussThreads)
gauss_rows_kernel(int nx, int ny, const double* __restrict__ data, const double* __restrict__ lats,
                  const double* __restrict__ off, double h, const double* __restrict__ sigmas,
                  int rows, int most, double* __restrict__ out) {
    extern __shared__ double2 sh2[];
    const int j = blockIdx.x, ip = gridDim.y - 1 - blockIdx.y;   // wide windows first
    const double sigma = sigmas[ip];
    const double sigma3 = 3.0 * sigma;
    const double dy = lats[1] - lats[0];
    const int hx = min(static_cast<int>(sigma3 / h), nx - 1);
    const double cos_lat0 = cos(lats[j] * DEG2RAD_T);
    const int hy = static_cast<int>(sigma3 / cos_lat0 / dy);
    const int n1 = max(0, j - hy), n2 = min(ny - 1, j + hy);
    const double c = -1.0 / (2.0 * (sigma * sigma));
    const int tid = threadIdx.x, grp = tid >> 6, l = tid & 63;
    const int pitch = gauss_pitch(hx), P = gauss_quarter(nx);
    double2* tab = sh2;                        // [rows][pitch]: W, W' at |d|
    double2* lonf = tab + (size_t)rows * most;     // [pitch]: sin^2, sin cos of d h / 2
    double2* sums = lonf + most;                   // [pitch]: W, W' over all latitudes
    double2* zz = sums + most;                     // [rows][4 P]: z, off z
    double* part = reinterpret_cast<double*>(zz + (size_t)rows * 4 * P);   // [4][kGaussCells]
    for (int d = tid; d < pitch; d += kGaussThreads) {
        double s, co;
        sincos(d * h * (DEG2RAD_T * 0.5), &s, &co);
        lonf[d] = make_double2(s * s, s * co);
        sums[d] = make_double2(0.0, 0.0);
    }
    for (int i0 = 0; i0 < nx; i0 += kGaussCells) {
        const int i = i0 + 4 * l;   // this thread's first cell
        const int iw = i0 + 4 * (l & ~31);   // its warp's
        double b0[4] = {}, b1[4] = {}, b2[4] = {};
        for (int q0 = n1; q0 <= n2; q0 += rows) {
            const int nq = min(rows, n2 - q0 + 1);
            __syncthreads();
            for (int q = grp; q < nq; q += 4) {
                const double lat1 = lats[q0 + q];
                const double s = sin((lat1 - lats[j]) * (DEG2RAD_T * 0.5));
                const double cc = cos_lat0 * cos(lat1 * DEG2RAD_T);
                for (int d = l; d < pitch; d += 64) {
                    const double2 f = lonf[d];
                    const double a = fma(cc, f.x, s * s);
                    const double w = d <= hx ? exp(c * dist2_deg(a)) : 0.0;
                    // dw/d(lon): the distance's slope to first order, enough
                    // beside off
                    const double k = 4.0 * RAD2DEG_T * RAD2DEG_T * fma(a, 2.0 / 3.0, 1.0);
                    tab[q * pitch + d] = make_double2(w, w * c * k * cc * f.y * DEG2RAD_T);
                }
                const double* z = data + (size_t)nx * (q0 + q);
                for (int m = l; m < 4 * P; m += 64)
                    zz[q * 4 * P + (m & 3) * P + (m >> 2)] =
                        m < nx ? make_double2(z[m], z[m] * off[m]) : make_double2(0.0, 0.0);
            }
            __syncthreads();
            if (i0 == 0)   // (the weights' own sums, by all threads)
                for (int d = tid; d < pitch; d += kGaussThreads) {
                    double2 t = sums[d];
                    for (int q = 0; q < nq; q++) {
                        t.x += tab[q * pitch + d].x;
                        t.y += tab[q * pitch + d].y;
                    }
                    sums[d] = t;
                }
            if (iw < nx) {
                // d in fours: no point of the warp's cells lies outside
                const int d0 = max(-((hx + 3) / 4 * 4), -((iw + 127) / 4 * 4 + 4));
                const int d1 = min(hx, nx - 1 - iw);
                for (int q = grp; q < nq; q += 4) {
                    const double2* t = tab + q * pitch;
                    const double2* zr = zz + (size_t)q * 4 * P;
                    // points i + d + u, u = 0..6: 0..2 from the step before
                    double z[7], o[7];
                    int K = (i + d0) >> 2;   // (i and d are multiples of 4)
                    auto take = [&](int u, int quarter, int k) {
                        double2 t = make_double2(0.0, 0.0);
                        if ((unsigned)k < (unsigned)P) t = zr[quarter * P + k];
                        z[u] = t.x;
                        o[u] = t.y;
                    };
#pragma unroll
                    for (int u = 0; u < 3; u++) take(u, u, K);
                    for (int d = d0; d <= d1; d += 4, K++) {
                        take(3, 3, K);
#pragma unroll
                        for (int u = 4; u < 7; u++) take(u, u - 4, K + 1);
#pragma unroll
                        for (int v = 0; v < 4; v++) {
                            const double2 w = t[d < 0 ? -d - v : d + v];
                            const double wd = d < 0 ? -w.y : w.y;
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                b0[u] = fma(w.x, z[v + u], b0[u]);
                                b1[u] = fma(wd, o[v + u], b1[u]);
                                b2[u] = fma(wd, z[v + u], b2[u]);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 3; u++) {
                            z[u] = z[u + 4];
                            o[u] = o[u + 4];
                        }
                    }
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const double oi = i + u < nx ? off[i + u] : 0.0;
            part[grp * kGaussCells + 4 * l + u] = b0[u] + (b1[u] - oi * b2[u]);
        }
        __syncthreads();
        const int k = i0 + tid;
        if (k < nx) {
            double sw = 0.0;
            const double oi = off[k];
            for (int m = max(0, k - hx); m <= min(nx - 1, k + hx); m++) {
                const double2 t = sums[abs(m - k)];
                sw += fma(m < k ? oi - off[m] : off[m] - oi, t.y, t.x);
            }
            const double swd = (part[tid] + part[kGaussCells + tid]) +
                               (part[2 * kGaussCells + tid] + part[3 * kGaussCells + tid]);
            out[((size_t)ip * ny + j) * nx + k] = swd / sw;
        }
    }
}

__global__ void gauss_geo_kernel(int nx, int ny, const double* __restrict__ data,
                                 const double* __restrict__ lons, const double* __restrict__ lats,
                                 double sigma, double* __restrict__ out) {
    extern __shared__ double sh[];   // [2][wn]: sin^2(dlat/2), cos(lat1)
    const int j = blockIdx.y;
    const double sigma3 = 3.0 * sigma;
    const double dx = lons[1] - lons[0];
    const double dy = lats[1] - lats[0];
    const int hx = static_cast<int>(sigma3 / dx);
    const double cos_lat0 = cos(lats[j] * DEG2RAD_T);
    const int hy = static_cast<int>(sigma3 / cos_lat0 / dy);
    const int n1 = max(0, j - hy);
    const int n2 = min(ny - 1, j + hy);
    const int wn = n2 - n1 + 1;
    double* s2lat = sh;
    double* clat1 = sh + wn;
    for (int q = threadIdx.x; q < wn; q += blockDim.x) {
        const double s = sin((lats[n1 + q] - lats[j]) * (DEG2RAD_T * 0.5));
        s2lat[q] = s * s;
        clat1[q] = cos(lats[n1 + q] * DEG2RAD_T);
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nx) return;
    const double inv_2sig2 = 1.0 / (2.0 * (sigma * sigma));
    const int m1 = max(0, i - hx);
    const int m2 = min(nx - 1, i + hx);
    double sw = 0.0, swd = 0.0;
    for (int m = m1; m <= m2; m++) {
        const double s = sin((lons[m] - lons[i]) * (DEG2RAD_T * 0.5));
        const double lon_c = cos_lat0 * (s * s);
        const double* col = data + m;
        for (int q = 0; q < wn; q++) {
            const double a = s2lat[q] + lon_c * clat1[q];
            const double w = exp(-dist2_deg(a) * inv_2sig2);
            sw += w;
            swd += w * col[(size_t)nx * (n1 + q)];
        }
    }
    out[i + (size_t)nx * j] = swd / sw;
}

// block row y: the period.  *odd is set where the smoothed topography is not
// finite.
__global__ void media_kernel(int nx, int ny, const double* __restrict__ zs,
                             const double* __restrict__ lon, const double* __restrict__ lat,
                             double* m11, double* m12, double* m22, double* angle, int* odd) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= (size_t)nx * ny) return;
    const size_t plane = blockIdx.y * (size_t)nx * ny;
    const double* z = zs + plane;
    if (!isfinite(z[k])) *odd = 1;
    m11 += plane;
    m12 += plane;
    m22 += plane;
    angle += plane;
    const int i = (int)(k % nx), j = (int)(k / nx);
    const double km = R_EARTH_T * DEG2RAD_T;
    const double clat = cos(lat[j] * DEG2RAD_T);
    auto F = [&](int a, int b) { return z[a + (size_t)nx * b]; };
    auto dxk = [&](int a) { return (lon[a] - lon[a - 1]) * km; };
    auto dyk = [&](int b) { return (lat[b] - lat[b - 1]) * km; };
    double fx, fy;
    if (i == 0) fx = (F(1, j) - F(0, j)) / (dxk(1) * clat);
    else if (i == nx - 1) fx = (F(nx - 1, j) - F(nx - 2, j)) / (dxk(nx - 1) * clat);
    else fx = (F(i + 1, j) - F(i - 1, j)) / (2.0 * (dxk(i) * clat));
    if (j == 0) fy = (F(i, 1) - F(i, 0)) / (1.0 * dyk(1));
    else if (j == ny - 1) fy = (F(i, ny - 1) - F(i, ny - 2)) / (1.0 * dyk(ny - 1));
    else fy = (F(i, j + 1) - F(i, j - 1)) / (2.0 * (1.0 * dyk(j)));
    const double fx2 = fx * fx, fy2 = fy * fy;
    angle[k] = atan(sqrt(fx2 + fy2)) * RAD2DEG_T;
    const double denom = 1.0 + fx2 + fy2;
    m11[k] = (1.0 + fy2) / denom;
    m22[k] = (1.0 + fx2) / denom;
    m12[k] = -(fx * fy / denom);
}

__global__ void depth_topo_kernel(int nx, int ny, int nz, int nper, const double* __restrict__ zg,
                                  const double* __restrict__ angle, double* k0, double* k1,
                                  double* k2) {
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (t >= (size_t)nx * ny * nper) return;
    const int ip = (int)(t % nper);
    const size_t col = t / nper;
    const int iy = (int)(col % ny), ix = (int)(col / ny);
    double cosang = cos(angle[(size_t)ip * nx * ny + ix + (size_t)nx * iy] * DEG2RAD_T);
    if (!isfinite(cosang) || fabs(cosang) < 1e-6) cosang = 1e-6;
    const double zmin = zg[0], zmax = zg[nz - 1];
    const size_t base = col * nz * nper + ip;
    double* ks[3] = {k0, k1, k2};
    double c[64];
    for (int a = 0; a < 3; a++) {
        double* K = ks[a];
        if (!K) continue;
        for (int q = 0; q < nz; q++) c[q] = K[base + (size_t)q * nper];
        for (int q = 0; q < nz; q++) {
            const double qx = fmin(fmax(zg[q] / cosang, zmin), zmax);
            double v;
            if (qx < zg[0]) v = c[0];
            else if (qx > zg[nz - 1]) v = c[nz - 1];
            else {
                int lo = 0, hi = nz;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (zg[mid] < qx) lo = mid + 1;
                    else hi = mid;
                }
                int i = lo;
                if (i == nz) --i;
                if (i > 0 && zg[i] > qx) --i;
                i = max(0, min(i, nz - 2));
                const double x1 = zg[i], x2 = zg[i + 1];
                const double tt = (qx - x1) / (x2 - x1);
                v = (1 - tt) * c[i] + tt * c[i + 1];
            }
            K[base + (size_t)q * nper] = v;
        }
    }
}

__global__ void grid_kernel(int nxr, int nyr, const double* __restrict__ xr,
                            const double* __restrict__ yr, const double* __restrict__ zr, int nx,
                            int ny, const double* __restrict__ x, const double* __restrict__ y,
                            double* out) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= (size_t)nx * ny) return;
    const int i = (int)(k % nx), j = (int)(k / nx);
    out[k] = interp2d_pt(xr, nxr, yr, nyr, zr, x[i], y[j]);
}
}  // namespace

constexpr int kGeoShared = 227 * 1024;   // bytes of a block at most
constexpr int kGeoRows = 48 * 1024 / 16;
bool gauss_geo_fits(int ny) { return ny <= kGeoShared / 16; }

cudaError_t launch_gauss_geo(int nx, int ny, const double* data, const double* lons,
                             const double* lats, double sigma, double* out, cudaStream_t st) {
    // (set for tall grids only: up to 48 KB need no limit)
    if (ny > kGeoRows) {
        const cudaError_t e = cudaFuncSetAttribute(
            gauss_geo_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGeoShared);
        if (e != cudaSuccess) return e;
    }
    dim3 grid((nx + 127) / 128, ny);
    gauss_geo_kernel<<<grid, 128, 2 * ny * sizeof(double), st>>>(nx, ny, data, lons, lats, sigma,
                                                                 out);
    return cudaGetLastError();
}

cudaError_t launch_gauss_rows(int nx, int ny, int nper, const double* data, const double* lats,
                              const double* off, double h, const double* sigmas, double sigma_max,
                              double* out, cudaStream_t st) {
    // latitudes at a time: whole turns of the four groups, two blocks an SM
    // (their registers allow no more), or else what fits one
    const long long hx = std::min<long long>((long long)(3.0 * sigma_max / h), nx - 1);
    const int most = gauss_pitch((int)hx);
    const size_t row = ((size_t)most + 4 * gauss_quarter(nx)) * sizeof(double2);
    const size_t rest = 2 * (size_t)most * sizeof(double2) + 4 * kGaussCells * sizeof(double);
    int rows = 12;
    while (rows > 4 && rest + rows * row > 110 * 1024) rows -= 4;
    while (rows > 1 && rest + rows * row > kGaussShared) rows--;
    const size_t bytes = rest + rows * row;
    if (bytes > kGaussShared) return cudaErrorInvalidConfiguration;   // (gauss_rows_fits)
    // (the limit belongs to the device and threads launch at the same time: the
    // largest that any call needs, not this one's)
    const cudaError_t e = cudaFuncSetAttribute(
        gauss_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGaussShared);
    if (e != cudaSuccess) return e;
    gauss_rows_kernel<<<dim3(ny, nper), kGaussThreads, bytes, st>>>(nx, ny, data, lats, off, h,
                                                                    sigmas, rows, most, out);
    return cudaGetLastError();
}

bool gauss_rows_fits(int nx) { return nx <= 2000; }

cudaError_t launch_topo_media(int nx, int ny, int nper, const double* z, const double* lon,
                              const double* lat, double* m11, double* m12, double* m22,
                              double* angle, int* odd, cudaStream_t st) {
    const size_t n = (size_t)nx * ny;
    media_kernel<<<dim3((unsigned)((n + 255) / 256), nper), 256, 0, st>>>(nx, ny, z, lon, lat, m11,
                                                                          m12, m22, angle, odd);
    return cudaGetLastError();
}

cudaError_t launch_depth_topo(int nx, int ny, int nz, int nper, const double* zg,
                              const double* angle, double* k0, double* k1, double* k2,
                              cudaStream_t st) {
    const size_t n = (size_t)nx * ny * nper;
    depth_topo_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(nx, ny, nz, nper, zg, angle, k0,
                                                                   k1, k2);
    return cudaGetLastError();
}

cudaError_t launch_grid_topo(int nxr, int nyr, const double* xr, const double* yr,
                             const double* zr, int nx, int ny, const double* x, const double* y,
                             double* out, cudaStream_t st) {
    const size_t n = (size_t)nx * ny;
    grid_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nxr, nyr, xr, yr, zr, nx, ny, x, y,
                                                             out);
    return cudaGetLastError();
}

}  // namespace sa
