// PDE kernel smoothing (PostProc::pde_smooth, reference src/postproc.cpp:388-463):
// explicit Euler steps of the spherical 7-point Laplacian with Neumann boundary
// copies over a row-major (nx, ny, nz) field, depth fastest: one launch per
// step, one for all steps of a small field, one for two of a large one.  Compiled with -fmad=false: every product and sum rounds as the
// reference's FP64 expression reads (row and depth factors are formed on the
// host in the reference's left-to-right order).
//
// The boundary copies of :130-158 (x faces, then y faces, then z faces) leave
// every boundary cell equal to the updated cell at the clamped index
// (ix, iy, k) -> (clamp(ix, 1, nx-2), clamp(iy, 1, ny-2), clamp(k, 1, nz-2)),
// so one pass of pde_step_kernel writes the whole step: a boundary thread
// recomputes the update of its clamped interior cell.  One read and one write
// of the field per step, neighbours from L1/L2.
#include "launch.h"

#include <cooperative_groups.h>
#include <cuda_pipeline.h>
#include <type_traits>
#include <utility>

namespace sa {

struct PdeConst {
    int nx, ny, nz;
    double B;     // ch * dy2_inv
    double D;     // cv * dz2_inv
};

// One cell's update from its neighbours along x, y and z (p above, m below):
// src/postproc.cpp:91-124 and, with dt = 1, :453.
__device__ __forceinline__ double pde_update(const PdeConst& P, double c, double xp, double xm,
                                             double yp, double ym, double zp, double zm,
                                             double rx, double ry, double de) {
    const double d2u_dx2 = rx * (xp + xm - 2.0 * c);
    const double d2u_dy2 = P.B * (yp + ym - 2.0 * c);
    const double du_dy = ry * (yp - ym);
    const double lat_term = d2u_dy2 - du_dy;
    const double d2u_dz2 = P.D * (zp + zm - 2.0 * c);
    const double du_dz = de * (zp - zm);
    const double depth_term = d2u_dz2 - du_dz;
    return c + 1.0 * (d2u_dx2 + lat_term + depth_term);
}

__global__ void __launch_bounds__(256) pde_step_kernel(PdeConst P, const double* __restrict__ u,
                                                       double* __restrict__ out,
                                                       const double* __restrict__ rowX,
                                                       const double* __restrict__ rowY,
                                                       const double* __restrict__ depE) {
    const size_t n = (size_t)P.nx * P.ny * P.nz;
    const size_t sy = (size_t)P.nz, sx = (size_t)P.ny * P.nz;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i % P.nz);
        const size_t col = i / P.nz;
        const int iy = (int)(col % P.ny);
        const int ix = (int)(col / P.ny);
        const int cx = min(max(ix, 1), P.nx - 2);
        const int cy = min(max(iy, 1), P.ny - 2);
        const int ck = min(max(k, 1), P.nz - 2);
        const size_t c = ((size_t)cx * P.ny + cy) * P.nz + ck;
        out[i] = pde_update(P, u[c], u[c + sx], u[c - sx], u[c + sy], u[c - sy], u[c + 1],
                            u[c - 1], rowX[cy], rowY[cy], depE[ck]);
    }
}

// Division by an invariant divisor d as a multiply-high and a shift
// (Granlund and Montgomery, PLDI 1994, section 4): s = ceil(log2 d),
// m = floor(2^32 (2^s - d) / d) + 1, q = (umulhi(n, m) + n) >> s, exact for
// every n < 2^31 (the sum then fits 32 bits).
struct FastDiv {
    unsigned d, m, s;
};
static FastDiv make_fastdiv(unsigned d) {
    unsigned s = 0;
    while ((1ull << s) < d) s++;
    const unsigned long long m = ((1ull << 32) * ((1ull << s) - d)) / d + 1;
    return {d, (unsigned)m, s};
}
__device__ __forceinline__ unsigned fdiv_q(unsigned n, const FastDiv& f) {
    return (__umulhi(n, f.m) + n) >> f.s;
}

// The same step with 32-bit cell indices (fields below 2^31 cells): the
// row, column and depth of a cell from two multiply-high divisions instead
// of 64-bit divisions, which made the index arithmetic the bulk of the
// instructions.
// Fields of some 60 000 to 2 million cells are bound by the launch of each
// step (about 2 us of kernel): launched as a programmatic dependent, a step's
// blocks are set up while the step before runs.  61x70x30 4.56 -> 3.60 us a
// step, 100x90x33 4.62 -> 3.28, 31x300x15 4.49 -> 2.47, 301x260x17 8.7 -> 7.2.
// (Blocks come while the step before writes u, so u and out are plain
// pointers: `__restrict__` would let u be read as if it never changed.)
__global__ void __launch_bounds__(256) pde_step_kernel32(PdeConst P, FastDiv fz, FastDiv fy,
                                                         const double* u, double* out,
                                                         const double* __restrict__ rowX,
                                                         const double* __restrict__ rowY,
                                                         const double* __restrict__ depE) {
    const unsigned n = (unsigned)P.nx * P.ny * P.nz;
    const unsigned sy = (unsigned)P.nz, sx = (unsigned)P.ny * P.nz;
    cudaTriggerProgrammaticLaunchCompletion();   // (the next step's blocks may come and wait)
    cudaGridDependencySynchronize();             // the step before is complete
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned col = fdiv_q(i, fz);
        const int k = (int)(i - col * fz.d);
        const unsigned ixu = fdiv_q(col, fy);
        const int iy = (int)(col - ixu * fy.d);
        const int ix = (int)ixu;
        const int cx = min(max(ix, 1), P.nx - 2);
        const int cy = min(max(iy, 1), P.ny - 2);
        const int ck = min(max(k, 1), P.nz - 2);
        const unsigned c = ((unsigned)cx * P.ny + cy) * P.nz + ck;
        out[i] = pde_update(P, u[c], u[c + sx], u[c - sx], u[c + sy], u[c - sy], u[c + 1],
                            u[c - 1], rowX[cy], rowY[cy], depE[ck]);
    }
}

// One interior cell's value to `out` and to the boundary cells that copy it.
__device__ __forceinline__ void pde_store(const PdeConst& P, double* __restrict__ out, int x,
                                          int y, int z, double v) {
    const int xa = x == 1 ? 0 : x, xb = x == P.nx - 2 ? P.nx - 1 : x;
    const int ya = y == 1 ? 0 : y, yb = y == P.ny - 2 ? P.ny - 1 : y;
    const int za = z == 1 ? 0 : z, zb = z == P.nz - 2 ? P.nz - 1 : z;
    for (int i = xa; i <= xb; i++)
        for (int j = ya; j <= yb; j++)
            for (int k = za; k <= zb; k++) out[((size_t)i * P.ny + j) * P.nz + k] = v;
}

// Two steps in one pass over memory.  A block marches along x over a tile of
// rows and depths with a margin of two cells; a thread owns kRows neighbouring
// rows at one depth and holds their last planes before and after the first
// step in registers.  The planes to come are copied to shared memory some
// steps ahead; the plane in the middle of either step stands there for the
// neighbours along y and z (one barrier a plane).  A boundary cell after a
// step is the copy of its clamped interior cell, so a pass writes interior
// cells only and (`clamped`) reads the interior cells in place of the
// boundary, which is written once after the last pass.
//
// Bound by the chain of a plane's two updates between barriers (FP64 pipe 46 %
// busy, issue slots 58 %, L1 67 %, HBM 30 %): 601x601x50, 108 us for two steps
// against 150 of two launches of one step, which read and write the field
// twice.  512 threads of 128 registers and one block per SM: two blocks of
// 320 at 96 take 126 us, two of 256 (a tile of 20 rows, 4 of them margin)
// 116, 640 at 96 114, 768 at 80 (spilling) 222.  Groups of rows padded against
// bank conflicts made no difference; the second step a plane behind the first,
// so that neither waits for the other, is 4 % slower.
constexpr int kRows = 4;
constexpr int kRing = 5;
constexpr int PASS_THREADS = 512;   // 128 registers
constexpr int kPassDepths = 64;     // depths of a block at most
// bytes of a block at most: kRows rows for each of its threads, two more of
// kPassDepths and a cell at either end, kRing planes before and 2 after a step
constexpr int kPassShared = (kRing + 2) * (kRows * PASS_THREADS + 2 * kPassDepths + 2) * 8;
struct PassTiles {
    int tx, ty, tz;   // interior cells per tile
    int nty;          // tiles along y
    int zl, groups;   // depths and row groups a block holds
    int clamped;
};

__global__ void __launch_bounds__(PASS_THREADS, 1)
pde_pass_kernel(PdeConst P, PassTiles L, const double* __restrict__ u, double* __restrict__ out,
                const double* __restrict__ rowX, const double* __restrict__ rowY,
                const double* __restrict__ depE) {
    extern __shared__ double sh[];
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const int x0 = 1 + blockIdx.y * L.tx, x1 = min(x0 + L.tx, nx - 1);
    const int y0 = 1 + (blockIdx.x % L.nty) * L.ty, y1 = min(y0 + L.ty, ny - 1);
    const int z0 = 1 + (blockIdx.x / L.nty) * L.tz, z1 = min(z0 + L.tz, nz - 1);
    const int ya = max(y0 - 2, 0), yb = min(y1 + 2, ny);
    const int za = max(z0 - 2, 0), zb = min(z1 + 2, nz);
    const int zl = L.zl;
    const int lg = threadIdx.x / zl, lz = threadIdx.x - lg * zl;
    const int z = za + lz, y = ya + lg * kRows;
    const bool in = lg < L.groups && z < zb;
    const bool zlo = in && z == 1, zhi = in && z == nz - 2;
    const bool zin = in && z >= 1 && z < nz - 1;
    const bool yedge = y0 == 1 || y1 == ny - 1;
    // a row before and after the tile and a cell at either end are never used
    // for a result, only read
    const int size = (kRows * L.groups + 2) * zl + 2;
    const int own = 1 + (1 + min(lg, L.groups - 1) * kRows) * zl + lz;
    const size_t plane = (size_t)ny * nz;
    double rx[kRows], ry[kRows];
    size_t from[kRows];   // offset in a plane of what is read
    bool row[kRows], put[kRows];
#pragma unroll
    for (int j = 0; j < kRows; j++) {
        row[j] = in && y + j < yb;
        put[j] = in && z >= z0 && z < z1 && y + j >= y0 && y + j < y1;
        rx[j] = row[j] ? rowX[y + j] : 0.0;
        ry[j] = row[j] ? rowY[y + j] : 0.0;
        const int cy = L.clamped ? min(max(y + j, 1), ny - 2) : y + j;
        const int cz = L.clamped ? min(max(z, 1), nz - 2) : z;
        from[j] = row[j] ? (size_t)cy * nz + cz : 0;
    }
    const double de = in ? depE[z] : 0.0;
    const int a1 = max(x0 - 1, 1);               // first plane of the first step
    const int xe = min(x1, nx - 2) + 1;          // last plane that is read
    auto xsrc = [&](int x) {
        return u + (size_t)(L.clamped ? min(max(x, 1), nx - 2) : x) * plane;
    };
    double* const S1 = sh + kRing * size;
    auto fetch = [&](int x) {   // a thread copies the cells that it owns
        double* s = sh + (x % kRing) * size + own;
        if (x <= xe) {
            const double* p = xsrc(x);
#pragma unroll
            for (int j = 0; j < kRows; j++)
                if (row[j]) __pipeline_memcpy_async(s + j * zl, p + from[j], 8);
        }
        __pipeline_commit();
    };
    double A[kRows], B[kRows], C[kRows], D[kRows], E[kRows], F[kRows];
#pragma unroll
    for (int i = 0; i < kRing - 1; i++) fetch(a1 + i);
#pragma unroll
    for (int j = 0; j < kRows; j++) {
        A[j] = row[j] ? xsrc(a1 - 1)[from[j]] : 0.0;
        C[j] = D[j] = E[j] = F[j] = 0.0;
    }
    __pipeline_wait_prior(kRing - 2);
#pragma unroll
    for (int j = 0; j < kRows; j++) B[j] = row[j] ? sh[(a1 % kRing) * size + own + j * zl] : 0.0;
    double* dst = out + (size_t)(a1 - 1) * plane + (size_t)y * nz + z;   // plane xs - 1
    // planes xs - 1, xs, xs + 1 before the first step: p, c, n;
    // xs - 2, xs - 1, xs after it: q, r, v
    auto both = [&](int xs, const double (&p)[kRows], const double (&c)[kRows],
                    double (&n)[kRows], double (&q)[kRows], const double (&r)[kRows],
                    double (&v)[kRows]) {
        const double* S0 = sh + (xs % kRing) * size + own;
        const double* N0 = sh + ((xs + 1) % kRing) * size + own;
        double* S = S1 + ((xs & 1) ? size : 0) + own;
        __pipeline_wait_prior(kRing - 3);   // planes up to xs + 1
        if (zin) {
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                if (j == 0 && y == ny - 1) continue;   // the group before writes it
                S[j * zl] = r[j];
                if (zlo) S[j * zl - 1] = r[j];
                if (zhi) S[j * zl + 1] = r[j];
            }
            // row ny - 1 of the next group is the copy of this one's last
            if (y + kRows == ny - 1) S[kRows * zl] = r[kRows - 1];
        }
        __syncthreads();
        fetch(xs + kRing - 1);   // over plane xs - 1, whose readers have passed
        if (xs < nx - 1) {
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                n[j] = N0[j * zl];
                const double yp = j + 1 < kRows ? c[j + 1] : S0[kRows * zl];
                const double ym = j > 0 ? c[j - 1] : S0[-zl];
                v[j] = pde_update(P, c[j], n[j], p[j], yp, ym, S0[j * zl + 1], S0[j * zl - 1],
                                  rx[j], ry[j], de);
            }
            if (yedge) {
                if (y == 0) v[0] = v[1];
#pragma unroll
                for (int j = 1; j < kRows; j++)
                    if (y + j == ny - 1) v[j] = v[j - 1];
            }
        } else {
#pragma unroll
            for (int j = 0; j < kRows; j++) v[j] = r[j];
        }
        if (xs > x0) {
            if (xs == 2) {
#pragma unroll
                for (int j = 0; j < kRows; j++) q[j] = r[j];
            }
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const double yp = j + 1 < kRows ? r[j + 1] : S[kRows * zl];
                const double ym = j > 0 ? r[j - 1] : S[-zl];
                const double w = pde_update(P, r[j], v[j], q[j], yp, ym, S[j * zl + 1],
                                            S[j * zl - 1], rx[j], ry[j], de);
                if (put[j]) dst[j * nz] = w;
            }
        }
        dst += plane;
    };
    for (int xs = a1; xs <= x1; xs += 3) {
        both(xs, A, B, C, D, E, F);
        if (xs + 1 > x1) break;
        both(xs + 1, B, C, A, E, F, D);
        if (xs + 2 > x1) break;
        both(xs + 2, C, A, B, F, D, E);
    }
    __pipeline_wait_prior(0);
}

// The boundary copies, with a copy of the field (out) or in place (out = u).
__global__ void __launch_bounds__(256)
pde_boundary_kernel(PdeConst P, const double* u, double* out) {
    const size_t n = (size_t)P.nx * P.ny * P.nz;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i % P.nz);
        const size_t col = i / P.nz;
        const int iy = (int)(col % P.ny), ix = (int)(col / P.ny);
        const size_t c = ((size_t)min(max(ix, 1), P.nx - 2) * P.ny + min(max(iy, 1), P.ny - 2)) *
                             P.nz + min(max(k, 1), P.nz - 2);
        if (out != u || c != i) out[i] = u[c];
    }
}

// All steps of a small field in one launch: a cluster of blocks holds it in
// shared memory, each a range of row groups (kRows neighbouring rows of one x)
// and copies of the plane's worth of groups before and after it, into which
// its neighbours write what they update; a thread has one depth of one group,
// a cluster barrier ends a step.  41x41x30: 2.1 us a step, most of it the
// barrier and the remote stores before it; a launch per step takes 1.9 us of
// kernel, a gap, and 2 to 3 us of the host, which it keeps busy all along
// (60 steps 293 us with a launch each, 160 now).
constexpr int kCluster = 16, kClusterThreads = 1024;
constexpr int kClusterShared = 227 * 1024;   // bytes of a block at most
__global__ void __launch_bounds__(kClusterThreads, 1)
pde_cluster_kernel(PdeConst P, int G, int W, int nstep, double* field,
                   const double* __restrict__ rowX, const double* __restrict__ rowY,
                   const double* __restrict__ depE) {
    extern __shared__ double sh[];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int nx = P.nx, ny = P.ny, nz = P.nz, tid = threadIdx.x;
    const int U = (nx - 2) * G;   // groups of the interior planes, from plane 1 on
    const int u0 = min(rank * W, U), u1 = min(u0 + W, U);
    const int un = kRows * nz, size = (W + 2 * G) * un;
    double* cX = sh + 2 * size;
    double* cY = cX + kRows * G;
    for (int i = tid; i < kRows * G; i += kClusterThreads) {
        cX[i] = i < ny ? rowX[i] : 0.0;
        cY[i] = i < ny ? rowY[i] : 0.0;
    }
    // groups u0 - G .. u1 + G - 1 of the field (group -G is plane 0's first)
    for (int i = tid; i < (u1 - u0 + 2 * G) * un; i += kClusterThreads) {
        const int l = i / un, q = i - l * un;
        const int g = u0 + l, x = g / G, y = (g - x * G) * kRows + q / nz;
        sh[i] = y < ny ? field[((size_t)x * ny + y) * nz + q % nz] : 0.0;
    }
    const int zi = nz - 2, lu = tid / zi;
    const bool live = lu < u1 - u0;
    const int z = 1 + (tid - lu * zi), x = 1 + (u0 + lu) / G, y0 = ((u0 + lu) % G) * kRows;
    const int off = (lu + G) * un + z;
    const int sx = G * un;
    const double de = live ? depE[z] : 0.0;
    double c[kRows];
    cluster.sync();
#pragma unroll
    for (int j = 0; j < kRows; j++) c[j] = live ? sh[off + j * nz] : 0.0;
    // the neighbours' copies of this thread's group
    double* const prev =
        live && rank > 0 && lu < G ? cluster.map_shared_rank(sh, rank - 1) + W * un : nullptr;
    double* const next = live && rank + 1 < kCluster && lu + G >= W
                             ? cluster.map_shared_rank(sh, rank + 1) - W * un
                             : nullptr;
    for (int s = 0; s < nstep; s++) {
        const double* A = sh + (s & 1) * size + off;
        const int to = (~s & 1) * size + off;
        if (live) {
            double nv[kRows];
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const int o = j * nz, y = y0 + j;
                const double m = c[j];
                double xp = A[o + sx], xm = A[o - sx], zp = A[o + 1], zm = A[o - 1];
                double yp = j + 1 < kRows ? c[j + 1] : A[o + nz];
                double ym = j > 0 ? c[j - 1] : A[o - nz];
                if (s > 0) {   // boundary cells are copies by now
                    if (x == nx - 2) xp = m;
                    if (x == 1) xm = m;
                    if (y == ny - 2) yp = m;
                    if (y == 1) ym = m;
                    if (z == nz - 2) zp = m;
                    if (z == 1) zm = m;
                }
                nv[j] = pde_update(P, m, xp, xm, yp, ym, zp, zm, cX[y], cY[y], de);
            }
#pragma unroll
            for (int j = 0; j < kRows; j++) {
                const int o = to + j * nz;
                if (y0 + j == 0 || y0 + j >= ny - 1) continue;
                c[j] = nv[j];
                sh[o] = nv[j];
                if (prev) prev[o] = nv[j];
                if (next) next[o] = nv[j];
            }
        }
        cluster.sync();
    }
    if (!live) return;
#pragma unroll
    for (int j = 0; j < kRows; j++)
        if (y0 + j > 0 && y0 + j < ny - 1) pde_store(P, field, x, y0 + j, z, c[j]);
}

namespace {

// (The limit on a kernel's dynamic shared memory belongs to the device, not to
// the launch after it, and threads launch at the same time: every call sets
// the largest that any call needs.)

// The cluster form where the field fits: two copies of a block's groups and
// their margins in its shared memory, a thread for each depth of its groups
// (fields to about 57 000 cells; with two depths a thread 61x70x30 takes
// 4.1 us a step, a launch each 3.6).
cudaError_t try_cluster(const PdeConst& P, int nstep, double* field, const double* rowX,
                        const double* rowY, const double* depE, bool* done, cudaStream_t st) {
    const long long G = (P.ny + kRows - 1) / kRows, U = (long long)(P.nx - 2) * G;
    const long long W = std::max((U + kCluster - 1) / kCluster, G);
    const long long smem =
        2 * ((W + 2 * G) * kRows * P.nz + kRows * G) * (long long)sizeof(double);
    *done = false;
    if (smem > kClusterShared || W * (P.nz - 2) > kClusterThreads) return cudaSuccess;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(pde_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kClusterShared)))
        return e;
    if ((e = cudaFuncSetAttribute(pde_cluster_kernel,
                                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
        return e;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kCluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, pde_cluster_kernel, &cfg) != cudaSuccess || fit < 1) {
        cudaGetLastError();   // no such cluster on this device
        return cudaSuccess;
    }
    *done = true;
    return cudaLaunchKernelEx(&cfg, pde_cluster_kernel, P, (int)G, (int)W, nstep, field, rowX,
                              rowY, depE);
}

}  // namespace

cudaError_t launch_pde_smooth(int nx, int ny, int nz, double B, double D, const double* rowX,
                              const double* rowY, const double* depE, int nstep, double* field,
                              double* work, cudaStream_t st) {
    PdeConst P{nx, ny, nz, B, D};
    const size_t n = (size_t)nx * ny * nz;
    bool done = false;
    cudaError_t e = try_cluster(P, nstep, field, rowX, rowY, depE, &done, st);
    if (e != cudaSuccess || done) return e;
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, (size_t)nsm * 8);
    const bool idx32 = n < (1ull << 31);
    const FastDiv fz = make_fastdiv((unsigned)nz), fy = make_fastdiv((unsigned)ny);
    double* a = field;
    double* b = work;
    auto single = [&]() {
        cudaError_t r = cudaSuccess;
        if (idx32) {
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[0].val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(blocks);
            cfg.blockDim = dim3(256);
            cfg.stream = st;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            r = cudaLaunchKernelEx(&cfg, pde_step_kernel32, P, fz, fy, (const double*)a, b, rowX,
                                   rowY, depE);
        }
        else pde_step_kernel<<<blocks, 256, 0, st>>>(P, a, b, rowX, rowY, depE);
        std::swap(a, b);
        return r != cudaSuccess ? r : cudaGetLastError();
    };
    // Depths in equal tiles of at most 60 and their margins, then as many rows
    // as a block's threads hold in equal tiles, then the planes in as many
    // ranges as there are blocks left.
    PassTiles L;
    const int ntz = nz <= kPassDepths ? 1 : (nz - 2 + kPassDepths - 5) / (kPassDepths - 4);
    L.tz = (nz - 2 + ntz - 1) / ntz;
    L.zl = ntz == 1 ? nz : L.tz + 4;
    const int rows = PASS_THREADS / L.zl * kRows - 4;
    L.nty = (ny - 2 + rows - 1) / rows;
    L.ty = (ny - 2 + L.nty - 1) / L.nty;
    L.groups = (std::min(L.ty + 4, ny) + kRows - 1) / kRows;
    const long long tiles = (long long)L.nty * ntz;
    const int ranges = (int)std::max<long long>(1, nsm / tiles);
    L.tx = std::max((nx - 2 + ranges - 1) / ranges, 16);
    const long long nr = (nx - 2 + L.tx - 1) / L.tx;
    // Two steps a pass where a pass has planes enough to fill its pipeline and
    // the blocks their threads: 301x301x40 13 us a step against 16,
    // 301x260x17 8.3 against 7.2, 200x180x40 7.8 against 7.7, 150x140x30 7.8
    // against 4.7, the latency of a range's planes being the same.
    if (n < (1ull << 21) || 2 * L.groups * L.zl < PASS_THREADS || nr * L.tx < 32 || nr > 65535) {
        for (int s = 0; s < nstep; s++)
            if ((e = single()) != cudaSuccess) return e;
        if (a != field)
            return cudaMemcpyAsync(field, a, n * sizeof(double), cudaMemcpyDeviceToDevice, st);
        return cudaSuccess;
    }
    const size_t smem =
        (kRing + 2) * ((size_t)(kRows * L.groups + 2) * L.zl + 2) * sizeof(double);
    if ((e = cudaFuncSetAttribute(pde_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kPassShared)))
        return e;
    const dim3 grid((unsigned)tiles, (unsigned)nr);
    int s = nstep & 1;
    if (s && (e = single()) != cudaSuccess) return e;
    L.clamped = 0;
    for (; s < nstep; s += 2) {
        pde_pass_kernel<<<grid, PASS_THREADS, smem, st>>>(P, L, a, b, rowX, rowY, depE);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        L.clamped = 1;
        std::swap(a, b);
    }
    pde_boundary_kernel<<<blocks, 256, 0, st>>>(P, a, field);
    return cudaGetLastError();
}

}  // namespace sa
