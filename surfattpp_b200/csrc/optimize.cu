// Optimizer primitives on device (vs-only parametrisation): deterministic FP64
// inner products and max-abs, the L-BFGS history vectors, axpy-type updates
// and the multiplicative model update with the Brocher relations.
// Reference: src/optimize.cpp:14-255, src/inversion.cpp:302-323, :465-490.
// Compiled with -fmad=false: elementwise results round as the reference's.
// All kernels are HBM-bound streams over n values.  Sums run over a fixed
// grid in a fixed order, the last block to finish adding the blocks' partial
// sums, so that a reduction is one launch and what follows from it (the
// two-loop recursion's coefficients, the normalisation) stays on the device:
// an L-BFGS step on 3.6 M values (store, direction, normalisation, angle,
// update) took 60 launches and 21 waits of the host (1100 us), now 16 and 4
// (368 us).
// The recursion's passes are launched as programmatic dependents, their blocks
// set up while the pass before runs (the direction 245 -> 227 us; 20 000
// values 107 -> 72 us, also by launching only blocks with an element).
#include "launch.h"

namespace sa {

namespace {
constexpr int RED_BLOCKS = 1184;   // 148 SMs x 8: fixed, so sums are reproducible
constexpr int RED_THREADS = 256;

__device__ __forceinline__ double brocher_vs2vp(double vs) {   // include/utils.h:237-245
    return 0.9409 + 2.0947 * vs - 0.8206 * vs * vs + 0.2683 * vs * vs * vs
         - 0.0251 * vs * vs * vs * vs;
}
__device__ __forceinline__ double brocher_vp2rho(double vp) {  // include/utils.h:247-254
    return 1.6612 * vp - 0.4721 * vp * vp + 0.0671 * vp * vp * vp - 0.0043 * vp * vp * vp * vp
         + 0.000106 * vp * vp * vp * vp * vp;
}

// One block's sum (OP 0) or maximum (OP 1) in thread 0.
template <int OP, int W>
__device__ double block_tree(double* sh) {
    __syncthreads();
    for (int w = W / 2; w > 0; w >>= 1) {
        for (int q = threadIdx.x; q < w; q += RED_THREADS)
            sh[q] = OP == 0 ? sh[q] + sh[q + w] : fmax(sh[q], sh[q + w]);
        __syncthreads();
    }
    const double v = sh[0];
    __syncthreads();
    return v;
}

// K sums over the grid, out[K] in every thread of the last block to come,
// for which it returns true.  partial [K][RED_BLOCKS], count zero before and
// after.  The order of the additions is that of the grid and of one 1024-wide
// tree, whichever block is last.
template <int K>
__device__ bool grid_sums(const double (&acc)[K], double* partial, unsigned* count,
                          double (&out)[K]) {
    __shared__ double sh[1024];
    __shared__ bool last;
    const int t = threadIdx.x;
    for (int k = 0; k < K; k++) {
        sh[t] = acc[k];
        const double v = block_tree<0, RED_THREADS>(sh);
        if (t == 0) partial[(size_t)k * RED_BLOCKS + blockIdx.x] = v;
    }
    if (t == 0) {
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
        if (last) *count = 0u;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    for (int k = 0; k < K; k++) {
        for (int q = t; q < 1024; q += RED_THREADS) {
            double v = 0.0;
            for (int i = q; i < (int)gridDim.x; i += 1024)
                v += __ldcg(partial + (size_t)k * RED_BLOCKS + i);
            sh[q] = v;
        }
        out[k] = block_tree<0, 1024>(sh);
    }
    return true;
}

// max |a| of absmax_kernel's partials, in every thread of the calling block
__device__ double absmax_of(const double* partial) {
    __shared__ double sh[RED_THREADS];
    double v = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += RED_THREADS) v = fmax(v, partial[i]);
    sh[threadIdx.x] = v;
    return block_tree<1, RED_THREADS>(sh);
}

#define RED_LOOP(i, n)                                                      \
    for (size_t i = blockIdx.x * (size_t)RED_THREADS + threadIdx.x; i < (n); \
         i += (size_t)RED_BLOCKS * RED_THREADS)

// out[0] = sum a b; with `angle` also out[1] = sum a a, out[2] = sum b b
template <int K>
__global__ void __launch_bounds__(RED_THREADS)
dot_kernel(size_t n, const double* __restrict__ a, const double* __restrict__ b, double* partial,
           unsigned* count, double* out) {
    double acc[K] = {}, res[K];
    RED_LOOP(i, n) {
        const double x = a[i], y = b[i];
        acc[0] += x * y;
        if (K == 3) {
            acc[1] += x * x;
            acc[K - 1] += y * y;
        }
    }
    if (grid_sums(acc, partial, count, res) && threadIdx.x == 0)
        for (int k = 0; k < K; k++) out[k] = res[k];
}

__global__ void __launch_bounds__(RED_THREADS)
absmax_kernel(size_t n, const double* __restrict__ a, double* partial) {
    __shared__ double sh[RED_THREADS];
    double acc = 0.0;
    RED_LOOP(i, n) acc = fmax(acc, fabs(a[i]));
    sh[threadIdx.x] = acc;
    const double v = block_tree<1, RED_THREADS>(sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

// g /= max unless max < DBL_EPSILON (REAL_EPS guard, src/inversion.cpp:316)
__global__ void __launch_bounds__(RED_THREADS)
normalise_kernel(size_t n, const double* __restrict__ partial, double* g, double* out) {
    const double c = absmax_of(partial);
    if (blockIdx.x == 0 && threadIdx.x == 0) *out = c;
    if (c < 2.220446049250313e-16) return;
    RED_LOOP(i, n) g[i] = g[i] / c;
}

// One iterate's copy (m_out not null), and the pair with the iterate before
// (m0 not null): s = log m1 - log m0, y = g1 - g0, sy = sum s y, yy = sum y y.
__global__ void __launch_bounds__(RED_THREADS)
lbfgs_store_kernel(size_t n, const double* m1, const double* g1, double* m_out, double* g_out,
                   const double* m0, const double* g0, double* s, double* y, double* partial,
                   unsigned* count, LbfgsScalars* S, int slot) {
    double acc[2] = {0.0, 0.0}, res[2];
    RED_LOOP(i, n) {
        const double m = m1[i], g = g1[i];
        if (m_out) {
            m_out[i] = m;
            g_out[i] = g;
        }
        if (m0) {
            const double sv = log(m) - log(m0[i]);   // src/optimize.cpp:190-191 (log space)
            const double yv = g - g0[i];             // :197
            s[i] = sv;
            y[i] = yv;
            acc[0] += sv * yv;
            acc[1] += yv * yv;
        }
    }
    if (m0 && grid_sums(acc, partial, count, res) && threadIdx.x == 0) {
        S->sy[slot] = res[0];
        S->yy[slot] = res[1];
    }
}

// One pass of the two-loop recursion (src/optimize.cpp:209-236) over dir and
// the inner product that the next pass's coefficient needs:
//   kind 0: nothing, then alpha(next) = rho(next) x.dir      (dir = g, `from`)
//   kind 1: dir -= alpha(slot) x, then alpha(next) = rho(next) d.dir
//   kind 2: dir = gamma (dir - alpha(slot) x), then c(next) = alpha - beta
//   kind 3: dir += c(slot) x, then c(next); kind 4 without a next
// `from` is read in place of dir (the gradient, first pass).
__global__ void __launch_bounds__(RED_THREADS)
lbfgs_pass_kernel(size_t n, int kind, const double* from, const double* __restrict__ x,
                  const double* __restrict__ d, double* dir, double* partial, unsigned* count,
                  LbfgsScalars* S, int slot, int next) {
    cudaTriggerProgrammaticLaunchCompletion();   // (the next pass's blocks may come and wait)
    cudaGridDependencySynchronize();             // the pass before is complete
    double c = 0.0, gamma = 1.0;
    if (kind == 1 || kind == 2) c = S->alpha[slot];
    if (kind == 3 || kind == 4) c = S->c[slot];
    if (kind == 2) {
        const double sy = S->sy[next], yy = S->yy[next];   // of the last pair, :219-228
        gamma = (sy > 0.0 && yy > 0.0) ? (sy / yy) : 1.0;
    }
    double acc[1] = {0.0}, res[1];
    RED_LOOP(i, n) {
        double v = from[i];
        if (kind == 1) v = v - c * x[i];
        else if (kind == 2) v = gamma * (v - c * x[i]);
        else if (kind >= 3) v = v + c * x[i];
        if (kind != 0) dir[i] = v;
        if (d) acc[0] += d[i] * v;
    }
    if (!d) return;
    if (grid_sums(acc, partial, count, res) && threadIdx.x == 0) {
        // kind 2: the first pair's c (its y is x), else the next pair's
        const int p = kind == 2 ? slot : next;
        const double rho = S->sy[p] > 0.0 ? 1.0 / S->sy[p] : 0.0;   // :203
        const double t = rho * res[0];
        if (kind <= 1) S->alpha[p] = t;
        else S->c[p] = S->alpha[p] - t;
    }
}

__global__ void model_update_kernel(size_t n, const double* __restrict__ vs,
                                    const double* __restrict__ dir, double alpha, double* vs_out,
                                    double* vp_out, double* rho_out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const double v = vs[i] * (1 - alpha * dir[i]);   // src/inversion.cpp:471
        vs_out[i] = v;
        if (vp_out || rho_out) {
            const double vp = brocher_vs2vp(v);             // :478-479
            if (vp_out) vp_out[i] = vp;
            if (rho_out) rho_out[i] = brocher_vp2rho(vp);
        }
    }
}

// postproc::kernel_precondition (src/postproc.cpp:487-517): with L = max
// |ker_den| (of absmax_kernel's partials), ker *= 1 / (ker_den / L) where
// ker_den / L > VERYTINY (include/config.h:71), and nothing when L < VERYTINY.
__global__ void __launch_bounds__(RED_THREADS)
precondition_kernel(size_t n, const double* __restrict__ ker_den,
                    const double* __restrict__ partial, double* ker) {
    const double L = absmax_of(partial);
    if (L < 1e-12) return;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const double norm = ker_den[i] / L;
        const double h = norm > 1e-12 ? 1.0 / norm : 1.0;
        ker[i] = ker[i] * h;
    }
}

unsigned grid_for(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 148 * 16); }
}  // namespace

namespace {
// the blocks with an element (at least one): the others would add zeros
unsigned red_grid(size_t n) {
    return (unsigned)std::max<size_t>(1, std::min<size_t>(RED_BLOCKS, (n + RED_THREADS - 1) / RED_THREADS));
}
}  // namespace

// partial: red_blocks() doubles of the call's own
cudaError_t launch_kernel_precondition(size_t n, const double* ker_den, double* partial,
                                       double* ker, cudaStream_t st) {
    absmax_kernel<<<red_grid(n), RED_THREADS, 0, st>>>(n, ker_den, partial);
    precondition_kernel<<<red_grid(n), RED_THREADS, 0, st>>>(n, ker_den, partial, ker);
    return cudaGetLastError();
}

// scratch: the partials of 3 sums, the counter
size_t red_blocks() { return RED_BLOCKS; }
size_t reduce_scratch_doubles() { return 3 * RED_BLOCKS + 1; }
namespace {
unsigned* red_count(double* scratch) {
    return reinterpret_cast<unsigned*>(scratch + 3 * RED_BLOCKS);
}
}  // namespace

cudaError_t launch_dot(size_t n, const double* a, const double* b, double* scratch, double* out,
                       cudaStream_t st) {
    dot_kernel<1><<<red_grid(n), RED_THREADS, 0, st>>>(n, a, b, scratch, red_count(scratch), out);
    return cudaGetLastError();
}

cudaError_t launch_dots3(size_t n, const double* a, const double* b, double* scratch, double* out,
                         cudaStream_t st) {
    dot_kernel<3><<<red_grid(n), RED_THREADS, 0, st>>>(n, a, b, scratch, red_count(scratch), out);
    return cudaGetLastError();
}

cudaError_t launch_normalise(size_t n, double* g, double* scratch, double* out, cudaStream_t st) {
    absmax_kernel<<<red_grid(n), RED_THREADS, 0, st>>>(n, g, scratch);
    normalise_kernel<<<red_grid(n), RED_THREADS, 0, st>>>(n, scratch, g, out);
    return cudaGetLastError();
}

cudaError_t launch_lbfgs_store(size_t n, const double* m1, const double* g1, double* m_out,
                               double* g_out, const double* m0, const double* g0, double* s,
                               double* y, double* scratch, LbfgsScalars* S, int slot,
                               cudaStream_t st) {
    lbfgs_store_kernel<<<red_grid(n), RED_THREADS, 0, st>>>(n, m1, g1, m_out, g_out, m0, g0, s, y,
                                                           scratch, red_count(scratch), S, slot);
    return cudaGetLastError();
}

cudaError_t launch_lbfgs_pass(size_t n, int kind, const double* from, const double* x,
                              const double* d, double* dir, double* scratch, LbfgsScalars* S,
                              int slot, int next, cudaStream_t st) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(red_grid(n));
    cfg.blockDim = dim3(RED_THREADS);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, lbfgs_pass_kernel, n, kind, from, x, d, dir, scratch,
                              red_count(scratch), S, slot, next);
}

cudaError_t launch_model_update_vs(size_t n, const double* vs, const double* dir, double alpha,
                                   double* vs_out, double* vp_out, double* rho_out,
                                   cudaStream_t st) {
    model_update_kernel<<<grid_for(n), 256, 0, st>>>(n, vs, dir, alpha, vs_out, vp_out, rho_out);
    return cudaGetLastError();
}

}  // namespace sa
