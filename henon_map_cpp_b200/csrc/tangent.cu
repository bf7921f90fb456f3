// Tangent-map and indicator kernels with the reference's per-call semantics.
//
// These are the elementwise operations behind the drop-in classes
// matrix_4d_vector_gpu, vector_4d_gpu and the indicator "constructs"
// (src/henon.cu:267-359, 2042-2655).  Every arithmetic step is separately
// rounded in the reference's order, and the transcendental functions are
// CUDA's own log/log10/atan2/sqrt, so results are bit-identical to the
// reference CUDA build with --fmad=false.  The fused multi-turn kernel that
// replaces the per-turn Python loop over these calls lives in fused.cu.
#include <cuda_runtime.h>

#include <cstdint>

#include "hm_device.cuh"
#include "hm_internal.h"

namespace hm {
namespace {

using dev::Rn;

// One thread per particle.  The sets of the per-turn loop are small (a few
// thousand particles or fewer) and a call is then the latency of one thread:
// blocks are as small as it takes to give every SM one (1000 particles in
// blocks of 256 kept four SMs busy with 32-way split loads, 8.3 us a call for
// the matrix kernels), matrices and vectors move as 32-byte loads and
// stores, and the windows of a construct are dealt to the warps of a block.
// Back to back, us a call, before -> now:
//                         1,000        20,000       262,144 particles
//     matrix product    8.3 -> 5.2   8.3 -> 4.3   38.5 -> 15.5
//     MEGNO             8.3 -> 5.2   8.3 -> 4.3   33.2 -> 12.5
//     MEGNO, 13 windows 12.1 -> 5.6  12.4 -> 8.3  49.4 -> 24.7
//     Lyapunov, 13      10.4 -> 5.3  10.4 -> 8.4  21.1 -> 18.8
//     tunes, 13         10.4 -> 6.3  10.4 -> 8.4  24.5 -> 18.6
// (about 4-5 us is what a launch from Python costs here).
constexpr int kThreads = 256;

int block_threads(size_t n, int sms) {
    int t = 32;
    while (t < kThreads && size_t(t) * size_t(sms) < n) t *= 2;
    return t;
}

unsigned blocks_for(size_t n, int threads) { return unsigned((n + threads - 1) / threads); }

// v[0..3] from and to 32-byte aligned memory (sm_100's 256-bit accesses).
__device__ __forceinline__ void load4(const double *p, double *v) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p));
}

__device__ __forceinline__ void store4(double *p, const double *v) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
                 "d"(v[2]), "d"(v[3])
                 : "memory");
}

__device__ __forceinline__ void load16(const double *p, double (&m)[16]) {
#pragma unroll
    for (int r = 0; r < 4; ++r) load4(p + 4 * r, m + 4 * r);
}

__device__ __forceinline__ void store16(double *p, const double (&m)[16]) {
#pragma unroll
    for (int r = 0; r < 4; ++r) store4(p + 4 * r, m + 4 * r);
}

// M <- DF(x; table[idx]) * M, or M <- DF when set (get_matrices_and_multiply
// / get_matrices_and_set, src/henon.cu:267-313).
__global__ void matrices_step_kernel(double *M, const double *x, const double *y,
                                     const double *table, uint32_t idx, double mu, size_t n,
                                     int set) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double cur[16], out[16];
    if (!set) load16(M + i * 16, cur);
    const dev::Turn t = dev::load_turn(table, idx);
    double df[16];
    dev::tangent_matrix_exact(x[i], y[i], t, mu, df);
    if (set) {
        store16(M + i * 16, df);
        return;
    }
    dev::matmul4_exact(df, cur, out);
    store16(M + i * 16, out);
}

__global__ void matrices_identity_kernel(double *M, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n * 16) return;
    const int k = int(i % 16);
    M[i] = (k == 0 || k == 5 || k == 10 || k == 15) ? 1.0 : 0.0;
}

// out[i] = M[i] * rv[i] with each row summed left to right
// (matrix_4d_vector_gpu::get_vector, src/henon.cu:1892-1905).
__global__ void matrices_apply_kernel(const double *M, const double *rv, double *out, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *m = M + i * 16;
    const double *v = rv + i * 4;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        double s = Rn::mul(m[r * 4 + 0], v[0]);
        s = Rn::add(s, Rn::mul(m[r * 4 + 1], v[1]));
        s = Rn::add(s, Rn::mul(m[r * 4 + 2], v[2]));
        s = Rn::add(s, Rn::mul(m[r * 4 + 3], v[3]));
        out[i * 4 + r] = s;
    }
}

// v <- M v, rows summed from 0.0 (matrix_vector_multiply, :316-338).
__global__ void vectors_multiply_kernel(const double *M, double *V, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double m[16], v[4], t[4];
    load16(M + i * 16, m);
    load4(V + i * 4, v);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < 4; ++c) s = Rn::add(s, Rn::mul(m[r * 4 + c], v[c]));
        t[r] = s;
    }
    store4(V + i * 4, t);
}

// v <- v / |v| (normalize_vectors, :341-359).
__global__ void vectors_normalize_kernel(double *V, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v[4];
    load4(V + i * 4, v);
    const double norm = dev::norm_exact<4>(v);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = Rn::div(v[k], norm);
    store4(V + i * 4, v);
}

// The kernels with windows run blockDim.x particles on blockDim.y warps'
// worth of threads each: thread (x, y) updates windows y, y + blockDim.y,
// ... of particle x, kAhead of them at a time with their loads issued
// together.
constexpr int kAhead = 4;

// For every window w with idx < n_w: raw_w += log|v| / n_w and
// b_w += log|v| * weights_w[idx] (kernel_lyap_birk, :2083-2098; windows as
// lyapunov_birkhoff_construct_multi::add, :2171-2183).
__global__ void lyapunov_kernel(double *raw, double *bsum, const double *V, const double *weights,
                                const uint64_t *w_off, const uint64_t *w_len, int n_windows,
                                size_t idx, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v[4];
    load4(V + i * 4, v);
    const double l = log(dev::norm_exact<4>(v));
    const int step = int(blockDim.y);
    for (int w0 = int(threadIdx.y); w0 < n_windows; w0 += kAhead * step) {
        bool open[kAhead];
        double len[kAhead], wt[kAhead], r[kAhead], b[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int w = w0 + q * step;
            const uint64_t nw = w < n_windows ? w_len[w] : 0u;
            open[q] = idx < nw;
            len[q] = double(nw);
            if (!open[q]) continue;
            wt[q] = weights[w_off[w] + idx];
            r[q] = raw[size_t(w) * n + i];
            b[q] = bsum[size_t(w) * n + i];
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            if (!open[q]) continue;
            const size_t o = size_t(w0 + q * step) * n + i;
            raw[o] = Rn::add(r[q], Rn::div(l, len[q]));
            bsum[o] = Rn::add(b[q], Rn::mul(l, wt[q]));
        }
    }
}

// MEGNO layers from the Frobenius norms of A (new) and B (old)
// (kernel_megno, :2253-2284).
__global__ void megno_kernel(double *l1, double *l2, double *l3, const double *A, const double *B,
                             size_t idx, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a[16], b[16];
    load16(A + i * 16, a);
    load16(B + i * 16, b);
    const double ta = dev::norm_exact<16>(a);
    const double tb = dev::norm_exact<16>(b);
    const double di = double(idx);
    const double a1 = Rn::add(l1[i], Rn::mul(log10(Rn::div(ta, tb)), di));
    const double a2 = Rn::add(l2[i], Rn::mul(Rn::div(1.0, di), a1));
    l1[i] = a1;
    l2[i] = a2;
    l3[i] = Rn::mul(Rn::div(1.0, di), a2);
}

// Birkhoff-weighted MEGNO per window (kernel_megno_birkhoff, :2366-2402).
__global__ void megno_birkhoff_kernel(double *l1, double *l2, const double *weights,
                                      const uint64_t *w_off, const uint64_t *T, int n_windows,
                                      const double *A, const double *B, size_t idx, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool in = i < n;
    double a1 = 0.0;
    const double di = double(idx);
    if (in) {
        double a[16], b[16];
        load16(A + i * 16, a);
        load16(B + i * 16, b);
        const double ta = dev::norm_exact<16>(a);
        const double tb = dev::norm_exact<16>(b);
        a1 = Rn::add(l1[i], Rn::mul(log10(Rn::div(ta, tb)), di));
    }
    // every thread of the particle has read l1
    if (blockDim.y > 1u) __syncthreads();
    if (!in) return;
    if (threadIdx.y == 0u) l1[i] = a1;
    const int step = int(blockDim.y);
    for (int w0 = int(threadIdx.y); w0 < n_windows; w0 += kAhead * step) {
        bool open[kAhead];
        double wt[kAhead], acc[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int w = w0 + q * step;
            open[q] = w < n_windows && idx <= T[w];
            if (!open[q]) continue;
            wt[q] = weights[w_off[w] + idx - 1];
            acc[q] = l2[size_t(w) * n + i];
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (open[q])
                l2[size_t(w0 + q * step) * n + i] =
                    Rn::add(acc[q], Rn::div(Rn::mul(a1, wt[q]), di));
    }
}

// First angles (kernel_tune_birkhoff_init, :2533-2546).
__global__ void tune_init_kernel(const double *x, const double *px, const double *y,
                                 const double *py, double *store_x, double *store_y, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    store_x[i] = atan2(px[i], x[i]);
    store_y[i] = atan2(py[i], y[i]);
}

// Phase advance wrapped to (0, 2pi], weighted into window 1 [0, T) or
// window 2 [T, 2T) (kernel_tune_birkhoff, :2548-2584).
__global__ void tune_add_kernel(const double *x, const double *px, const double *y,
                                const double *py, double *store_x, double *store_y, double *t1x,
                                double *t1y, double *t2x, double *t2y, const double *weights,
                                const uint64_t *w_off, const uint64_t *T, int n_windows,
                                size_t idx, size_t n) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool in = i < n;
    double ax = 0.0, ay = 0.0, dx = 0.0, dy = 0.0;
    if (in) {
        ax = atan2(px[i], x[i]);
        ay = atan2(py[i], y[i]);
        dx = Rn::sub(ax, store_x[i]);
        dy = Rn::sub(ay, store_y[i]);
        const double two_pi = 2 * M_PI;
        dx = dx > 0 ? dx : Rn::add(dx, two_pi);
        dy = dy > 0 ? dy : Rn::add(dy, two_pi);
    }
    // every thread of the particle has read the angles before
    if (blockDim.y > 1u) __syncthreads();
    if (!in) return;
    if (threadIdx.y == 0u) {
        store_x[i] = ax;
        store_y[i] = ay;
    }
    const int step = int(blockDim.y);
    for (int w0 = int(threadIdx.y); w0 < n_windows; w0 += kAhead * step) {
        double *tx[kAhead], *ty[kAhead];
        double wt[kAhead], vx[kAhead], vy[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int w = w0 + q * step;
            const uint64_t len = w < n_windows ? T[w] : 0u;
            tx[q] = nullptr;
            if (idx >= 2 * len) continue;
            const size_t o = size_t(w) * n + i;
            tx[q] = (idx < len ? t1x : t2x) + o;
            ty[q] = (idx < len ? t1y : t2y) + o;
            wt[q] = weights[w_off[w] + (idx < len ? idx : idx - len)];
            vx[q] = *tx[q];
            vy[q] = *ty[q];
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q)
            if (tx[q]) {
                *tx[q] = Rn::add(vx[q], Rn::mul(dx, wt[q]));
                *ty[q] = Rn::add(vy[q], Rn::mul(dy, wt[q]));
            }
    }
}

// Block of a kernel with windows: up to kThreads threads, the rows past the
// first dealing with further windows while the set is small (a large one
// keeps the device busy with one thread per particle, which then computes
// the logarithm or the angles once).
dim3 window_block(size_t n, int n_windows, int sms) {
    const int t = block_threads(n, sms);
    int rows = 1;
    while (rows < 8 && rows * kAhead < n_windows && t * rows * 2 <= kThreads &&
           size_t(rows) * 2u * n <= size_t(sms) * 1024u)
        rows *= 2;
    return dim3(unsigned(t), unsigned(rows));
}

}  // namespace

cudaError_t launch_matrices_step(double *M, const double *x, const double *y, const double *table,
                                 uint32_t idx, double mu, size_t n, bool set, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int t = block_threads(n, sm_count());
    matrices_step_kernel<<<blocks_for(n, t), t, 0, s>>>(M, x, y, table, idx, mu, n, set ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_matrices_identity(double *M, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    matrices_identity_kernel<<<blocks_for(n * 16, kThreads), kThreads, 0, s>>>(M, n);
    return cudaGetLastError();
}

cudaError_t launch_matrices_apply(const double *M, const double *rv, double *out, size_t n,
                                  cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int t = block_threads(n, sm_count());
    matrices_apply_kernel<<<blocks_for(n, t), t, 0, s>>>(M, rv, out, n);
    return cudaGetLastError();
}

cudaError_t launch_vectors_multiply(const double *M, double *V, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int t = block_threads(n, sm_count());
    vectors_multiply_kernel<<<blocks_for(n, t), t, 0, s>>>(M, V, n);
    return cudaGetLastError();
}

cudaError_t launch_vectors_normalize(double *V, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int t = block_threads(n, sm_count());
    vectors_normalize_kernel<<<blocks_for(n, t), t, 0, s>>>(V, n);
    return cudaGetLastError();
}

cudaError_t launch_lyapunov(double *raw, double *bsum, const double *V, const double *weights,
                            const uint64_t *w_off, const uint64_t *w_len, int n_windows,
                            size_t idx, size_t n, cudaStream_t s) {
    if (n == 0 || n_windows == 0) return cudaSuccess;
    const dim3 b = window_block(n, n_windows, sm_count());
    lyapunov_kernel<<<blocks_for(n, int(b.x)), b, 0, s>>>(raw, bsum, V, weights, w_off, w_len,
                                                          n_windows, idx, n);
    return cudaGetLastError();
}

cudaError_t launch_megno(double *l1, double *l2, double *l3, const double *A, const double *B,
                         size_t idx, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int t = block_threads(n, sm_count());
    megno_kernel<<<blocks_for(n, t), t, 0, s>>>(l1, l2, l3, A, B, idx, n);
    return cudaGetLastError();
}

cudaError_t launch_megno_birkhoff(double *l1, double *l2, const double *weights,
                                  const uint64_t *w_off, const uint64_t *T, int n_windows,
                                  const double *A, const double *B, size_t idx, size_t n,
                                  cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const dim3 b = window_block(n, n_windows, sm_count());
    megno_birkhoff_kernel<<<blocks_for(n, int(b.x)), b, 0, s>>>(l1, l2, weights, w_off, T,
                                                                n_windows, A, B, idx, n);
    return cudaGetLastError();
}

cudaError_t launch_tune_init(const double *x, const double *px, const double *y, const double *py,
                             double *store_x, double *store_y, size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int t = block_threads(n, sm_count());
    tune_init_kernel<<<blocks_for(n, t), t, 0, s>>>(x, px, y, py, store_x, store_y, n);
    return cudaGetLastError();
}

cudaError_t launch_tune_add(const double *x, const double *px, const double *y, const double *py,
                            double *store_x, double *store_y, double *t1x, double *t1y,
                            double *t2x, double *t2y, const double *weights,
                            const uint64_t *w_off, const uint64_t *T, int n_windows, size_t idx,
                            size_t n, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const dim3 b = window_block(n, n_windows, sm_count());
    tune_add_kernel<<<blocks_for(n, int(b.x)), b, 0, s>>>(x, px, y, py, store_x, store_y, t1x,
                                                          t1y, t2x, t2y, weights, w_off, T,
                                                          n_windows, idx, n);
    return cudaGetLastError();
}

}  // namespace hm
