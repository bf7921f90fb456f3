// Tune estimates from turn-by-turn orbits (sm_100a).
//
// Orbits the caller stored (storage tunes) hold S snapshots of n particles
// per coordinate, laid out [sample][particle] (storage_4d_gpu's layout), so
// a warp reads 32 particles of one sample in one coalesced access:
// * mean_remove_kernel: subtracts each coordinate's orbit mean
//   (src/henon.cu:3040-3051);
// * birkhoff_kernel: Birkhoff-weighted phase advance over sample windows
//   (birkhoff_tune / birkhoff_tune_vec, src/dynamic_indicator.cpp:81-131,
//   198-253);
// * hann_gather_kernel + cuFFT + fft_peak_kernel: Hann-windowed spectrum of
//   x + i px and the interpolated peak (compute_fft, interpolation, A,
//   fft_tune_vec, src/dynamic_indicator.cpp:32-61, 134-196, 255-330).
// The tracker's own tune path (birkhoff_tunes / all_tunes,
// src/henon.cu:2890-3078) records the orbit itself, particle-major
// ([particle][sample] per coordinate: each particle's samples contiguous),
// with each coordinate's running sum and the first NaN sample, and then
// never rewrites it; the mean is subtracted as samples are read:
// * orbit_record_kernel: tracks n_turns turns and writes every state
//   (sample 0 = the start);
// * birkhoff_seg_kernel / birkhoff_finish_kernel: Birkhoff sums in segments
//   of turns over many threads;
// * fft_tune_kernel: one window's spectrum computed whole in one block's
//   shared memory, and its peak; windows too long for one block take
//   fft_gather2_kernel + cuFFT + fft_peak2_kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "hm_device.cuh"
#include "hm_internal.h"

namespace hm {
namespace {

using dev::Rn;

// Tracks n_turns turns and writes every state (sample 0 = the start).  The
// turn is the tracker's: forward with table[live_step + k], or backward with
// table[live_step - 1 - k] (REV), with the tracker's reproducible kicks
// (KICK: added before the forward turn, subtracted after the backward
// one).  Also each coordinate's sum over the samples (from 0.0, in sample
// order: the reference's std::accumulate for all_tunes' mean,
// src/henon.cu:3040-3051) and the first NaN sample.
//
// A tune call has few particles (16,384 are 3.5 warps per SM) and each orbit
// is one serial chain of turns, so the time is that of one warp's turns.
// Two warps share the work of 32 particles: the first runs the turns in
// groups of 16 samples without per-turn control flow (dev::block_turns'
// scheme, with a redo of the group where a coordinate was large) and puts
// each sample into shared memory; the second writes the group before to the
// orbit as whole 128-byte lines (the orbit is particle-major, so a warp's
// samples of one turn would land in 32 different rows) and brings in the
// turn records of the group after next.  One block barrier per group.
// 16,384 particles x 1e4 turns: 3.39 ms with one warp doing all of it and
// testing every turn (528 cycles a turn), 1.32 ms now, bound by the 5.2 GB
// that it writes (0.62 ms with 2,048 particles).
// Lanes past the last particle run the loop on zeros (a fixed point) and
// write nothing.
constexpr uint32_t kRecGroup = dev::kBlockTurns;
constexpr uint32_t kRecRow = kRecGroup + 1u;  // a lane's samples, padded for the banks
constexpr uint32_t kRecBuf = 4u * 32u * kRecRow;  // doubles of a group: [coordinate][lane][sample]

template <int ARITH, bool OCT, bool REV, bool KICK>
__global__ void __launch_bounds__(64) orbit_record_kernel(OrbitRecordArgs a) {
    __shared__ __align__(16) double samples[2][kRecBuf];
    __shared__ __align__(16) double2 recs[2][2u * kRecGroup];
    const unsigned lane = threadIdx.x & 31u;
    const size_t first = size_t(blockIdx.x) * 32u, i = first + lane;
    const size_t n = a.n, S = size_t(a.n_turns) + 1u;
    const bool valid = i < n;
    const uint32_t groups = uint32_t((S + kRecGroup - 1u) / kRecGroup);
    constexpr uint32_t G = kRecGroup, W = kRecRow;

    if (threadIdx.x >= 32u) {
        // ---- the writing warp ------------------------------------------------
        // Lane l brings in half l & 1 of the record of the group's turn l / 2
        // (zeros past the last turn, which no turn reads).
        auto fetch = [&](uint32_t g) {
            const uint32_t k = g * G + (lane >> 1);
            if (k >= a.n_turns) return make_double2(0.0, 0.0);
            const uint32_t idx = REV ? a.live_step - 1u - k : a.live_step + k;
            return __ldg(reinterpret_cast<const double2 *>(a.table) + 2u * size_t(idx) +
                         (lane & 1u));
        };
        recs[0][lane] = fetch(0u);
        recs[1][lane] = fetch(1u);
        __syncthreads();
        double2 next = fetch(2u);
        for (uint32_t g = 0; g < groups; ++g) {
            __syncthreads();  // group g is complete, its records are used
            recs[g & 1u][lane] = next;
            next = fetch(g + 3u);
            const double *st = samples[g & 1u];
            const uint32_t base = g * G, cnt = uint32_t(S - base < G ? S - base : G);
            // lanes 0-15 one particle's samples, lanes 16-31 the next one's
            const uint32_t gg = lane % G;
            size_t o = (first + lane / G) * a.pitch + base + gg;
            const double *src = st + (lane / G) * W + gg;
            if (gg < cnt)
#pragma unroll 4
                for (uint32_t pl = lane / G; pl < 32u && first + pl < n;
                     pl += 32u / G, o += (32u / G) * a.pitch, src += (32u / G) * W) {
                    a.ox[o] = src[0];
                    a.opx[o] = src[32u * W];
                    a.oy[o] = src[2u * 32u * W];
                    a.opy[o] = src[3u * 32u * W];
                }
        }
        return;
    }

    // ---- the tracking warp ---------------------------------------------------
    double x = 0.0, px = 0.0, y = 0.0, py = 0.0;  // what a lost lane records
    uint32_t steps = 0;
    if (valid) {
        x = a.x[i];
        px = a.px[i];
        y = a.y[i];
        py = a.py[i];
        steps = a.steps[i];
    }
    bool alive = valid && !dev::is_lost(x, px, y, py);
    uint32_t first_nan = alive ? a.n_turns + 1u : 0u;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    dev::Particle p[1] = {alive ? dev::make_particle(x, px, y, py)
                                : dev::make_particle(0.0, 0.0, 0.0, 0.0)};
    const dev::Barrier bar = dev::make_barrier<ARITH>(a.b2bits);
    const double mu = a.mu;
    __syncthreads();
    for (uint32_t g = 0; g < groups; ++g) {
        const uint32_t k0 = g * G;
        const uint32_t cnt = uint32_t(S - k0 < G ? S - k0 : G);  // samples of the group
        double *const st = samples[g & 1u] + lane * W;
        const double2 *const q = recs[g & 1u];
        auto put = [&](uint32_t u, double v0, double v1, double v2, double v3) {
            st[u] = v0;
            st[32u * W + u] = v1;
            st[2u * 32u * W + u] = v2;
            st[3u * 32u * W + u] = v3;
            s0 = Rn::add(s0, v0);
            s1 = Rn::add(s1, v1);
            s2 = Rn::add(s2, v2);
            s3 = Rn::add(s3, v3);
        };
        const dev::Particle from = p[0];
        const double f0 = s0, f1 = s1, f2 = s2, f3 = s3;
        // Each sample is the state before its turn.
        const bool whole = !KICK && k0 + G <= a.n_turns && a.pair_hi != 0u;
        bool redo = !whole;
        if (whole) {
            float big = 0.0f;
#pragma unroll
            for (uint32_t u = 0; u < G; ++u) {
                put(u, p[0].x, p[0].px, p[0].y, p[0].py);
                const double2 r = q[2u * u], t = q[2u * u + 1u];
                dev::turn<ARITH, OCT, REV>(p[0], dev::Turn{r.x, r.y, t.x, t.y}, mu);
                if (u & 1u)
                    big = dev::hi_max(dev::hi_max(big, p[0].x, p[0].px), p[0].y, p[0].py);
            }
            redo = __any_sync(dev::kFullMask,
                              (__float_as_uint(big) & 0x7fffffffu) >= a.pair_hi);
            // A lane lost before this group ran it on zeros; what it records
            // stays as it was.
            if (!redo && !alive) {
                s0 = f0;
                s1 = f1;
                s2 = f2;
                s3 = f3;
                for (uint32_t u = 0; u < G; ++u) put(u, x, px, y, py);
            }
            if (!redo && alive) steps = REV ? steps - G : steps + G;
        }
        if (redo) {  // the group turn by turn
            p[0] = from;
            s0 = f0;
            s1 = f1;
            s2 = f2;
            s3 = f3;
            for (uint32_t u = 0; u < cnt; ++u) {
                if (alive) put(u, p[0].x, p[0].px, p[0].y, p[0].py);
                else put(u, x, px, y, py);
                const uint32_t k = k0 + u;
                if (k >= a.n_turns || !alive) continue;
                const double2 r = q[2u * u], t = q[2u * u + 1u];
                const uint32_t idx = REV ? a.live_step - 1u - k : a.live_step + k;
                if (KICK && !REV)
                    dev::apply_kick<false>(p[0], dev::kick_direction(a.kick_seed, a.id0 + i, idx),
                                           a.kick_module);
                dev::turn<ARITH, OCT, REV>(p[0], dev::Turn{r.x, r.y, t.x, t.y}, mu);
                if (KICK && REV)
                    dev::apply_kick<true>(p[0], dev::kick_direction(a.kick_seed, a.id0 + i, idx),
                                          a.kick_module);
                if (dev::inside_after_turn<ARITH>(p[0], bar)) {
                    steps = REV ? steps - 1u : steps + 1u;
                } else {
                    x = px = y = py = dev::quiet_nan();
                    alive = false;
                    first_nan = k + 1u;
                    p[0] = dev::make_particle(0.0, 0.0, 0.0, 0.0);
                }
            }
        }
        __syncthreads();
    }
    if (!valid) return;
    a.x[i] = alive ? p[0].x : x;
    a.px[i] = alive ? p[0].px : px;
    a.y[i] = alive ? p[0].y : y;
    a.py[i] = alive ? p[0].py : py;
    a.steps[i] = steps;
    if (a.sums) {
        a.sums[i] = s0;
        a.sums[n + i] = s1;
        a.sums[2 * n + i] = s2;
        a.sums[3 * n + i] = s3;
        // With the mean removed, one NaN sample makes the mean, and so every
        // sample, NaN.
        if (first_nan <= a.n_turns) first_nan = 0u;
    }
    if (a.first_nan) a.first_nan[i] = first_nan;
}

__device__ double interp_a(double a, double b, double c);

// mean = sum / samples, as the reference divides std::accumulate's result.
__device__ __forceinline__ double mean_of(const double *means, size_t n, size_t i, int c,
                                          size_t S) {
    return means ? Rn::div(means[size_t(c) * n + i], double(S)) : 0.0;
}

// v - mean, separately rounded (the reference subtracts the mean from every
// stored sample); without a mean the sample itself.
__device__ __forceinline__ double centred(double v, const double *means, double m) {
    return means ? Rn::sub(v, m) : v;
}

// Four consecutive samples as one 32-byte load (sm_100; p 32-byte aligned).
__device__ __forceinline__ void load4(const double *p, double (&v)[4]) {
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
        : "l"(p));
}

// Birkhoff phase-advance sums of one segment for one plane of one particle,
// every window at once: the transition s -> s+1 adds w_j[s - from_j] dtheta_s
// to window j when from_j <= s < to_j, dtheta wrapped by +2 pi when negative
// (birkhoff_tune, src/dynamic_indicator.cpp:81-131).  A segment holds the
// transitions into its samples [g seg_len, (g + 1) seg_len), seg_len a
// multiple of 4.  Windows in groups of kWinGroup (blockIdx.y) so that the
// sums stay in registers.
//
// Samples are taken four at a time: neighbouring threads read rows of
// `pitch` doubles, so an 8-byte load of a warp costs 32 tag look-ups for 256
// bytes, and this way a quarter of them.  A window that holds all four
// transitions, or none, is told by one test instead of four.  16,384
// particles x 1e4 turns, 4 windows and the full orbit: 2.74 ms, bound by the
// instructions of atan2 (sample by sample, each window tested each time:
// 4.47 ms; 3.85 once the rows were aligned).
constexpr int kWinGroup = 8;

__global__ void __launch_bounds__(128, 5) birkhoff_seg_kernel(const BirkhoffSegArgs a) {
    // The block's windows: the samples that the first and last of its
    // transitions lead to, and the weight of a transition into sample s, w[s].
    struct Window {
        uint32_t first, last;
        const double *w;
    };
    __shared__ Window win[kWinGroup];
    const int w0 = int(blockIdx.y) * kWinGroup;
    const int nw = min(kWinGroup, a.n_win - w0);
    if (int(threadIdx.x) < nw) {
        const uint32_t from = a.from[w0 + threadIdx.x];
        win[threadIdx.x] = Window{from + 1u, a.to[w0 + threadIdx.x],
                                  a.w + ((long long)a.w_off[w0 + threadIdx.x] - (long long)from - 1)};
    }
    __syncthreads();
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t n = a.n;
    const size_t sp = t / n;  // segment * 2 + plane
    if (sp >= 2u * size_t(a.n_seg)) return;
    const size_t i = t - sp * n;
    const uint32_t seg = uint32_t(sp >> 1);
    const int plane = int(sp & 1u);
    const double mq = mean_of(a.means, n, i, 2 * plane, a.S);
    const double mp = mean_of(a.means, n, i, 2 * plane + 1, a.S);
    double acc[kWinGroup] = {};
    const double *const q = (plane ? a.y : a.x) + i * a.pitch;  // this particle's samples
    const double *const p = (plane ? a.py : a.px) + i * a.pitch;
    const uint32_t b0 = seg * a.seg_len;
    const uint32_t b1 = uint32_t(a.S - b0 < a.seg_len ? a.S : size_t(b0) + a.seg_len);
    double prev = 0.0;
    if (b0 > 0u) prev = atan2(centred(p[b0 - 1u], a.means, mp), centred(q[b0 - 1u], a.means, mq));
    // The row's padding is readable past sample S - 1; no window holds a
    // transition into it.
    for (uint32_t b = b0; b < b1; b += 4u) {
        double qv[4], pv[4], d[4];
        load4(q + b, qv);
        load4(p + b, pv);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double th = atan2(centred(pv[u], a.means, mp), centred(qv[u], a.means, mq));
            d[u] = Rn::sub(th, prev);
            if (d[u] < 0.0) d[u] = Rn::add(d[u], 2.0 * M_PI);
            prev = th;
        }
#pragma unroll
        for (int j = 0; j < kWinGroup; ++j) {
            if (j >= nw) break;
            const Window v = win[j];
            if (b > v.last || b + 3u < v.first) continue;
            if (b >= v.first && b + 3u <= v.last) {
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[j] = Rn::add(acc[j], Rn::mul(v.w[b + u], d[u]));
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (b + u >= v.first && b + u <= v.last)
                        acc[j] = Rn::add(acc[j], Rn::mul(v.w[b + u], d[u]));
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kWinGroup; ++j)
        if (j < nw)
            a.partial[((size_t(w0 + j) * 2 + plane) * a.n_seg + seg) * n + i] = acc[j];
}

// 1 - (sum of the segments' sums, in segment order) / (2 pi); NaN for a
// window marked check_nan that holds a NaN sample (birkhoff_tune_vec checks
// the caller's windows, not the appended full orbit).
__global__ void birkhoff_finish_kernel(const BirkhoffSegArgs a) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t n = a.n;
    const size_t wp = t / n;  // window * 2 + plane
    if (wp >= 2u * size_t(a.n_win)) return;
    const size_t i = t - wp * n;
    const int j = int(wp >> 1), plane = int(wp & 1u);
    const double *part = a.partial + (size_t(j) * 2 + plane) * a.n_seg * n + i;
    double sum = 0.0;
    for (uint32_t g = 0; g < a.n_seg; ++g) sum = Rn::add(sum, part[size_t(g) * n]);
    double tune = Rn::sub(1.0, Rn::div(sum, Rn::mul(2.0, M_PI)));
    if (a.check_nan[j] && a.first_nan[i] <= a.to[j]) tune = dev::quiet_nan();
    a.out[i * a.cols + 2 * size_t(a.out_col[j]) + plane] = tune;
}

// Hann window 2 sin^2(pi k / len) (compute_fft, src/dynamic_indicator.cpp:
// 32-61), the same expression as hann_gather_kernel's.
__global__ void hann_table_kernel(double *h, uint32_t len) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= len) return;
    const double s = sin(M_PI * double(k) / double(len));
    h[k] = 2 * pow(s, 2);
}

// z[plane n + i][k] = ((q - mean) + i (p - mean)) h_k over the window's
// samples from .. from + len - 1: one row of len values per column (plane,
// particle), cuFFT's native batch layout.  The orbit's samples are
// contiguous per particle, so rows are read and written along samples.
__global__ void __launch_bounds__(256) fft_gather2_kernel(const double *x, const double *px,
                                                          const double *y, const double *py,
                                                          const double *means, size_t n,
                                                          uint32_t from, uint32_t len,
                                                          const double *h, double2 *z, size_t S,
                                                          size_t pitch, int plane) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n * len) return;
    const size_t i = t / len;
    const uint32_t k = uint32_t(t - i * len);
    const double *q = plane ? y : x, *p = plane ? py : px;
    const double mq = mean_of(means, n, i, 2 * plane, S);
    const double mp = mean_of(means, n, i, 2 * plane + 1, S);
    const size_t o = i * pitch + from + k;
    const double re = centred(q[o], means, mq), im = centred(p[o], means, mp);
    const double hk = h[k];
    z[(size_t(plane) * n + i) * len + k] = make_double2(re * hk, im * hk);
}

// One warp per column (plane, particle): first maximum of |z_k| over k
// (lanes stride the row, then a shuffle reduction keeping the smallest k
// among equal maxima), then the interpolation of
// src/dynamic_indicator.cpp:139-176 -> |1 - v|; NaN when the window's
// samples from .. last_sample hold a NaN.
__global__ void fft_peak2_kernel(const double2 *z, uint32_t len, size_t n, uint32_t last_sample,
                                 const uint32_t *first_nan, double *out, size_t out_cols,
                                 int col) {
    const size_t c = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
    const unsigned lane = threadIdx.x & 31u;
    if (c >= 2 * n) return;
    const int plane = c >= n ? 1 : 0;
    const size_t i = c - size_t(plane) * n;
    const double2 *row = z + c * len;
    auto mag = [&](uint32_t k) {
        const double2 v = row[k];
        return sqrt(v.x * v.x + v.y * v.y);
    };
    const bool nan = first_nan[i] <= last_sample;
    double best = -1.0;
    uint32_t best_k = 0xffffffffu;
    if (!nan) {
        for (uint32_t k = lane; k < len; k += 32) {
            const double m = mag(k);
            if (m > best) {  // k grows within a lane: the first maximum is kept
                best = m;
                best_k = k;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_down_sync(dev::kFullMask, best, o);
        const uint32_t ok = __shfl_down_sync(dev::kFullMask, best_k, o);
        if (ob > best || (ob == best && ok < best_k)) {
            best = ob;
            best_k = ok;
        }
    }
    if (lane != 0) return;
    double value;
    if (nan) {
        value = dev::quiet_nan();
    } else {
        uint32_t index = best_k;
        const double N = double(len);
        if (index == 0) {
            value = 1.0;
        } else if (index == len - 1) {
            value = 0.0;
        } else {
            uint32_t i1, i2;
            if (mag(index - 1) > mag(index + 1)) {
                i1 = index - 1;
                i2 = index;
                index = index - 1;
            } else {
                i1 = index;
                i2 = index + 1;
            }
            const double v = (double(index) / N) +
                             (1.0 / (2.0 * M_PI)) *
                                 asin(interp_a(mag(i1), mag(i2), cos(2.0 * M_PI / N)) *
                                      sin(2.0 * M_PI / N));
            value = fabs(1.0 - v);
        }
    }
    out[i * out_cols + 2 * size_t(col) + plane] = value;
}

// v -= mean(v) per particle and coordinate, one thread per (coordinate,
// particle), particles fastest; the mean is the left-to-right sum from 0.0
// divided by the sample count (std::accumulate / size).
__global__ void mean_remove_kernel(double *x, double *px, double *y, double *py, size_t n,
                                   size_t S) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t q = t / n;  // coordinate
    if (q >= 4u) return;
    const size_t i = t - q * n;
    double *c = q == 0u ? x : q == 1u ? px : q == 2u ? y : py;
    double s = 0.0;
#pragma unroll 8
    for (size_t k = 0; k < S; ++k) s = Rn::add(s, c[k * n + i]);
    const double m = Rn::div(s, double(S));
#pragma unroll 8
    for (size_t k = 0; k < S; ++k) c[k * n + i] = Rn::sub(c[k * n + i], m);
}

// Birkhoff tune over samples [from, to] of (q, p): 1 - sum_i w_i dtheta_i /
// (2 pi), dtheta wrapped by +2pi when negative, w = birkhoff_weights(to -
// from); NaN when check_nan and any sample of the window is NaN.
// Birkhoff tune of one plane over samples [from, to] of particle i; *has_nan
// reports a NaN in any of the four coordinates of the window (q, p of this
// plane and o1, o2 of the other).  The sample loads do not depend on the
// running sum, so the loop is unrolled to keep several in flight.
__device__ double birkhoff_window(const double *q, const double *p, const double *o1,
                                  const double *o2, size_t n, size_t i, uint32_t from,
                                  uint32_t to, const double *w, bool *has_nan) {
    double sum = 0.0;
    bool nan_seen = false;
    const size_t f = size_t(from) * n + i;
    double prev = atan2(p[f], q[f]);
    nan_seen |= isnan(q[f]) || isnan(p[f]) || isnan(o1[f]) || isnan(o2[f]);
#pragma unroll 4
    for (uint32_t s = from; s < to; ++s) {
        const size_t o = size_t(s + 1) * n + i;
        const double qq = q[o], pp = p[o];
        nan_seen |= isnan(qq) || isnan(pp) || isnan(o1[o]) || isnan(o2[o]);
        const double th = atan2(pp, qq);
        double d = Rn::sub(th, prev);
        if (d < 0.0) d = Rn::add(d, 2.0 * M_PI);
        sum = Rn::add(sum, Rn::mul(w[s - from], d));
        prev = th;
    }
    *has_nan = nan_seen;
    return Rn::sub(1.0, Rn::div(sum, Rn::mul(2.0, M_PI)));
}

// One thread per (window, plane, particle), particles fastest: a warp
// walks one window of one plane for 32 consecutive particles (coalesced
// loads, no divergence between windows of different lengths), and for few
// particles the windows and planes supply the parallelism.
__global__ void birkhoff_kernel(const double *x, const double *px, const double *y,
                                const double *py, size_t n, const uint32_t *from,
                                const uint32_t *to, const uint64_t *w_off, const double *w,
                                int n_win, double *out) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t wp = t / n;  // window * 2 + plane
    if (wp >= 2u * size_t(n_win)) return;
    const size_t i = t - wp * n;
    const int j = int(wp >> 1);
    const bool plane_y = (wp & 1u) != 0u;
    bool nan_seen = false;
    double tune = plane_y ? birkhoff_window(y, py, x, px, n, i, from[j], to[j], w + w_off[j], &nan_seen)
                          : birkhoff_window(x, px, y, py, n, i, from[j], to[j], w + w_off[j], &nan_seen);
    // birkhoff_tune_vec checks all four coordinates of the window for the
    // windows it was given, not for the appended full orbit.
    const bool is_full = j == n_win - 1;
    if (!is_full && nan_seen) tune = dev::quiet_nan();
    out[i * size_t(2 * n_win) + 2 * size_t(j) + (plane_y ? 1u : 0u)] = tune;
}

// z_k = (x + i px)[from + k] * 2 sin^2(pi k / len) for one window, one row
// of len complex values per particle; nan_flags[i] set when any sample of
// the window is NaN.
__global__ void hann_gather_kernel(const double *q, const double *p, size_t n, uint32_t from,
                                   uint32_t len, size_t first, size_t count, double2 *buf,
                                   int *nan_flags) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= count * len) return;
    const size_t r = t / len, k = t % len;
    const size_t i = first + r;
    const double re = q[size_t(from + k) * n + i], im = p[size_t(from + k) * n + i];
    if (isnan(re) || isnan(im)) nan_flags[r] = 1;
    const double s = sin(M_PI * double(k) / double(len));
    const double h = 2 * pow(s, 2);
    buf[r * len + k] = make_double2(re * h, im * h);
}

// A(a, b, c) of the peak interpolation (src/dynamic_indicator.cpp:134-137).
__device__ double interp_a(double a, double b, double c) {
    return (-(a + b * c) * (a - b) +
            b * sqrt(pow(c, 2) * pow((a + b), 2) - 2 * a * b * (2 * pow(c, 2) - c - 1))) /
           (pow(a, 2) + pow(b, 2) + 2 * a * b * c);
}

// One warp per particle: argmax of |FFT| (first maximum), then the
// interpolation of src/dynamic_indicator.cpp:139-176 -> |1 - value|.
__global__ void fft_peak_kernel(const double2 *buf, uint32_t len, size_t count,
                                const int *nan_flags, double *out, size_t out_stride,
                                size_t first) {
    const size_t warp = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
    const unsigned lane = threadIdx.x & 31u;
    if (warp >= count) return;
    const double2 *row = buf + warp * len;
    double best = -1.0;
    uint32_t best_k = 0xffffffffu;
    for (uint32_t k = lane; k < len; k += 32) {
        const double2 z = row[k];
        const double m = sqrt(z.x * z.x + z.y * z.y);
        if (m > best || (m == best && k < best_k)) {
            best = m;
            best_k = k;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_down_sync(dev::kFullMask, best, o);
        const uint32_t ok = __shfl_down_sync(dev::kFullMask, best_k, o);
        if (ob > best || (ob == best && ok < best_k)) {
            best = ob;
            best_k = ok;
        }
    }
    if (lane != 0) return;
    double value;
    if (nan_flags[warp]) {
        value = dev::quiet_nan();
    } else {
        uint32_t index = best_k;
        const double N = double(len);
        auto mag = [&](uint32_t k) {
            const double2 z = row[k];
            return sqrt(z.x * z.x + z.y * z.y);
        };
        if (index == 0) {
            value = 1.0;
        } else if (index == len - 1) {
            value = 0.0;
        } else {
            uint32_t i1, i2;
            if (mag(index - 1) > mag(index + 1)) {
                i1 = index - 1;
                i2 = index;
                index = index - 1;
            } else {
                i1 = index;
                i2 = index + 1;
            }
            const double v = (double(index) / N) +
                             (1.0 / (2.0 * M_PI)) *
                                 asin(interp_a(mag(i1), mag(i2), cos(2.0 * M_PI / N)) *
                                      sin(2.0 * M_PI / N));
            value = fabs(1.0 - v);
        }
    }
    out[(first + warp) * out_stride] = value;
}

// ---- FFT tunes in shared memory --------------------------------------------------
// One block per row (plane, particle) of one window: the samples are read
// from the orbit (mean subtracted, Hann window applied), transformed in
// shared memory, and the block writes the interpolated peak.  The transform of
// length M is an in-place mixed-radix network of radices 2, 3, 4, 5, 8 and
// 16.  Forward, decimation in frequency: stage s splits each block of
// N = r * span values (radix r) into r butterflies of stride `span`,
//     y_k = sum_q x_q w_r^{qk},  stored times w_N^{jk} (j: offset in the span),
// which takes natural order in and leaves X_k at a digit-reversed position
// (FftPlanDev::pos).  The inverse network runs the stages backwards with
// conjugate twiddles applied before each butterfly (decimation in time),
// which takes that order back to natural order (times M).  A window whose
// length has no prime factor above 5 is transformed directly (M = L) by the
// forward network, and its peak is found in the digit-reversed order.
// Other lengths take Bluestein's convolution (L. Bluestein, "A linear
// filtering approach to the computation of the discrete Fourier transform",
// IEEE Trans. Audio Electroacoust. 18 (1970) 451-455), which uses both
// networks:
//     X_k = c_k sum_n (z_n c_n) conj(c_{k-n}),  c_n = exp(-i pi n^2 / L),
// the cyclic convolution of length M >= 2L - 1 being the inverse network of
// the pointwise product of the forward network's outputs (that of b_m =
// conj(c_m) is precomputed, in the same order).  |c_k| = 1 and the peak
// interpolation depends on magnitude ratios only, so the peak is taken on
// |conv_k| directly.
//
// A long row's time is its passes over shared memory with a barrier after each,
// so there are as few as possible: radix 16 where the power of two allows; the
// first stage takes its values from the orbit; Bluestein's last forward stage,
// the product and the first inverse stage, which work on the same values,
// are one pass; the last stage looks for the maximum as it writes.  2^13
// values: 8 passes instead of 13.  32,768 rows, before -> now: windows of 4001
// (M = 8192) 6.67 -> 5.33 ms, 5001 (10240) 7.91 -> 6.6, 10,000 (direct) 6.1 -> 6.2; 38-41 % of the issue slots and 24-37 % of the
// FP64 pipe busy: one row fills an SM, so its passes, arithmetic and reads
// of the orbit follow one another.

__device__ __forceinline__ double2 c_add(double2 a, double2 b) {
    return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 c_sub(double2 a, double2 b) {
    return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 c_mul(double2 a, double2 b) {  // a b
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 c_mulc(double2 a, double2 b) {  // a conj(b)
    return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -(a.x * b.y)));
}
__device__ __forceinline__ double2 c_i(double2 a) {  // i a
    return make_double2(-a.y, a.x);
}

// Shared-memory slots of a row: M rounded up to a multiple of 8.
__host__ __device__ __forceinline__ uint32_t fft_row_slots(const FftPlanDev &pl) {
    return (pl.M + 7u) & ~7u;
}

// exp(-2 pi i t / M) from the two shared-memory tables (t < M).
__device__ __forceinline__ double2 fft_twiddle(const double2 *coarse, const double2 *fine,
                                               uint32_t t) {
    return c_mul(coarse[t >> 6], fine[t & 63u]);
}

// The DFT of R values in registers (R = 2, 3, 4, 5, 8, 16), forward
// (w = exp(-2 pi i / R)) or inverse (conjugate w).
template <bool INV>
__device__ __forceinline__ void dft4(double2 &x0, double2 &x1, double2 &x2, double2 &x3) {
    const double2 t0 = c_add(x0, x2), t1 = c_sub(x0, x2);
    const double2 t2 = c_add(x1, x3), t3 = c_sub(x1, x3);
    const double2 it3 = c_i(t3);
    x0 = c_add(t0, t2);
    x2 = c_sub(t0, t2);
    x1 = INV ? c_add(t1, it3) : c_sub(t1, it3);
    x3 = INV ? c_sub(t1, it3) : c_add(t1, it3);
}

// a w16^m, w16 = exp(-2 pi i / 16) (INV: the conjugate); m = 0..9 as needed.
template <int M16, bool INV>
__device__ __forceinline__ double2 mul_w16(double2 a) {
    constexpr double h = 0.70710678118654752440;   // cos(pi / 4)
    constexpr double c1 = 0.92387953251128675613;  // cos(pi / 8)
    constexpr double s1 = 0.38268343236508977173;  // sin(pi / 8)
    if constexpr (M16 == 0) return a;
    if constexpr (M16 == 4) return INV ? c_i(a) : make_double2(a.y, -a.x);
    if constexpr (M16 == 2)
        return INV ? make_double2(h * (a.x - a.y), h * (a.x + a.y))
                   : make_double2(h * (a.x + a.y), h * (a.y - a.x));
    if constexpr (M16 == 6)
        return INV ? make_double2(-h * (a.x + a.y), h * (a.x - a.y))
                   : make_double2(h * (a.y - a.x), -h * (a.x + a.y));
    // 1: (c1, -s1), 3: (s1, -c1), 9: (-c1, s1)
    constexpr double re = M16 == 1 ? c1 : (M16 == 3 ? s1 : -c1);
    constexpr double im = M16 == 1 ? -s1 : (M16 == 3 ? -c1 : s1);
    return INV ? c_mulc(a, make_double2(re, im)) : c_mul(a, make_double2(re, im));
}

template <int R, bool INV>
__device__ __forceinline__ void dft_small(double2 (&v)[R]) {
    if constexpr (R == 16) {
        // X_{a + 4 b} = sum_c w16^{ca} w4^{cb} sum_d x_{4d + c} w4^{da}
#pragma unroll
        for (int c = 0; c < 4; ++c) dft4<INV>(v[c], v[4 + c], v[8 + c], v[12 + c]);
        v[5] = mul_w16<1, INV>(v[5]);
        v[6] = mul_w16<2, INV>(v[6]);
        v[7] = mul_w16<3, INV>(v[7]);
        v[9] = mul_w16<2, INV>(v[9]);
        v[10] = mul_w16<4, INV>(v[10]);
        v[11] = mul_w16<6, INV>(v[11]);
        v[13] = mul_w16<3, INV>(v[13]);
        v[14] = mul_w16<6, INV>(v[14]);
        v[15] = mul_w16<9, INV>(v[15]);
#pragma unroll
        for (int a = 0; a < 4; ++a) dft4<INV>(v[4 * a], v[4 * a + 1], v[4 * a + 2], v[4 * a + 3]);
        // v[4a + b] holds X_{a + 4b}
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = a + 1; b < 4; ++b) {
                const double2 t = v[4 * a + b];
                v[4 * a + b] = v[4 * b + a];
                v[4 * b + a] = t;
            }
    } else if constexpr (R == 2) {
        const double2 a = v[0], b = v[1];
        v[0] = c_add(a, b);
        v[1] = c_sub(a, b);
    } else if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        // even and odd halves, then X_k = E_k + w8^k O_k, X_{k+4} = E_k - w8^k O_k
        double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
        double2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        dft4<INV>(e0, e1, e2, e3);
        dft4<INV>(o0, o1, o2, o3);
        constexpr double h = 0.70710678118654752440;  // sqrt(2) / 2
        // w8 o1, w8^2 o2, w8^3 o3 (forward w8 = h (1 - i); inverse h (1 + i))
        const double2 p1 = INV ? make_double2(h * (o1.x - o1.y), h * (o1.x + o1.y))
                               : make_double2(h * (o1.x + o1.y), h * (o1.y - o1.x));
        const double2 p2 = INV ? c_i(o2) : make_double2(o2.y, -o2.x);
        const double2 p3 = INV ? make_double2(-h * (o3.x + o3.y), h * (o3.x - o3.y))
                               : make_double2(h * (o3.y - o3.x), -h * (o3.x + o3.y));
        v[0] = c_add(e0, o0);
        v[4] = c_sub(e0, o0);
        v[1] = c_add(e1, p1);
        v[5] = c_sub(e1, p1);
        v[2] = c_add(e2, p2);
        v[6] = c_sub(e2, p2);
        v[3] = c_add(e3, p3);
        v[7] = c_sub(e3, p3);
    } else if constexpr (R == 5) {
        // cos(2 pi / 5), cos(4 pi / 5), sin(2 pi / 5), sin(4 pi / 5)
        constexpr double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
        constexpr double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
        const double2 x0 = v[0];
        const double2 t1 = c_add(v[1], v[4]), t2 = c_add(v[2], v[3]);
        const double2 u1 = c_sub(v[1], v[4]), u2 = c_sub(v[2], v[3]);
        v[0] = c_add(x0, c_add(t1, t2));
        const double2 a1 = make_double2(fma(c2, t2.x, fma(c1, t1.x, x0.x)),
                                        fma(c2, t2.y, fma(c1, t1.y, x0.y)));
        const double2 a2 = make_double2(fma(c1, t2.x, fma(c2, t1.x, x0.x)),
                                        fma(c1, t2.y, fma(c2, t1.y, x0.y)));
        const double2 ib1 = c_i(make_double2(fma(s1, u1.x, s2 * u2.x), fma(s1, u1.y, s2 * u2.y)));
        const double2 ib2 = c_i(make_double2(fma(s2, u1.x, -(s1 * u2.x)),
                                             fma(s2, u1.y, -(s1 * u2.y))));
        v[1] = INV ? c_add(a1, ib1) : c_sub(a1, ib1);
        v[4] = INV ? c_sub(a1, ib1) : c_add(a1, ib1);
        v[2] = INV ? c_add(a2, ib2) : c_sub(a2, ib2);
        v[3] = INV ? c_sub(a2, ib2) : c_add(a2, ib2);
    } else {
        static_assert(R == 3, "radix");
        constexpr double s = 0.86602540378443864676;  // sin(2 pi / 3)
        const double2 x0 = v[0];
        const double2 t = c_add(v[1], v[2]), u = c_sub(v[1], v[2]);
        v[0] = c_add(x0, t);
        const double2 a = make_double2(fma(-0.5, t.x, x0.x), fma(-0.5, t.y, x0.y));
        const double2 ib = c_i(make_double2(s * u.x, s * u.y));
        v[1] = INV ? c_add(a, ib) : c_sub(a, ib);
        v[2] = INV ? c_sub(a, ib) : c_add(a, ib);
    }
}

// Shared-memory slot of row value i: with SWZ (3 or 4) the low three bits of
// i (its place among 8 consecutive values, one 128-byte bank row of double2)
// are XORed with the three from bit SWZ on, so that the small strides of the
// last stages fall into different banks: a last stage of radix 16 has its
// threads 16 values apart, one of radix 8, 4 or 2 at most 8.  A bijection
// on every aligned group of 8, so rows of a multiple of 8 values stay in
// place.
template <int SWZ>
__device__ __forceinline__ uint32_t slot(uint32_t i) {
    return SWZ ? (i ^ ((i >> SWZ) & 7u)) : i;
}

// The twiddles w^k, k < R, w = exp(-2 pi i t / M): w, w^4 and w^8 from the
// tables, the others at most three products from those.  Radix 8 makes
// w^5 .. w^7 as it uses them: with all of them in registers beside its eight
// values the short rows' kernel spilled.
template <int R>
struct Twiddles {
    static constexpr int kKept = R == 8 ? 5 : R;
    double2 w[kKept];
    __device__ __forceinline__ Twiddles(const double2 *tc, const double2 *tf, uint32_t t) {
        w[0] = make_double2(1.0, 0.0);
        w[1] = fft_twiddle(tc, tf, t);
        if constexpr (R > 2) w[2] = c_mul(w[1], w[1]);
        if constexpr (R > 3) w[3] = c_mul(w[1], w[2]);
        if constexpr (R > 4) w[4] = R > 5 ? fft_twiddle(tc, tf, 4u * t) : c_mul(w[2], w[2]);
        if constexpr (R > 8) {
#pragma unroll
            for (int k = 5; k < 8; ++k) w[k] = c_mul(w[4], w[k - 4]);
            w[8] = fft_twiddle(tc, tf, 8u * t);
#pragma unroll
            for (int k = 9; k < 16; ++k) w[k] = c_mul(w[8], w[k - 8]);
        }
    }
    __device__ __forceinline__ double2 pow(int k) const {
        if constexpr (R == 8) return k < 5 ? w[k] : c_mul(w[4], w[k - 4]);
        else return w[k];
    }
};

struct NoTwiddles {
    __device__ __forceinline__ NoTwiddles(const double2 *, const double2 *, uint32_t) {}
};

// First maximum of |X_k|^2 (monotone in |X_k|), ties to the smallest k.
struct Peak {
    double m2;
    uint32_t k;
    __device__ __forceinline__ void see(double2 v, uint32_t at) {
        const double m = v.x * v.x + v.y * v.y;
        if (m > m2 || (m == m2 && at < k)) {
            m2 = m;
            k = at;
        }
    }
};

// A row, or a part of it that later stages keep to themselves: its plan, its
// values, the twiddle tables in shared memory, and the threads that work on
// it.
struct FftRow {
    const FftPlanDev &pl;
    double2 *row;
    const double2 *tc, *tf;
    uint32_t off, size;  // the part's values
    uint32_t t, T;       // this thread's index among the part's threads
};

// Butterflies t, t + T, ... of a stage of radix R: block b / span at offset
// j = b % span, kept without divisions.
template <int R, class F>
__device__ __forceinline__ void butterflies(const FftRow &r, uint32_t span, F body) {
    const uint32_t nb = r.size / R, T = r.T;
    uint32_t blk = r.t / span, j = r.t - blk * span;
    const uint32_t dq = T / span, dr = T - dq * span;
    constexpr int kUnroll = R >= 8 ? 1 : 2;  // larger radices fill the registers alone
#pragma unroll kUnroll
    for (uint32_t b = r.t; b < nb; b += T) {
        body(j, r.off + blk * span * R + j);
        blk += dq;
        j += dr;
        if (j >= span) {
            j -= span;
            ++blk;
        }
    }
}

// Where a stage's values come from and go to.
enum : int {
    kFromRow = 0,   // row to row
    kFromOrbit = 1, // the first forward stage: value i is in(i)
    kToPeak = 2,    // the last stage: also seen by the peak
};

// One stage of radix R: forward, butterfly then twiddles; inverse, conjugate
// twiddles then the inverse butterfly.  A stage of span 1 has j = 0 and no
// twiddles (TW false).  The twiddles w_N^{jk}, N = R span, are
// exp(-2 pi i j k prod / M).
template <int R, bool INV, int SWZ, bool TW, int MODE, class In>
__device__ __forceinline__ void fft_stage(const FftRow &r, uint32_t span, uint32_t prod, In in,
                                          Peak &peak) {
    double2 *const row = r.row;
    butterflies<R>(r, span, [&](uint32_t j, uint32_t base) {
        double2 v[R];
        const std::conditional_t<TW, Twiddles<R>, NoTwiddles> w(r.tc, r.tf, j * prod);
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if constexpr (MODE == kFromOrbit) v[q] = in(base + q * span);
            else v[q] = row[slot<SWZ>(base + q * span)];
            if constexpr (TW && INV)
                if (q > 0) v[q] = c_mulc(v[q], w.pow(q));
        }
        dft_small<R, INV>(v);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if constexpr (TW && !INV)
                if (k > 0) v[k] = c_mul(v[k], w.pow(k));
            const uint32_t at = base + k * span;
            row[slot<SWZ>(at)] = v[k];
            if constexpr (MODE == kToPeak) {
                if constexpr (INV) {
                    if (at < r.pl.L) peak.see(v[k], at);
                } else {
                    peak.see(v[k], r.pl.freq[at]);
                }
            }
        }
    });
}

template <int R, bool INV, int SWZ, int MODE, class In>
__device__ __forceinline__ void fft_stage_any(const FftRow &r, uint32_t span, uint32_t prod,
                                              In in, Peak &peak) {
    if (span == 1) fft_stage<R, INV, SWZ, false, MODE>(r, span, prod, in, peak);
    else fft_stage<R, INV, SWZ, true, MODE>(r, span, prod, in, peak);
}

template <int MAXR, bool INV, int SWZ, int MODE, class In>
__device__ void fft_stage_of(const FftRow &r, int s, In in, Peak &peak) {
    const uint32_t span = r.pl.stage_len[s], prod = r.pl.stage_prod[s];
    switch (r.pl.radix[s]) {
        case 16:
            if constexpr (MAXR >= 16) fft_stage_any<16, INV, SWZ, MODE>(r, span, prod, in, peak);
            break;
        case 8: fft_stage_any<8, INV, SWZ, MODE>(r, span, prod, in, peak); break;
        case 4: fft_stage_any<4, INV, SWZ, MODE>(r, span, prod, in, peak); break;
        case 2: fft_stage_any<2, INV, SWZ, MODE>(r, span, prod, in, peak); break;
        case 5: fft_stage_any<5, INV, SWZ, MODE>(r, span, prod, in, peak); break;
        default: fft_stage_any<3, INV, SWZ, MODE>(r, span, prod, in, peak); break;
    }
}

// Bluestein's turning point: the last forward stage (span 1, no twiddles),
// the product with the kernel's transform and the first inverse stage.
template <int R, int SWZ>
__device__ __forceinline__ void fft_turn(const FftRow &r) {
    const uint32_t nb = r.pl.M / R, b1 = (r.off + r.size) / R;
    for (uint32_t b = r.off / R + r.t; b < b1; b += r.T) {
        double2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = r.row[slot<SWZ>(b * R + q)];
        dft_small<R, false>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = c_mul(v[q], __ldg(r.pl.bhat + q * nb + b));
        dft_small<R, true>(v);
#pragma unroll
        for (int q = 0; q < R; ++q) r.row[slot<SWZ>(b * R + q)] = v[q];
    }
}

template <int MAXR, int SWZ>
__device__ void fft_turn_of(const FftRow &r) {
    switch (r.pl.radix[r.pl.n_stages - 1]) {
        case 16:
            if constexpr (MAXR >= 16) fft_turn<16, SWZ>(r);
            break;
        case 8: fft_turn<8, SWZ>(r); break;
        case 4: fft_turn<4, SWZ>(r); break;
        case 2: fft_turn<2, SWZ>(r); break;
        case 5: fft_turn<5, SWZ>(r); break;
        default: fft_turn<3, SWZ>(r); break;
    }
}

// Two kernels, by the length M of the transform.  Long rows (MAXR = 16, M >=
// kFftLongRow): an SM's shared memory holds one of them, so the block has
// few passes: 512 threads of 128 registers, one radix-16 butterfly each for
// 8192 values, the first stage from the orbit, groups of threads.  Of shorter
// rows (MAXR = 8) an SM holds several, whose passes overlap one another if
// there are enough of them: radices to 8 in 64 registers, up to 256 threads
// (at least 64), the row first brought into shared memory together with the
// twiddles, one wait for both.  8,000 rows, us, with a pass for every step in 64
// registers, with the long rows' kernel alone, and now:
//     samples (M)       99 (200)  499 (1000)  1000   2999 (6000)  3071 (6144)   4800
//     before             61          154       119       1147         1369       733
//     long rows' kernel 127          216       206       1489         1234      1007
//     now                63          179       124       1052          943       666
// From M = 7200 on the long rows' kernel is the faster: 3,599 samples 1617 us,
// with the other 1866.
constexpr uint32_t kFftGroups = 4;

template <int MAXR>
constexpr int kFftThreadsMax = MAXR >= 16 ? 512 : 256;

template <int MAXR, int SWZ>
__global__ void __launch_bounds__(kFftThreadsMax<MAXR>, MAXR >= 16 ? 1 : 4)
    fft_tune_kernel(const FftTuneArgs a) {
    extern __shared__ __align__(16) double2 fft_sm[];
    __shared__ double red_m[kFftThreadsMax<MAXR> / 32];
    __shared__ uint32_t red_k[kFftThreadsMax<MAXR> / 32];
    const FftPlanDev &pl = a.plan;
    double2 *row = fft_sm;
    double2 *tc = row + fft_row_slots(pl);
    double2 *tf = tc + pl.n_coarse;
    const size_t rix = blockIdx.x;  // plane * n + particle
    const int plane = rix >= a.n ? 1 : 0;
    const size_t i = rix - size_t(plane) * a.n;
    // Only one or a few rows fit in an SM's shared memory, so a block's
    // reads would not overlap other rows' transforms: each block asks L2 for
    // the window of the row that starts about one wave of resident blocks
    // later (prefetch.global.L2, one per 128-byte line, addresses within
    // the row).
    if (a.stride_s == 1) {  // rows contiguous
        const size_t r2 = rix + a.prefetch_ahead;
        if (r2 < 2 * a.n) {
            const int plane2 = r2 >= a.n ? 1 : 0;
            const size_t i2 = r2 - size_t(plane2) * a.n;
            const size_t bytes = size_t(pl.L) * sizeof(double);
            const size_t o2 = i2 * a.stride_i + a.from;
            const char *rq = reinterpret_cast<const char *>((plane2 ? a.y : a.x) + o2);
            const char *rp = reinterpret_cast<const char *>((plane2 ? a.py : a.px) + o2);
            const uint32_t lines = uint32_t((bytes + 127u) / 128u) + 1u;
            for (uint32_t l = threadIdx.x; l < 2u * lines; l += blockDim.x) {
                const size_t off = min(size_t(l % lines) * 128u, bytes - sizeof(double));
                const char *ptr = (l < lines ? rq : rp) + off;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
            }
        }
    }
    if (a.first_nan && a.first_nan[i] <= a.last_sample) {  // a NaN sample in the window: NaN tune
        if (threadIdx.x == 0)
            for (int c = 0; c < a.n_out_cols; ++c)
                a.out[i * a.cols + 2 * size_t(a.out_cols[c]) + plane] = dev::quiet_nan();
        return;
    }
    for (uint32_t t = threadIdx.x; t < pl.n_coarse; t += blockDim.x) tc[t] = pl.tw_coarse[t];
    for (uint32_t t = threadIdx.x; t < 64u; t += blockDim.x) tf[t] = pl.tw_fine[t];
    if constexpr (MAXR >= 16) __syncthreads();
    const double *q = plane ? a.y : a.x, *p = plane ? a.py : a.px;
    const double mq = mean_of(a.means, a.n, i, 2 * plane, a.S);
    const double mp = mean_of(a.means, a.n, i, 2 * plane + 1, a.S);
    // z_k = ((q - mean) + i (p - mean)) h_k, for Bluestein times c_k and with
    // zeros up to M.
    const size_t o0 = i * a.stride_i + size_t(a.from) * a.stride_s;
    int nan_seen = 0;
    auto in = [&](uint32_t k) {
        if (k >= pl.L) return make_double2(0.0, 0.0);
        const size_t o = o0 + size_t(k) * a.stride_s;
        const double re = centred(q[o], a.means, mq), im = centred(p[o], a.means, mp);
        nan_seen |= isnan(re) || isnan(im);
        const double hk = a.hann[k];
        const double2 z = make_double2(re * hk, im * hk);
        return pl.bluestein ? c_mul(z, __ldg(pl.chirp + k)) : z;
    };
    const FftRow whole{pl, row, tc, tf, 0u, pl.M, threadIdx.x, blockDim.x};
    const int last = pl.n_stages - 1;
    // After a first stage of radix r the row is r independent transforms.
    // Where r is a multiple of kFftGroups (powers of two) and there is a stage
    // in between, each group of the block's threads takes its share of them
    // through the middle stages, waiting for its own threads only: the groups
    // drift apart, so that one's shared-memory passes overlap another's
    // arithmetic (8192 values, 32,768 rows: 5.38 instead of 5.62 ms).  Lengths
    // with fives keep them first: with 16 first and groups, 10240 values took
    // 7.27 ms instead of 6.49, their butterflies not dealing out evenly.
    const bool split = MAXR >= 16 && last > 1 && pl.radix[0] % kFftGroups == 0;
    const uint32_t groups = split ? kFftGroups : 1u;
    const uint32_t per = MAXR >= 16 ? blockDim.x / groups : blockDim.x;
    const uint32_t group = MAXR >= 16 ? threadIdx.x / per : 0u;
    const FftRow part{pl,  row, tc, tf, MAXR >= 16 ? group * (pl.M / groups) : 0u,
                      MAXR >= 16 ? pl.M / groups : pl.M,
                      MAXR >= 16 ? threadIdx.x - group * per : threadIdx.x, per};
    static_assert(kFftGroups == 4u, "one named barrier per group below");
    auto part_sync = [&]() {
        if constexpr (MAXR < 16) {
            __syncthreads();
            return;
        }
        // (barrier numbers as constants: five in all, not sixteen)
        switch (group) {
            case 0: asm volatile("bar.sync 1, %0;" ::"r"(per) : "memory"); break;
            case 1: asm volatile("bar.sync 2, %0;" ::"r"(per) : "memory"); break;
            case 2: asm volatile("bar.sync 3, %0;" ::"r"(per) : "memory"); break;
            default: asm volatile("bar.sync 4, %0;" ::"r"(per) : "memory"); break;
        }
    };
    Peak peak{-1.0, 0xffffffffu};
    int s = 0;  // forward stages done
    bool loaded = false;
    if constexpr (MAXR >= 16)
        if (last > 0) {
            fft_stage_of<MAXR, false, SWZ, kFromOrbit>(whole, 0, in, peak);
            s = 1;
            loaded = true;
        }
    if (!loaded) {
#pragma unroll 4
        for (uint32_t k = threadIdx.x; k < pl.M; k += blockDim.x) row[slot<SWZ>(k)] = in(k);
    }
    // Without first-NaN records the window's own samples decide
    // (fft_tune_vec's rule, scanning the window).
    if (__syncthreads_or(a.first_nan == nullptr && nan_seen)) {
        if (threadIdx.x == 0)
            for (int c = 0; c < a.n_out_cols; ++c)
                a.out[i * a.cols + 2 * size_t(a.out_cols[c]) + plane] = dev::quiet_nan();
        return;
    }
    for (; s < last; ++s) {
        fft_stage_of<MAXR, false, SWZ, kFromRow>(part, s, in, peak);
        part_sync();
    }
    if (pl.bluestein) {
        fft_turn_of<MAXR, SWZ>(part);
        part_sync();
        for (s = last - 1; s > 0; --s) {
            fft_stage_of<MAXR, true, SWZ, kFromRow>(part, s, in, peak);
            part_sync();
        }
        __syncthreads();
        if (last > 0) {
            fft_stage_of<MAXR, true, SWZ, kToPeak>(whole, 0, in, peak);
        } else {
            for (uint32_t k = threadIdx.x; k < pl.L; k += blockDim.x) peak.see(row[slot<SWZ>(k)], k);
        }
    } else if (last >= 0) {
        fft_stage_of<MAXR, false, SWZ, kToPeak>(part, last, in, peak);
    } else {  // one sample
        if (threadIdx.x == 0) peak.see(row[0], 0u);
    }
    // the peak's neighbours are read below, after the barrier of the reduction
    auto at = [&](uint32_t k) { return row[slot<SWZ>(pl.bluestein || last < 0 ? k : pl.pos[k])]; };
    double best = peak.m2;
    uint32_t best_k = peak.k;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_down_sync(dev::kFullMask, best, o);
        const uint32_t ok = __shfl_down_sync(dev::kFullMask, best_k, o);
        if (ob > best || (ob == best && ok < best_k)) {
            best = ob;
            best_k = ok;
        }
    }
    if (lane == 0) {
        red_m[warp] = best;
        red_k[warp] = best_k;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (unsigned w = 1; w < blockDim.x / 32u; ++w)
        if (red_m[w] > best || (red_m[w] == best && red_k[w] < best_k)) {
            best = red_m[w];
            best_k = red_k[w];
        }
    auto mag = [&](uint32_t k) {
        const double2 v = at(k);
        return sqrt(v.x * v.x + v.y * v.y);
    };
    // interpolation (src/dynamic_indicator.cpp:139-176), as fft_peak2_kernel
    const uint32_t len = pl.L;
    double value;
    uint32_t index = best_k;
    const double N = double(len);
    if (index == 0 || index >= len) {
        value = 1.0;
    } else if (index == len - 1) {
        value = 0.0;
    } else {
        uint32_t i1, i2;
        if (mag(index - 1) > mag(index + 1)) {
            i1 = index - 1;
            i2 = index;
            index = index - 1;
        } else {
            i1 = index;
            i2 = index + 1;
        }
        const double v = (double(index) / N) +
                         (1.0 / (2.0 * M_PI)) *
                             asin(interp_a(mag(i1), mag(i2), cos(2.0 * M_PI / N)) *
                                  sin(2.0 * M_PI / N));
        value = fabs(1.0 - v);
    }
    for (int c = 0; c < a.n_out_cols; ++c)
        a.out[i * a.cols + 2 * size_t(a.out_cols[c]) + plane] = value;
}

template <int ARITH, bool OCT>
void launch_record_ok(const OrbitRecordArgs &a, unsigned blocks, cudaStream_t s) {
    const bool kick = !isnan(a.kick_module);
    if (a.inverse) {
        if (kick) orbit_record_kernel<ARITH, OCT, true, true><<<blocks, 64, 0, s>>>(a);
        else orbit_record_kernel<ARITH, OCT, true, false><<<blocks, 64, 0, s>>>(a);
    } else {
        if (kick) orbit_record_kernel<ARITH, OCT, false, true><<<blocks, 64, 0, s>>>(a);
        else orbit_record_kernel<ARITH, OCT, false, false><<<blocks, 64, 0, s>>>(a);
    }
}

}  // namespace

cudaError_t launch_orbit_record(const OrbitRecordArgs &a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    // 32 particles per block: the orbits of few particles are spread over as
    // many SMs as possible.
    const unsigned blocks = unsigned((a.n + 31) / 32);
    const bool oct = a.mu != 0.0;
    if (a.arith == HM_ARITH_FAST) {
        if (oct) launch_record_ok<HM_ARITH_FAST, true>(a, blocks, s);
        else launch_record_ok<HM_ARITH_FAST, false>(a, blocks, s);
    } else {
        if (oct) launch_record_ok<HM_ARITH_EXACT, true>(a, blocks, s);
        else launch_record_ok<HM_ARITH_EXACT, false>(a, blocks, s);
    }
    return cudaGetLastError();
}

cudaError_t launch_birkhoff_segments(const BirkhoffSegArgs &a, cudaStream_t s) {
    if (a.n == 0 || a.n_win == 0) return cudaSuccess;
    const size_t threads = 2u * size_t(a.n_seg) * a.n;
    const dim3 grid(unsigned((threads + 127) / 128), unsigned((a.n_win + kWinGroup - 1) / kWinGroup));
    birkhoff_seg_kernel<<<grid, 128, 0, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t t2 = 2u * size_t(a.n_win) * a.n;
    birkhoff_finish_kernel<<<unsigned((t2 + 127) / 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_hann_table(double *h, uint32_t len, cudaStream_t s) {
    if (len == 0) return cudaSuccess;
    hann_table_kernel<<<(len + 255) / 256, 256, 0, s>>>(h, len);
    return cudaGetLastError();
}

cudaError_t launch_fft_gather2(const double *x, const double *px, const double *y,
                               const double *py, const double *means, size_t n, uint32_t from,
                               uint32_t len, const double *h, double2 *z, size_t S,
                               size_t pitch, cudaStream_t s) {
    if (n == 0 || len == 0) return cudaSuccess;
    const unsigned grid = unsigned((n * len + 255) / 256);
    for (int plane = 0; plane < 2; ++plane) {
        fft_gather2_kernel<<<grid, 256, 0, s>>>(x, px, y, py, means, n, from, len, h, z, S, pitch,
                                                plane);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_fft_peak2(const double2 *z, uint32_t len, size_t n, uint32_t last_sample,
                             const uint32_t *first_nan, double *out, size_t cols, int col,
                             cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const size_t threads = 2 * n * 32;
    fft_peak2_kernel<<<unsigned((threads + 255) / 256), 256, 0, s>>>(z, len, n, last_sample,
                                                                    first_nan, out, cols, col);
    return cudaGetLastError();
}

size_t fft_tune_smem_bytes(const FftPlanDev &plan) {
    return (size_t(fft_row_slots(plan)) + plan.n_coarse + 64u) * sizeof(double2);
}

cudaError_t launch_fft_tunes(const FftTuneArgs &a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    if (a.plan.M == 0 || a.plan.M > kFftMaxLen || a.plan.L == 0) return cudaErrorInvalidValue;
    const size_t smem = fft_tune_smem_bytes(a.plan);
    const bool long_row = a.plan.M >= kFftLongRow;
    auto kernel = long_row ? (a.plan.swizzle == 4   ? fft_tune_kernel<16, 4>
                              : a.plan.swizzle == 3 ? fft_tune_kernel<16, 3>
                                                    : fft_tune_kernel<16, 0>)
                           : (a.plan.swizzle == 3 ? fft_tune_kernel<8, 3> : fft_tune_kernel<8, 0>);
    if (smem > 40u * 1024u) {
        const cudaError_t e =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return e;
    }
    // About one butterfly of the largest radix per thread and stage; whole
    // warps in each group of a long row.
    const uint32_t step = long_row ? 32u * kFftGroups : 32u;
    const uint32_t least = long_row ? step : 64u;
    const uint32_t most = uint32_t(long_row ? kFftThreadsMax<16> : kFftThreadsMax<8>);
    const uint32_t want = (a.plan.M / (long_row ? 16u : 8u) + step - 1u) / step * step;
    const int threads = int(std::min(most, std::max(least, want)));
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    FftTuneArgs b = a;
    b.prefetch_ahead = uint32_t(std::max(1, sms * std::max(1, per_sm)));
    kernel<<<unsigned(2 * a.n), threads, smem, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_mean_remove(double *x, double *px, double *y, double *py, size_t n, size_t S,
                               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    mean_remove_kernel<<<unsigned((4u * n + 127) / 128), 128, 0, s>>>(x, px, y, py, n, S);
    return cudaGetLastError();
}

cudaError_t launch_birkhoff_tunes(const double *x, const double *px, const double *y,
                                  const double *py, size_t n, const uint32_t *from,
                                  const uint32_t *to, const uint64_t *w_off, const double *w,
                                  int n_win, double *out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const size_t threads = n * 2u * size_t(n_win);
    birkhoff_kernel<<<unsigned((threads + 127) / 128), 128, 0, s>>>(x, px, y, py, n, from, to,
                                                                    w_off, w, n_win, out);
    return cudaGetLastError();
}

cudaError_t launch_hann_gather(const double *q, const double *p, size_t n, uint32_t from,
                               uint32_t len, size_t first, size_t count, double2 *buf,
                               int *nan_flags, cudaStream_t s) {
    const size_t total = count * len;
    if (total == 0) return cudaSuccess;
    hann_gather_kernel<<<unsigned((total + 255) / 256), 256, 0, s>>>(q, p, n, from, len, first,
                                                                      count, buf, nan_flags);
    return cudaGetLastError();
}

cudaError_t launch_fft_peak(const double2 *buf, uint32_t len, size_t count, const int *nan_flags,
                            double *out, size_t out_stride, size_t first, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    const size_t threads = count * 32;
    fft_peak_kernel<<<unsigned((threads + 255) / 256), 256, 0, s>>>(buf, len, count, nan_flags,
                                                                    out, out_stride, first);
    return cudaGetLastError();
}

}  // namespace hm
