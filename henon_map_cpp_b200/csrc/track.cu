// Fused multi-turn tracking kernels for the 4D modulated Henon map (sm_100a).
//
// One launch advances a list of live particles by a chunk of turns with the
// particle state held in registers (several particles per thread for
// instruction-level parallelism).  The per-turn rotation record
// {sin wx, cos wx, sin wy, cos wy} is the same for every live particle (all
// live particles share the same `steps`), so each warp reads one broadcast
// record per turn.  Losses are looked for once per block of turns, and the
// turn of a loss is found by redoing its block (dev::block_turns); a lost
// particle is written out (NaN coordinates, frozen steps) and survivors are
// re-compacted
// into a dense list at the end of the chunk so that the next chunk's warps
// are full.
//
// Reference semantics: henon_step, src/henon.cu:420-542, built from the
// primitives of src/henon.cu:113-173; launch loop of
// henon_tracker_gpu::track, src/henon.cu:3155-3185.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "hm_device.cuh"
#include "hm_internal.h"

namespace hm {

// Multiprocessors of the current device (cached per device ordinal).
int sm_count() {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> cache[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 1;
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v <= 0) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            return 1;
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

namespace {

using dev::Barrier;
using dev::kFullMask;
using dev::Particle;
using dev::quiet_nan;
using dev::Rn;
using dev::Turn;

// One turn of the K particles of a thread.  The common case costs the map
// and, per thread, an OR of the coordinates' high words and one integer
// compare (dev::small_or); a warp with a thread whose coordinates are not
// all small takes the rare path, which settles the barrier test per
// particle and freezes lost particles (set_to_nan, src/henon.cu:123-129)
// with steps = the turns they survived.  A lost particle's registers are
// set to zero, a fixed point of the map, so that it never trips the OR
// again.
template <int ARITH, bool OCT, bool REV, int K>
__device__ __forceinline__ void turn_all(const TrackChunk &c, const Barrier &bar, double mu,
                                         const Turn &t, uint32_t k, Particle (&p)[K],
                                         const uint32_t (&id)[K], bool (&live)[K],
                                         bool &warp_live) {
    uint32_t ored = 0u;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        dev::turn<ARITH, OCT, REV>(p[j], t, mu);
        ored |= dev::hi_or(p[j]);
    }
    if (__any_sync(kFullMask, !dev::small_or(ored, bar))) {
        const uint32_t s = REV ? c.turn0 - k : c.turn0 + k;
        bool any_live = false;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            if (live[j] && !dev::small_inside(p[j], bar) &&
                !dev::inside<ARITH>(dev::radius_fma(p[j]), p[j], bar)) {
                const uint32_t i = id[j];
                c.ux[i] = quiet_nan();
                c.upx[i] = quiet_nan();
                c.uy[i] = quiet_nan();
                c.upy[i] = quiet_nan();
                c.usteps[i] = s;
                live[j] = false;
                p[j] = dev::make_particle(0.0, 0.0, 0.0, 0.0);
            }
            any_live |= live[j];
        }
        warp_live = __any_sync(kFullMask, any_live);
    }
}

// The chunk's turns with the turn records read from global memory: every
// lane of a warp loads the same 32-byte record (one broadcast transaction,
// an L1 hit after the first warp), prefetched one turn ahead.
template <int ARITH, bool OCT, bool REV, int K>
__device__ __forceinline__ void turns_direct(const TrackChunk &c, const Barrier &bar,
                                             Particle (&p)[K], const uint32_t (&id)[K],
                                             bool (&live)[K], bool warp_live) {
    const double mu = c.mu;
    const uint32_t nt = c.n_turns;
    Turn t = nt ? dev::load_turn(c.table, REV ? c.turn0 - 1u : c.turn0) : Turn{0.0, 0.0, 0.0, 0.0};
    for (uint32_t k = 0; warp_live && k < nt; ++k) {
        const uint32_t kn = (k + 1 < nt) ? k + 1 : k;
        const Turn tn = dev::load_turn(c.table, REV ? c.turn0 - 1u - kn : c.turn0 + kn);
        turn_all<ARITH, OCT, REV, K>(c, bar, mu, t, k, p, id, live, warp_live);
        t = tn;
    }
}

// Shared memory of a staged launch: two stage buffers of turn records and two
// checkpoints {x, px, y, py} per particle.
__host__ __device__ constexpr size_t staged_smem_bytes(uint32_t stage_turns, uint32_t threads,
                                                       int per_thread) {
    return size_t(stage_turns) * 2u * 32u + size_t(threads) * per_thread * 64u;
}

__device__ __forceinline__ Turn staged_record(const double *rec, uint32_t kn, uint32_t kk,
                                              bool rev) {
    const double2 *q = reinterpret_cast<const double2 *>(rec + 4u * (rev ? kn - 1u - kk : kk));
    const double2 a = q[0], b = q[1];
    return Turn{a.x, a.y, b.x, b.y};
}

// The chunk's turns with the turn records staged in shared memory: the
// chunk is cut into stages of c.stage_turns turns whose records (a
// contiguous span of the table) one thread brings in with a bulk copy,
// double-buffered, so that the copy of stage s+1 overlaps the turns of
// stage s.  Every warp then reads each record from shared memory as a
// broadcast.  Warps whose particles are all lost keep taking part in the
// per-stage barriers; the block stops when none of its warps is live.
//
// A stage runs in blocks of turns with no per-turn control
// flow (dev::block_turns): the thread saves its particles to shared memory
// and applies the block's turns.  If the coordinates looked at stayed below
// the bound, no particle can have been lost in the block, which is then
// exactly what the per-turn test would have produced.  Otherwise the warp
// restores the saved particles and redoes the block: looking at every turn,
// whose bound is higher, if that may still pass, else with the per-turn test
// (turn_all).  The warp votes on a block while it already runs the next one
// (hence two checkpoints): a vote before each block made every warp wait
// for the end of its chain of turns, 54 instead of 50 cycles a turn with one
// warp per scheduler and 43.9 instead of 43.2 with four.  Sixteen turns keep
// a loss cheap (at most 32 turns repeated) where a fifth of the particles is
// lost in 512 turns; blocks of 8 cost 1.4 cycles a turn more and runs of 128
// turns 4 % of the dynamic-aperture scan.
//
// A small barrier has orbits that live above a bound (at mu = 0 that of every
// second turn is 1.35 for barrier 10, 0.50 for 2 and 0.31 for 1, that of every
// turn half the barrier): after kVainRedos blocks of a stage that were redone
// for nothing the warp looks, or tests, that way for the rest of the stage.
// A single one is more often an orbit on its way out: with 2 in place of 4 the
// loss-heavy start of a scan took 8 % more with two particles per thread
// (1024^2 points on [0, 0.6]^2, 3,000 turns, mu = 0.2: 6.7 and 6.3 ms), and a
// small barrier 2-10 % less.  ms for 10^4 turns, with per-turn looks in runs of
// 32, with blocks that were all retested, now:
//     barrier             0.8    1      2      3      10
//     90,000 particles    4.16   4.52   4.07   4.05   2.02
//       (mu = 0.2)        5.75   5.61   4.73   4.24   1.87
//                         3.31   3.31   2.24   2.16   1.80
//     3,600 particles     2.22   1.94   1.74   1.75   0.47
//       (mu = 0)          2.42   2.12   1.76   0.56   0.33
//                         1.95   1.64   0.45   0.36   0.33
enum class Look {
    kPairs,  // at every second turn
    kEvery,  // at every turn
    kTest,   // the test itself
};
constexpr uint32_t kVainRedos = 4;

// Returns false when a copy did not land within the bounded wait (the
// chunk's results are then invalid and c.fault is set).
template <int ARITH, bool OCT, bool REV, int K>
__device__ __forceinline__ bool turns_staged(const TrackChunk &c, const Barrier &bar,
                                             Particle (&p)[K], const uint32_t (&id)[K],
                                             bool (&live)[K], bool warp_live) {
    // [2][S][4] turn records, then [2][K][blockDim.x] checkpoints.
    extern __shared__ __align__(128) double stage_buf[];
    __shared__ __align__(8) uint64_t full[2];
    const double mu = c.mu;
    const uint32_t nt = c.n_turns, S = c.stage_turns;
    const uint32_t n_stages = (nt + S - 1) / S;
    double2 *const ckpt = reinterpret_cast<double2 *>(stage_buf + size_t(S) * 8u);
    const bool leader = threadIdx.x == 0;
    auto issue = [&](uint32_t st) {
        const uint32_t k0 = st * S;
        const uint32_t kn = min(S, nt - k0);
        const uint32_t lo = REV ? c.turn0 - k0 - kn : c.turn0 + k0;
        dev::bulk_load(stage_buf + size_t(st & 1u) * S * 4u, c.table + size_t(lo) * 4u,
                       kn * 32u, &full[st & 1u]);
    };
    // A chunk of one stage has nothing to overlap: the block copies its
    // records itself, and no copy can time out.
    const bool one_stage = n_stages == 1;
    if (one_stage) {
        const double2 *const src = reinterpret_cast<const double2 *>(
            c.table + size_t(REV ? c.turn0 - nt : c.turn0) * 4u);
        double2 *const dst = reinterpret_cast<double2 *>(stage_buf);
        for (uint32_t i = threadIdx.x; i < 2u * nt; i += blockDim.x) dst[i] = __ldg(src + i);
    } else if (leader) {
        dev::mbar_init(&full[0], 1);
        dev::mbar_init(&full[1], 1);
        dev::mbar_init_fence();
    }
    __syncthreads();
    if (leader && !one_stage) {
        if (n_stages > 0) issue(0);
        if (n_stages > 1) issue(1);
    }
    bool timed_out = false;
    uint32_t st = 0;
    for (; st < n_stages; ++st) {
        const uint32_t buf = st & 1u;
        // Warp-uniform, so that the turn loop's warp votes see every lane.
        const bool landed = one_stage || dev::mbar_wait(&full[buf], (st >> 1) & 1u);
        if (!__all_sync(kFullMask, landed)) timed_out = true;
        const uint32_t k0 = st * S;
        const uint32_t kn = min(S, nt - k0);
        const double *rec = stage_buf + size_t(buf) * S * 4u;
        if (!timed_out) {
            // A caller's records are checked to be rotations, which the
            // test of every second turn needs.
            Look look = c.pair_hi != 0u ? Look::kPairs : Look::kEvery;
            if (look == Look::kPairs && c.check_records) {
                const double2 *q = reinterpret_cast<const double2 *>(rec);
                bool unit = true;
                for (uint32_t kk = threadIdx.x & 31u; kk < kn; kk += 32u)
                    unit = unit && dev::is_rotation(q[2u * kk], q[2u * kk + 1u]);
                if (!__all_sync(kFullMask, unit)) look = Look::kEvery;
            }
            constexpr uint32_t B = dev::kBlockTurns;
            const uint32_t pair_hi = c.pair_hi;
            const double2 *const q0 =
                reinterpret_cast<const double2 *>(rec) + (REV ? 2u * (kn - 1u) : 0u);
            auto record = [&](uint32_t kk) { return REV ? q0 - 2u * kk : q0 + 2u * kk; };
            double2 *save = ckpt, *saved = ckpt + size_t(2u * K) * blockDim.x;
            auto checkpoint = [&]() {
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    double2 *const to = save + 2u * (j * blockDim.x + threadIdx.x);
                    to[0] = make_double2(p[j].x, p[j].px);
                    to[1] = make_double2(p[j].y, p[j].py);
                }
            };
            auto swap = [&]() {
                double2 *const t = save;
                save = saved;
                saved = t;
            };
            auto restore = [&]() {
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    const double2 *const from = saved + 2u * (j * blockDim.x + threadIdx.x);
                    const double2 a = from[0], b = from[1];
                    p[j] = dev::make_particle(a.x, a.y, b.x, b.y);
                }
            };
            bool check = false;  // this thread's verdict on the block before ...
            uint32_t top = 0u;   // ... and the largest coordinate it saw
            uint32_t soft = 0u, vain = 0u;  // blocks redone without a loss, by the two tests
            for (uint32_t j0 = 0; warp_live && j0 < kn;) {
                if (look == Look::kTest) {
                    for (; warp_live && j0 < kn; ++j0)
                        turn_all<ARITH, OCT, REV, K>(c, bar, mu, staged_record(rec, kn, j0, REV),
                                                     k0 + j0, p, id, live, warp_live);
                    break;
                }
                bool again = false;  // the warp's
                // The hot loops hold nothing but blocks: with the redo's code
                // inside a turn took 3 cycles more.
                const uint32_t jb = j0 + (kn - j0) / B * B;
                const double2 *q = record(j0);
                if (look == Look::kPairs) {
#pragma unroll 2
                    for (; j0 < jb; j0 += B, q += REV ? -int(2u * B) : int(2u * B)) {
                        checkpoint();
                        again = __any_sync(kFullMask, check);
                        const uint32_t seen = dev::block_turns<ARITH, OCT, REV, K>(p, q, mu);
                        if (again) break;
                        check = seen >= pair_hi;
                        top = seen;
                        swap();
                    }
                } else {
#pragma unroll 1
                    for (; j0 < jb; j0 += B, q += REV ? -int(2u * B) : int(2u * B)) {
                        checkpoint();
                        again = __any_sync(kFullMask, check);
                        const uint32_t seen = dev::block_turns<ARITH, OCT, REV, K, true>(p, q, mu);
                        if (again) break;
                        check = seen >= bar.small_hi;
                        top = seen;
                        swap();
                    }
                }
                if (!again && j0 < kn) {  // a short block
                    checkpoint();
                    again = __any_sync(kFullMask, check);
                    if (!again) {
                        top = dev::each_turn<ARITH, OCT, REV, K>(p, record(j0), kn - j0, mu);
                        check = top >= bar.small_hi;
                        j0 += B;
                        swap();
                    }
                }
                if (!again && j0 >= kn) again = __any_sync(kFullMask, check);
                if (again) {  // the block that ended at j0
                    restore();
                    bool test = __any_sync(kFullMask, top >= bar.small_hi);
                    if (!test) {
                        // Above the bound of every second turn alone.
                        top = dev::each_turn<ARITH, OCT, REV, K>(p, record(j0 - B), B, mu);
                        test = __any_sync(kFullMask, top >= bar.small_hi);
                        if (test) restore();
                        else if (++soft == kVainRedos) look = Look::kEvery;
                    }
                    if (test) {  // turn by turn
                        const uint32_t j1 = min(j0, kn);
                        int was = 0, is = 0;  // this thread's live particles
#pragma unroll
                        for (int j = 0; j < K; ++j) was += live[j] ? 1 : 0;
                        for (uint32_t kk = j0 - B; warp_live && kk < j1; ++kk)
                            turn_all<ARITH, OCT, REV, K>(c, bar, mu,
                                                         staged_record(rec, kn, kk, REV), k0 + kk,
                                                         p, id, live, warp_live);
#pragma unroll
                        for (int j = 0; j < K; ++j) is += live[j] ? 1 : 0;
                        if (!__any_sync(kFullMask, was != is) && ++vain == kVainRedos)
                            look = Look::kTest;
                    }
                    check = false;
                }
            }
        }
        // Every warp is done with this buffer (and knows whether any warp of
        // the block is still live or has given up waiting).
        const bool block_fault = __syncthreads_or(timed_out);
        const bool block_live = __syncthreads_or(warp_live);
        if (block_fault || !block_live) break;
        if (leader && st + 2 < n_stages) {
            dev::async_proxy_fence();
            issue(st + 2);
        }
    }
    // Copies still in flight must land before the block's shared memory is
    // released: the one issued for stage st + 1 and, after a wait that gave
    // up, the one of stage st itself.  These waits are bounded too.
    const bool gave_up = __syncthreads_or(timed_out);
    if (gave_up && st < n_stages) dev::mbar_wait(&full[st & 1u], (st >> 1) & 1u);
    if (st + 1 < n_stages) {
        const uint32_t nx = st + 1;
        if (!dev::mbar_wait(&full[nx & 1u], (nx >> 1) & 1u)) timed_out = true;
    }
    const bool fault = __syncthreads_or(timed_out);
    if (fault && leader && c.fault) atomicOr(c.fault, 1u);
    return !fault;
}

// ---- kicked turns --------------------------------------------------------------
// The kicks do not depend on the orbit, so a warp makes those of kKickTurns
// turns of its 32 particles together and then runs the turns.  Each kick
// takes the first point of each of two attempts' sequences that lies in the
// unit disc (dev::kick_direction), 1.5 Philox blocks on average; with the
// rejection loop inside the turn a warp waited for its slowest lane, 3.6
// blocks a turn.  Here every lane makes the first attempt of its own kicks,
// the rejected ones (38 %) go to a list, and each further attempt is made for
// the whole list by full warps: 1.9 blocks a turn.
//
// 262,144 particles x 2,000 turns, mu = 0.2: 10.0 ms before, 6.4 now, 66 % of
// the issue slots and 37 % of the FP64 pipe busy; 299 instructions per warp
// and turn (421 before), about half of them the generator's.  Groups of 4
// turns 7.5 ms, of 16 6.8 (fewer warps fit).  A last group of fewer turns
// makes their kicks only (9 turns of 262,144 particles 49.7 -> 38.9 us).
//
// Shared memory of a warp: the points (then the kicks) of its turns, the list,
// the particles' indices and the turns' records.
constexpr uint32_t kKickTurns = 8;
// Turns of a chunk from which groups pay: a single turn's kicks are made by
// each lane for itself (262,144 particles, us for one turn: 9.3 so, 11.8 as a
// group of one; for two turns 14.8 as a group, 14.5 so).
constexpr uint32_t kKickGroup = 2;

struct KickShared {
    double2 a[kKickTurns * 32], b[kKickTurns * 32];  // {u1, u2}, {u3, u4} of [turn][lane]
    double2 rec[2 * kKickTurns];
    uint16_t list[kKickTurns * 32];
    uint32_t id[32];
};

// One attempt at the kick of (turn, id): keeps the point of each disc that
// has none yet; `got` holds bit 0 (first disc) and bit 1.
__device__ __forceinline__ uint32_t kick_attempt(uint32_t k0, uint32_t k1, uint32_t id,
                                                 uint32_t turn, uint32_t attempt, uint32_t got,
                                                 double2 *a, double2 *b) {
    const uint4 r = dev::philox4x32_10(make_uint4(turn, attempt, id, 0u), k0, k1);
    const double a1 = dev::kick_uniform(r.x), a2 = dev::kick_uniform(r.y);
    const double a3 = dev::kick_uniform(r.z), a4 = dev::kick_uniform(r.w);
    const bool in1 = dev::in_disc(Rn::add(Rn::mul(a1, a1), Rn::mul(a2, a2)));
    const bool in2 = dev::in_disc(Rn::add(Rn::mul(a3, a3), Rn::mul(a4, a4)));
    if (in1 && !(got & 1u)) *a = make_double2(a1, a2);
    if (in2 && !(got & 2u)) *b = make_double2(a3, a4);
    return got | (in1 ? 1u : 0u) | (in2 ? 2u : 0u);
}

// The kicks (direction times module) of the turns with table indices
// t0, t0 + dt, ... (kn of them) of the warp's live particles.
__device__ __forceinline__ void make_kicks(KickShared &w, const TrackChunk &c, uint32_t id,
                                           bool live, uint32_t t0, int dt, uint32_t kn) {
    const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint32_t k0 = uint32_t(c.kick_seed), k1 = uint32_t(c.kick_seed >> 32);
    uint32_t n_list = 0;
    auto first = [&](uint32_t u) {
        const uint32_t slot = u * 32u + lane;
        // what kick_direction falls back to when no attempt gives a point
        w.a[slot] = make_double2(0.0, 0.0);
        w.b[slot] = make_double2(1.0, 0.0);
        const uint32_t got =
            kick_attempt(k0, k1, id, t0 + uint32_t(int(u) * dt), 0u, 0u, &w.a[slot], &w.b[slot]);
        const bool more = live && got != 3u;
        const unsigned m = __ballot_sync(kFullMask, more);
        if (more) w.list[n_list + __popc(m & below)] = uint16_t(slot | (got << 14));
        n_list += __popc(m);
    };
    if (kn == kKickTurns) {
#pragma unroll 4
        for (uint32_t u = 0; u < kKickTurns; ++u) first(u);
    } else {
#pragma unroll 1
        for (uint32_t u = 0; u < kn; ++u) first(u);
    }
    for (uint32_t at = 1; n_list > 0u && at < dev::kKickAttempts; ++at) {
        __syncwarp();
        uint32_t left = 0;
        for (uint32_t base = 0; base < n_list; base += 32u) {
            const bool mine = base + lane < n_list;
            uint32_t e = mine ? w.list[base + lane] : 0u;
            __syncwarp();  // read before the entries kept are written over it
            bool more = false;
            if (mine) {
                const uint32_t slot = e & 0x3fffu;
                const uint32_t got = kick_attempt(k0, k1, w.id[slot & 31u],
                                                  t0 + uint32_t(int(slot >> 5) * dt), at, e >> 14,
                                                  &w.a[slot], &w.b[slot]);
                more = got != 3u;
                e = slot | (got << 14);
            }
            const unsigned m = __ballot_sync(kFullMask, more);
            if (more) w.list[left + __popc(m & below)] = uint16_t(e);
            left += __popc(m);
        }
        n_list = left;
    }
    __syncwarp();
    // (u1, u2, u3 f, u4 f), f = sqrt((1 - s1) / s2), times the module
    const double km = c.kick_module;
    auto scale = [&](uint32_t u) {
        const double2 a = w.a[u * 32u + lane], b = w.b[u * 32u + lane];
        const double s1 = Rn::add(Rn::mul(a.x, a.x), Rn::mul(a.y, a.y));
        const double s2 = Rn::add(Rn::mul(b.x, b.x), Rn::mul(b.y, b.y));
        const double f = __dsqrt_rn(Rn::div(Rn::sub(1.0, s1), s2));
        w.a[u * 32u + lane] = make_double2(Rn::mul(a.x, km), Rn::mul(a.y, km));
        w.b[u * 32u + lane] = make_double2(Rn::mul(Rn::mul(b.x, f), km), Rn::mul(Rn::mul(b.y, f), km));
    };
    if (kn == kKickTurns) {
#pragma unroll 4
        for (uint32_t u = 0; u < kKickTurns; ++u) scale(u);
    } else {
#pragma unroll 1
        for (uint32_t u = 0; u < kn; ++u) scale(u);
    }
}

// Adds (forward) or subtracts (backward) a kick and refreshes the squares.
template <bool SUB>
__device__ __forceinline__ void add_kick(Particle &p, double2 a, double2 b) {
    if (SUB) {
        p = dev::make_particle(Rn::sub(p.x, a.x), Rn::sub(p.px, a.y), Rn::sub(p.y, b.x),
                               Rn::sub(p.py, b.y));
    } else {
        p = dev::make_particle(Rn::add(p.x, a.x), Rn::add(p.px, a.y), Rn::add(p.y, b.x),
                               Rn::add(p.py, b.y));
    }
}

// Particle `id`, lost in turn k of the chunk.
template <bool REV>
__device__ __forceinline__ void lose(const TrackChunk &c, uint32_t id, bool &live, uint32_t k) {
    c.ux[id] = quiet_nan();
    c.upx[id] = quiet_nan();
    c.uy[id] = quiet_nan();
    c.upy[id] = quiet_nan();
    c.usteps[id] = REV ? c.turn0 - k : c.turn0 + k;
    live = false;
}

// A chunk of fewer than kKickGroup turns with kicks: each lane makes its own.
template <int ARITH, bool OCT, bool REV>
__device__ __forceinline__ void turns_kicked_few(const TrackChunk &c, const Barrier &bar,
                                                 Particle &p, uint32_t id, bool &live) {
    for (uint32_t k = 0; live && k < c.n_turns; ++k) {
        const uint32_t t = REV ? c.turn0 - 1u - k : c.turn0 + k;
        const dev::KickDirection d = dev::kick_direction(c.kick_seed, id, t);
        if (!REV) dev::apply_kick<false>(p, d, c.kick_module);
        dev::turn<ARITH, OCT, REV>(p, dev::load_turn(c.table, t), c.mu);
        if (REV) dev::apply_kick<true>(p, d, c.kick_module);
        if (!dev::inside_after_turn<ARITH>(p, bar)) lose<REV>(c, id, live, k);
    }
}

// The chunk's turns with kicks (one particle per thread): groups of
// kKickTurns turns, redone with the per-turn test where a live particle's
// coordinate reached the bound.  A lost particle's registers move with the
// kicks of its slot; nothing reads them.
template <int ARITH, bool OCT, bool REV>
__device__ __forceinline__ void turns_kicked(const TrackChunk &c, const Barrier &bar,
                                             Particle &p, uint32_t id, bool &live,
                                             bool warp_live) {
    const double mu = c.mu;
    extern __shared__ __align__(128) double stage_buf[];
    KickShared &w = reinterpret_cast<KickShared *>(stage_buf)[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    w.id[lane] = id;
    auto turn = [&](uint32_t u) {
        const double2 a = w.a[u * 32u + lane], b = w.b[u * 32u + lane];
        const double2 r = w.rec[2u * u], t = w.rec[2u * u + 1u];
        if (!REV) add_kick<false>(p, a, b);
        dev::turn<ARITH, OCT, REV>(p, Turn{r.x, r.y, t.x, t.y}, mu);
        if (REV) add_kick<true>(p, a, b);
    };
    for (uint32_t k0 = 0; warp_live && k0 < c.n_turns; k0 += kKickTurns) {
        const uint32_t kn = min(kKickTurns, c.n_turns - k0);
        const uint32_t t0 = REV ? c.turn0 - 1u - k0 : c.turn0 + k0;
        if (lane < 2u * kn) {  // half `lane & 1` of the record of turn lane / 2
            const uint32_t t = REV ? t0 - (lane >> 1) : t0 + (lane >> 1);
            w.rec[lane] = __ldg(reinterpret_cast<const double2 *>(c.table) + 2u * size_t(t) +
                                (lane & 1u));
        }
        __syncwarp();
        make_kicks(w, c, id, live, t0, REV ? -1 : 1, kn);
        __syncwarp();
        const Particle from = p;
        float big = 0.0f;
        auto look = [&]() { big = dev::hi_max(dev::hi_max(big, p.x, p.px), p.y, p.py); };
        if (kn == kKickTurns) {
#pragma unroll
            for (uint32_t u = 0; u < kKickTurns; ++u) {
                turn(u);
                look();
            }
        } else {
            for (uint32_t u = 0; u < kn; ++u) {
                turn(u);
                look();
            }
        }
        const bool over = live && (__float_as_uint(big) & 0x7fffffffu) >= bar.small_hi;
        if (__any_sync(kFullMask, over)) {
            p = from;
            for (uint32_t u = 0; u < kn; ++u) {
                turn(u);
                if (live && !dev::inside_after_turn<ARITH>(p, bar)) lose<REV>(c, id, live, k0 + u);
            }
            warp_live = __any_sync(kFullMask, live);
        }
        if (!live) p = dev::make_particle(0.0, 0.0, 0.0, 0.0);
        __syncwarp();
    }
}

// One chunk of turns for the particles of one block (K per thread).
template <int ARITH, bool OCT, bool REV, int K, bool STAGED, bool KICK>
__device__ __forceinline__ void track_chunk(const TrackChunk &c) {
    const uint32_t n_in = c.in_count ? *c.in_count : c.n_user;
    const uint32_t base = blockIdx.x * (blockDim.x * K);
    if (base >= n_in) return;  // whole block past the list

    Particle p[K];
    uint32_t id[K];
    bool live[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const uint32_t e = base + j * blockDim.x + threadIdx.x;
        double x = 0.0, px = 0.0, y = 0.0, py = 0.0;
        live[j] = e < n_in;
        id[j] = e;
        if (live[j]) {
            if (c.in_idx) {
                id[j] = c.in_idx[e];
                x = c.in_x[e];
                px = c.in_px[e];
                y = c.in_y[e];
                py = c.in_py[e];
            } else {
                x = c.ux[e];
                px = c.upx[e];
                y = c.uy[e];
                py = c.upy[e];
                // check_nan (src/henon.cu:118-121): a NaN particle is left
                // untouched, steps included.
                live[j] = !(isnan(x) || isnan(px) || isnan(y) || isnan(py));
            }
        }
        // Slots without a live particle hold zeros, a fixed point of the map.
        if (!live[j]) x = px = y = py = 0.0;
        p[j] = dev::make_particle(x, px, y, py);
    }

    const Barrier bar = dev::make_barrier<ARITH>(c.b2bits);
    bool thread_live = false;
#pragma unroll
    for (int j = 0; j < K; ++j) thread_live |= live[j];
    const bool warp_live = __any_sync(kFullMask, thread_live);
    if constexpr (KICK) {
        static_assert(K == 1, "kicked turns run one particle per thread");
        // STAGED: the kicks of a group of turns in shared memory
        if constexpr (STAGED)
            turns_kicked<ARITH, OCT, REV>(c, bar, p[0], id[0], live[0], warp_live);
        else
            turns_kicked_few<ARITH, OCT, REV>(c, bar, p[0], id[0], live[0]);
    } else if (STAGED) {
        if (!turns_staged<ARITH, OCT, REV, K>(c, bar, p, id, live, warp_live)) return;
    } else {
        turns_direct<ARITH, OCT, REV, K>(c, bar, p, id, live, warp_live);
    }

    if (c.out_idx == nullptr) {
        // Last chunk: survivors go back to the caller's arrays.
#pragma unroll
        for (int j = 0; j < K; ++j) {
            if (live[j]) {
                const uint32_t i = id[j];
                c.ux[i] = p[j].x;
                c.upx[i] = p[j].px;
                c.uy[i] = p[j].y;
                c.upy[i] = p[j].py;
                c.usteps[i] = c.steps_final;
            }
        }
        return;
    }
    // Re-compaction: each warp appends its survivors to the next list with
    // one atomic per slot; order inside a warp is preserved.
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const unsigned m = __ballot_sync(kFullMask, live[j]);
        if (m == 0u) continue;
        const int leader = __ffs(m) - 1;
        uint32_t off = 0;
        if (lane == unsigned(leader)) off = atomicAdd(c.out_count, uint32_t(__popc(m)));
        off = __shfl_sync(kFullMask, off, leader);
        if (live[j]) {
            const uint32_t o = off + __popc(m & ((1u << lane) - 1u));
            c.out_idx[o] = id[j];
            c.out_x[o] = p[j].x;
            c.out_px[o] = p[j].px;
            c.out_y[o] = p[j].y;
            c.out_py[o] = p[j].py;
        }
    }
}

// Up to 128 registers, two blocks of 256 threads per SM: FP64 results are
// ready after 8 cycles and one instruction keeps the pipe busy for two, so
// two warps per scheduler nearly fill it and what counts is that ptxas has
// the registers to load the records of the next turns ahead.  Cycles per
// warp and turn with 1, 2, 4 and 8 warps per scheduler, one particle per
// thread (the FP64 instructions alone: 38 / 66):
//     exact, mu = 0      56.4  48.4  45.5  44.3   (before: 69.9  53.2  50.9  48.9)
//     exact, mu != 0     80.7  74.8  72.7  71.6   (before: 91.9  79.9  76.4  74.6)
// Before: per-turn looks, runs of 32 turns, 64 registers.  With 64 registers
// the blocks of turns took 68.3, 48.8, 47.1 and 44.9 at mu = 0.  The kernels
// that read the records from global memory run a few turns: 64 registers,
// for twice the loads in flight.
template <int ARITH, bool OCT, bool REV, int K, bool STAGED>
__global__ void __launch_bounds__(256, K <= 2 ? (STAGED ? 2 : 4) : 1) track_chunk_kernel(const TrackChunk c) {
    track_chunk<ARITH, OCT, REV, K, STAGED, false>(c);
}

// 80 registers: six blocks of 128 threads, as many as the shared memory holds
// (with 96, five: 6.74 against 6.40 ms).
template <int ARITH, bool OCT, bool REV>
__global__ void __launch_bounds__(256, 3) track_kicked_kernel(const TrackChunk c) {
    track_chunk<ARITH, OCT, REV, 1, true, true>(c);
}

template <int ARITH, bool OCT, bool REV>
__global__ void __launch_bounds__(256, 4) track_kicked_few_kernel(const TrackChunk c) {
    track_chunk<ARITH, OCT, REV, 1, false, true>(c);
}

// Dynamic plus static shared memory above 48 KB needs the opt-in (the
// staged kernels' static part is their two mbarriers).
template <class Kernel>
cudaError_t allow_smem(Kernel kernel, size_t smem) {
    if (smem <= 40u * 1024u) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
}

template <int ARITH, bool OCT, bool REV, int K>
cudaError_t launch_s(const TrackChunk &c, unsigned blocks, int threads, cudaStream_t s) {
    if (c.stage_turns == 0) {
        track_chunk_kernel<ARITH, OCT, REV, K, false><<<blocks, threads, 0, s>>>(c);
    } else {
        const size_t smem = staged_smem_bytes(c.stage_turns, uint32_t(threads), K);
        auto kernel = track_chunk_kernel<ARITH, OCT, REV, K, true>;
        const cudaError_t e = allow_smem(kernel, smem);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, smem, s>>>(c);
    }
    return cudaGetLastError();
}

constexpr uint64_t kMinBlocksPerSm = 2u;

template <int ARITH, bool OCT, bool REV>
cudaError_t launch_k(const TrackChunk &c, const TrackLaunch &l, uint32_t n_upper,
                     cudaStream_t s) {
    int threads = l.threads;
    if (!isnan(c.kick_module)) {
        const unsigned blocks = unsigned((uint64_t(n_upper) + threads - 1) / threads);
        if (blocks == 0) return cudaSuccess;
        if (c.n_turns < kKickGroup) {
            track_kicked_few_kernel<ARITH, OCT, REV><<<blocks, threads, 0, s>>>(c);
            return cudaGetLastError();
        }
        const size_t smem = size_t(threads / 32) * sizeof(KickShared);
        auto kernel = track_kicked_kernel<ARITH, OCT, REV>;
        const cudaError_t e = allow_smem(kernel, smem);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, smem, s>>>(c);
        return cudaGetLastError();
    }
    // Several particles per thread add instruction-level parallelism once
    // the device is full; a short list would instead leave SMs idle (a
    // particle is one serial chain of turns whatever its thread holds), so
    // K is halved while the grid would give fewer than two blocks per SM.
    // A launch that reads its records from global memory runs few turns and
    // waits for its loads: at least two particles per thread then, from
    // three blocks per SM on (us for 8 turns with one and two, mu = 0:
    // 90,000 particles 4.1 and 4.3, 262,144 7.6 and 6.2, 1,048,576 23.7 and
    // 18.3; for 16 turns at mu = 0.2: 6.7 / 7.2, 14.9 / 13.1, 51.2 / 43.9).
    const bool direct = c.stage_turns == 0;
    int K = direct ? std::max(l.per_thread, 2) : l.per_thread;
    const uint64_t sms = uint64_t(sm_count());
    const uint64_t min_blocks = kMinBlocksPerSm * sms;
    const uint64_t pair_blocks = direct ? 3u * sms : min_blocks;
    while (K > 1 && (uint64_t(n_upper) + uint64_t(threads) * K - 1) / (uint64_t(threads) * K) <
                        pair_blocks)
        K /= 2;
    // Likewise smaller blocks: they spread a short list more evenly (40,000
    // particles in blocks of 128 give some SMs three blocks, most two).  A
    // few turns do not pay for starting more SMs (1,024 particles, one turn:
    // 2.1 us in blocks of 32, 1.8 in blocks of 128).
    while (!direct && threads > 32 && threads % 64 == 0 &&
           (uint64_t(n_upper) + uint64_t(threads) * K - 1) / (uint64_t(threads) * K) < min_blocks)
        threads /= 2;
    const uint64_t per_block = uint64_t(threads) * uint64_t(K);
    const unsigned blocks = unsigned((uint64_t(n_upper) + per_block - 1) / per_block);
    if (blocks == 0) return cudaSuccess;
    switch (K) {
        case 1: return launch_s<ARITH, OCT, REV, 1>(c, blocks, threads, s);
        case 2: return launch_s<ARITH, OCT, REV, 2>(c, blocks, threads, s);
        case 4: return launch_s<ARITH, OCT, REV, 4>(c, blocks, threads, s);
        default: return cudaErrorInvalidValue;
    }
}

template <int ARITH>
cudaError_t launch_a(const TrackChunk &c, const TrackLaunch &l, uint32_t n, cudaStream_t s) {
    if (l.octupole)
        return l.reverse ? launch_k<ARITH, true, true>(c, l, n, s)
                         : launch_k<ARITH, true, false>(c, l, n, s);
    return l.reverse ? launch_k<ARITH, false, true>(c, l, n, s)
                     : launch_k<ARITH, false, false>(c, l, n, s);
}

// ---- observables ------------------------------------------------------------
// GPU getters of particles_4d_gpu (src/henon.cu:67-111): computed for every
// entry, NaN particles give NaN.  Sums are left to right, separately rounded.
__global__ void observable_kernel(const double *x, const double *px,
                                  const double *y, const double *py, double *out,
                                  size_t n, int kind) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = x[i], b = px[i], c = y[i], d = py[i];
    double v;
    switch (kind) {
        case HM_OBS_RADIUS:
            v = sqrt(Rn::add(Rn::add(Rn::add(Rn::mul(a, a), Rn::mul(b, b)), Rn::mul(c, c)),
                             Rn::mul(d, d)));
            break;
        case HM_OBS_ACTION:
            v = Rn::add(Rn::add(Rn::add(Rn::mul(a, a), Rn::mul(b, b)), Rn::mul(c, c)),
                        Rn::mul(d, d));
            break;
        case HM_OBS_ACTION_X: v = Rn::add(Rn::mul(a, a), Rn::mul(b, b)); break;
        case HM_OBS_ACTION_Y: v = Rn::add(Rn::mul(c, c), Rn::mul(d, d)); break;
        case HM_OBS_ANGLE_X: v = atan2(b, a); break;
        default: v = atan2(d, c); break;
    }
    out[i] = v;
}

// ---- FP64 peak ---------------------------------------------------------------
// Eight independent FMA chains per thread; the denominator of the FP64
// roofline (an FMA counts as two flops).
__global__ void __launch_bounds__(256) fp64_peak_kernel(double *sink, int iters,
                                                         double m, double a) {
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 1.0 + 1e-3 * (threadIdx.x + j);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = fma(v[j], m, a);
        }
    }
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[j];
    if (s == 12345.678) sink[blockIdx.x] = s;  // never true; keeps the chains live
}

}  // namespace

cudaError_t launch_track_chunk(const TrackChunk &c, const TrackLaunch &l,
                               uint32_t n_in_upper, cudaStream_t s) {
    if (l.threads <= 0 || l.threads > 256 || (l.threads & 31) != 0)
        return cudaErrorInvalidValue;
    return l.arith == HM_ARITH_FAST ? launch_a<HM_ARITH_FAST>(c, l, n_in_upper, s)
                                    : launch_a<HM_ARITH_EXACT>(c, l, n_in_upper, s);
}

cudaError_t launch_observable(const double *x, const double *px, const double *y,
                              const double *py, double *out, size_t n, int kind,
                              cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const unsigned blocks = unsigned((n + 255) / 256);
    observable_kernel<<<blocks, 256, 0, s>>>(x, px, y, py, out, n, kind);
    return cudaGetLastError();
}

cudaError_t launch_fp64_peak(double *sink, int blocks, int threads, int iters,
                             cudaStream_t s, double *flops) {
    fp64_peak_kernel<<<blocks, threads, 0, s>>>(sink, iters, 0.9999999, 1e-7);
    *flops = double(blocks) * threads * double(iters) * 16.0 * 8.0 * 2.0;
    return cudaGetLastError();
}

}  // namespace hm
