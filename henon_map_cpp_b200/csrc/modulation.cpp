// Host-side tune-modulation tables and Birkhoff weights.
//
// The per-turn rotation angles omega(n) and their sin/cos are computed on the
// host with the C library's libm, exactly as the reference does
// (src/modulation.cpp:3-134, src/henon.cu:2657-2694): the device only reads
// the resulting tables, so the expression order below is chosen to give
// bit-identical doubles to the reference on the same host.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <exception>
#include <random>
#include <string>
#include <thread>
#include <vector>

#include "hm_internal.h"

namespace hm {
namespace {

// Harmonics of the SPS power-converter ripple: coefficient c_j and angular
// frequency k_j * 2*pi/868.12 (src/modulation.cpp:13-29).  The constants
// are the physical model; they have to be the reference's values.
constexpr int kSpsHarmonics = 7;
constexpr double kSpsCoefficient[kSpsHarmonics] = {
    1.000e-4, 0.218e-4, 0.708e-4, 0.254e-4, 0.100e-4, 0.078e-4, 0.218e-4};
constexpr int kSpsMultiple[kSpsHarmonics] = {1, 2, 3, 6, 7, 10, 12};

// Runs body(lo, hi) over [0, n) in pieces of kPiece, dealt to the host's
// threads (this one among them) by a counter.  A thread that cannot be
// started is done without.  Starting one costs 20-30 us, as much as about a
// thousand turns' sines and cosines, so small ranges take few.
constexpr size_t kPiece = 1024;

template <class F> void parallel_pieces(size_t n, F body) {
    const size_t pieces = (n + kPiece - 1) / kPiece;
    // (asked once: it reads a file, 2 us of a table of one turn's 10)
    static const size_t hw = std::max<size_t>(1, std::thread::hardware_concurrency());
    std::atomic<size_t> next{0};
    auto work = [&] {
        for (size_t q; (q = next.fetch_add(1)) < pieces;)
            body(q * kPiece, std::min(n, (q + 1) * kPiece));
    };
    std::vector<std::thread> pool;
    try {
        while (pool.size() + 1 < std::min(hw, pieces)) pool.emplace_back(work);
    } catch (const std::exception &) {
    }
    work();
    for (auto &th : pool) th.join();
}

// The SPS ripple sum_j c_j cos(Omega_j * turn), harmonics summed in
// ascending j (sps_modulation, src/modulation.cpp:31-60).
struct SpsRipple {
    double omega_k[kSpsHarmonics];
    SpsRipple() {
        const double fundamental = 2 * M_PI / 868.12;
        for (int j = 0; j < kSpsHarmonics; ++j) omega_k[j] = double(kSpsMultiple[j]) * fundamental;
    }
    double operator()(double turn) const {
        double ripple = 0.0;
        for (int j = 0; j < kSpsHarmonics; ++j)
            ripple += kSpsCoefficient[j] * std::cos(omega_k[j] * turn);
        return ripple;
    }
};

}  // namespace

// omega(n) = 2*pi*tune * (1 + eps * sum_j c_j cos(Omega_j * n)),
// n = start .. end-1, harmonics summed in ascending j
// (sps_modulation, src/modulation.cpp:31-60).
std::vector<double> sps_modulation(double tune, double epsilon, int32_t start,
                                   int32_t end) {
    std::vector<double> out(end > start ? size_t(end - start) : 0);
    const SpsRipple ripple;
    const double two_pi_tune = 2 * M_PI * tune;
    parallel_pieces(out.size(), [&](size_t lo, size_t hi) {
        // The reference adds an unsigned index to the int start: the turn
        // number is formed in 32-bit unsigned arithmetic.
        for (size_t i = lo; i < hi; ++i)
            out[i] = two_pi_tune *
                     (1 + epsilon * ripple(double(uint32_t(uint32_t(i) + uint32_t(start)))));
    });
    return out;
}

// omega(i) = 2*pi*tune * (1 + eps * cos(2*pi*omega*i)), i counted from 0
// (basic_modulation, src/modulation.cpp:3-11).
std::vector<double> basic_modulation(double tune, double omega, double epsilon,
                                     int32_t start, int32_t end) {
    std::vector<double> out(end > start ? size_t(end - start) : 0);
    const double two_pi_tune = 2 * M_PI * tune;
    const double two_pi_omega = 2 * M_PI * omega;
    for (size_t i = 0; i < out.size(); ++i)
        out[i] = two_pi_tune * (1 + epsilon * std::cos(two_pi_omega * int(i)));
    return out;
}

hm_status check_modulation(const std::string &kind, double omega_0) {
    if (kind != "sps" && kind != "basic" && kind != "none" && kind != "gaussian" &&
        kind != "uniform")
        return fail(HM_ERR_UNKNOWN_MODULATION, "Unknown modulation kind");
    if (kind == "basic" && std::isnan(omega_0))
        return fail(HM_ERR_INVALID_ARG, "basic modulation needs a finite omega_0");
    return ok();
}

hm_status modulation(const std::string &kind, uint32_t n_turns, double omega_x,
                     double omega_y, double omega_0, double epsilon,
                     uint32_t offset, std::vector<double> &wx,
                     std::vector<double> &wy) {
    HM_TRY(check_modulation(kind, omega_0));
    const int32_t start = int32_t(offset);
    const int32_t end = int32_t(offset + n_turns);
    if (kind == "sps") {
        wx = sps_modulation(omega_x, epsilon, start, end);
        wy = sps_modulation(omega_y, epsilon, start, end);
    } else if (kind == "basic") {
        wx = basic_modulation(omega_x, omega_0, epsilon, start, end);
        wy = basic_modulation(omega_y, omega_0, epsilon, start, end);
    } else if (kind == "none") {
        // The reference fills empty vectors (src/modulation.cpp:119-123) and
        // then reads past them; here the tables hold the constant angles.
        wx.assign(n_turns, omega_x);
        wy.assign(n_turns, omega_y);
    } else {  // gaussian, uniform
        // Random tunes drawn per turn (src/modulation.cpp:62-99): angle =
        // 2*pi*sample with sample ~ N(omega, eps) or U(omega, eps).
        std::random_device rd;
        auto draw = [&](double a, std::vector<double> &out) {
            std::mt19937 gen(rd());
            out.resize(n_turns);
            if (kind == "gaussian") {
                std::normal_distribution<double> dist(a, epsilon);
                for (auto &v : out) v = 2 * M_PI * dist(gen);
            } else {
                std::uniform_real_distribution<double> dist(a, epsilon);
                for (auto &v : out) v = 2 * M_PI * dist(gen);
            }
        };
        draw(omega_x, wx);
        draw(omega_y, wy);
    }
    return ok();
}

size_t table_turns(const std::string &kind, uint32_t n_turns, uint32_t offset) {
    if (kind != "sps" && kind != "basic") return n_turns;
    const int32_t start = int32_t(offset), end = int32_t(offset + n_turns);
    return end > start ? size_t(end - start) : 0;
}

// sin and cos of omega(n) with the host libm (src/henon.cu:2672-2686), for
// several tables at once on all host threads.  SPS angles are formed where
// their sines are taken, both planes from one ripple sum; the other kinds
// (two of them draw random tunes in order) are formed first.
hm_status turn_records(const std::vector<TableSpec> &specs) {
    std::vector<std::vector<double>> wx(specs.size()), wy(specs.size());
    std::vector<size_t> first(1, 0);
    for (size_t k = 0; k < specs.size(); ++k) {
        const TableSpec &t = specs[k];
        if (t.kind != "sps")
            HM_TRY(modulation(t.kind, t.n_turns, t.omega_x, t.omega_y, t.omega_0, t.epsilon,
                              t.offset, wx[k], wy[k]));
        first.push_back(first.back() + t.n_turns);
    }
    const SpsRipple ripple;
    parallel_pieces(first.back(), [&](size_t lo, size_t hi) {
        size_t k = size_t(std::upper_bound(first.begin(), first.end(), lo) - first.begin()) - 1;
        for (size_t g = lo; g < hi; ++g) {
            while (g >= first[k + 1]) ++k;
            const TableSpec &t = specs[k];
            const size_t i = g - first[k];
            double ox, oy;
            if (wx[k].empty()) {
                const double r = 1 + t.epsilon * ripple(double(uint32_t(uint32_t(i) + t.offset)));
                ox = 2 * M_PI * t.omega_x * r;
                oy = 2 * M_PI * t.omega_y * r;
            } else {
                ox = wx[k][i];
                oy = wy[k][i];
            }
            double *const rec = t.records + 4 * i;
            rec[0] = std::sin(ox);
            rec[1] = std::cos(ox);
            rec[2] = std::sin(oy);
            rec[3] = std::cos(oy);
        }
    });
    return ok();
}

// The ripple S_n of omega(n) = 2*pi*tune*(1 + eps*S_n) for the kinds whose
// angle is differentiable in (tune, eps): "sps" (the harmonic sum above) and
// "basic" (cos(2*pi*omega_0*i)).
hm_status modulation_ripple(const std::string &kind, uint32_t n_turns, double omega_0,
                            uint32_t offset, std::vector<double> &ripple) {
    ripple.assign(n_turns, 0.0);
    if (kind == "sps") {
        const SpsRipple sps;
        parallel_pieces(n_turns, [&](size_t lo, size_t hi) {
            for (size_t i = lo; i < hi; ++i) ripple[i] = sps(double(uint32_t(uint32_t(i) + offset)));
        });
        return ok();
    }
    if (kind == "basic") {
        const double two_pi_omega = 2 * M_PI * omega_0;
        for (uint32_t i = 0; i < n_turns; ++i) ripple[i] = std::cos(two_pi_omega * int(i));
        return ok();
    }
    return fail(HM_ERR_NOT_SUPPORTED,
                "derivatives need an 'sps' or 'basic' modulation (random tunes have none)");
}

// w_i = exp(-1/(t(1-t))), t = i/n, normalised by the left-to-right sum
// (birkhoff_weights, src/dynamic_indicator.cpp:63-79).
std::vector<double> birkhoff_weights(uint32_t n) {
    std::vector<double> w(n);
    for (uint32_t i = 0; i < n; ++i) {
        const double t = double(i) / double(n);
        w[i] = std::exp(-1 / (t * (1.0 - t)));
    }
    double sum = 0.0;
    for (double v : w) sum += v;
    for (double &v : w) v = v / sum;
    return w;
}

}  // namespace hm
