// Host side of the libm calibration: builds the fp64 helper table for the
// log candidate and turns (candidate, host libm) pairs into flip bitmaps and
// per-region filter thresholds.  See rng.cuh for the scheme.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include <string>
#include <thread>
#include <vector>

#include "rng.cuh"

namespace hses {

constexpr uint32_t kUnits = 1u << 24;

// 64 x {1/c, log c}; c is the centre of each sub-interval of [0.75, 1.5)
// except the two that touch 1.0, where c = 1 (log c = 0, z*1 - 1 exact).
inline void build_log_table(double* tab /* 128 doubles */) {
    for (int j = 0; j < 64; ++j) {
        double c;
        if (j == 31 || j == 32) c = 1.0;
        else if (j < 32) c = 0.75 + (j + 0.5) / 128.0;
        else c = 1.0 + (j - 32 + 0.5) / 64.0;
        tab[2 * j] = 1.0 / c;
        tab[2 * j + 1] = (c == 1.0) ? 0.0 : log(c);
    }
}

struct CalibResult {
    std::vector<uint32_t> flip;   // 2^24 bits
    uint32_t delta[256];
    uint64_t n_flips = 0;
    uint32_t max_dist = 0;        // largest distance-from-midpoint among flipped inputs
    std::string error;            // non-empty when a candidate is not a neighbour of libm
};

// bits[i] is the rounded candidate and code[i] = dist | (rounded_up << 31) as
// produced by round_candidate(); want(i) is the host libm value for input i.
// `first` skips inputs the device handles separately (i = 0 for the logarithm).
template <class Want>
inline void calibrate(const uint32_t* cand_bits, const uint32_t* cand_code, uint32_t first,
                      Want want, CalibResult& out) {
    out.flip.assign(kUnits / 32, 0u);
    for (int r = 0; r < 256; ++r) out.delta[r] = 0;
    unsigned nt = std::thread::hardware_concurrency();
    if (nt == 0) nt = 1;
    if (nt > 16) nt = 16;
    // regions (top byte of the input) are split across threads: every thread
    // owns whole 32-bit words of the bitmap and whole entries of delta.
    std::vector<std::thread> pool;
    std::vector<uint64_t> flips(nt, 0);
    std::vector<uint32_t> maxd(nt, 0);
    std::vector<std::string> errs(nt);
    for (unsigned t = 0; t < nt; ++t) {
        pool.emplace_back([&, t]() {
            for (uint32_t region = t; region < 256; region += nt) {
                uint32_t d = 0;
                for (uint32_t i = region << 16; i < ((region + 1) << 16); ++i) {
                    if (i < first) continue;
                    float w = want(i);
                    uint32_t wb;
                    memcpy(&wb, &w, 4);
                    if (wb == cand_bits[i]) continue;
                    uint32_t alt = (cand_code[i] >> 31) ? cand_bits[i] - 1u : cand_bits[i] + 1u;
                    uint32_t dist = cand_code[i] & 0x7fffffffu;
                    if (wb != alt) {
                        if (errs[t].empty())
                            errs[t] = "libm calibration: candidate for input " + std::to_string(i) +
                                      " is not adjacent to the host libm value";
                        continue;
                    }
                    out.flip[i >> 5] |= 1u << (i & 31u);
                    ++flips[t];
                    if (dist + 1 > d) d = dist + 1;
                }
                out.delta[region] = d;
                if (d > maxd[t]) maxd[t] = d;
            }
        });
    }
    for (auto& th : pool) th.join();
    for (unsigned t = 0; t < nt; ++t) {
        out.n_flips += flips[t];
        if (maxd[t] > out.max_dist) out.max_dist = maxd[t];
        if (out.error.empty() && !errs[t].empty()) out.error = errs[t];
    }
}

// ---- the kernels' fp32 candidate (NoiseCal) -----------------------------------------------------------------
// Rows of the two tables (the log rows' filter width left at 0).  log: 1/c rounded to eight bits and the logarithm of
// exactly that value, its high part on a grid of 2^-18.  cos: t near the middle of the row's interval where cos t and sin t
// lie unusually close to fp32 values (Gal's accurate tables); the intervals at the two zeros of the cosine use the
// zero itself, so that the distance to it, and with it the result, is accurate relative to its size.
inline void build_noise_tables(float4* log_tab /* kLogRows */, float4* cos_tab /* kCosRows */) {
    for (int j = 0; j < kLogRows; ++j) {
        double c;
        if (j == 31 || j == 32) c = 1.0;
        else if (j < 32) c = 0.75 + (j + 0.5) / 128.0;
        else c = 1.0 + (j - 32 + 0.5) / 64.0;
        const float inv = (float)(nearbyint(128.0 / c) / 128.0);   // eight bits: r = z/c - 1 then loses at most one bit
        const double l = inv == 1.0f ? 0.0 : -log((double)inv);
        const double hi = nearbyint(l * 262144.0) / 262144.0;
        log_tab[j] = float4{(float)((double)inv / 16777216.0), (float)hi, (float)(l - hi), 0.0f};
    }
    const double pi = 3.14159265358979323846;
    for (int k = 0; k < kCosRows; ++k) {
        const bool zero = k == 63 || k == 64 || k == 191 || k == 192;
        float t = (float)(zero ? (k < 128 ? 0.5 : 1.5) * pi : 2.0 * pi * (k + 0.5) / 256.0);
        if (!zero) {
            const uint32_t t0 = f2u(t);
            double best = 1e9;
            for (int s = -2000; s <= 2000; ++s) {
                const float c = u2f(t0 + (uint32_t)s);
                const double e = fabs(sin((double)c) - (double)(float)sin((double)c));
                if (e < best) {
                    best = e;
                    t = c;
                }
            }
        }
        const double ct = cos((double)t), st = sin((double)t);
        const float c = zero ? 0.0f : (float)ct;
        cos_tab[k] = float4{t, c, (float)st, (float)(ct - (double)c)};
    }
}

struct NoiseCalResult {
    std::vector<uint32_t> flip;     // 2^24 bits: 1 where the host value is the second rounding
    std::vector<float> width;       // filter width per table row, relative to hi
    uint64_t in_doubt = 0;          // inputs whose two roundings differ
    std::string error;
};
// hi[i], lo[i]: the candidate of every input; row_of(i) its table row; want(i) the host libm.  A row's width is the
// largest relative distance at which the host rounds to the other side of the boundary next to hi + lo, raised
// until every input of the row has the host's value among its two roundings.
template <class RowOf, class Want>
inline void calibrate_noise(const float* hi, const float* lo, int rows, RowOf row_of, Want want, NoiseCalResult& out) {
    unsigned nt = std::thread::hardware_concurrency();
    nt = nt == 0 ? 1 : nt > 16 ? 16 : nt;
    auto parallel = [&](auto body) {
        std::vector<std::thread> pool;
        for (unsigned t = 0; t < nt; ++t)
            pool.emplace_back([&, t]() { body(t, (uint32_t)((uint64_t)kUnits / 32 * t / nt) * 32, (uint32_t)((uint64_t)kUnits / 32 * (t + 1) / nt) * 32); });
        for (auto& th : pool) th.join();
    };
    std::vector<float> host(kUnits);
    std::vector<std::vector<double>> need(nt, std::vector<double>(rows, 0.0));
    std::vector<int> far(nt, 0);
    parallel([&](unsigned t, uint32_t b, uint32_t e) {
        for (uint32_t i = b; i < e; ++i) {
            const float w = want(i), s = hi[i] + lo[i];
            host[i] = w;
            if (f2u(s) == f2u(w)) continue;
            if (w != nextafterf(s, w)) far[t] = 1;
            const double mid = 0.5 * ((double)s + (double)w), dist = fabs((double)hi[i] + (double)lo[i] - mid);
            double& n = need[t][row_of(i)];
            const double rel = dist / fabs((double)hi[i]);
            if (rel > n) n = rel;
        }
    });
    out.width.assign(rows, 0.0f);
    for (int r = 0; r < rows; ++r) {
        double n = 0.0;
        for (unsigned t = 0; t < nt; ++t) n = need[t][r] > n ? need[t][r] : n;
        out.width[r] = (float)(n * 1.0001 + 0x1p-44);
    }
    for (unsigned t = 0; t < nt; ++t)
        if (far[t]) out.error = "libm calibration: a candidate is not adjacent to the host libm value";
    out.flip.assign(kUnits / 32, 0u);
    std::vector<uint64_t> doubt(nt, 0);
    for (int round = 0; out.error.empty(); ++round) {
        std::vector<std::vector<uint8_t>> bad(nt, std::vector<uint8_t>(rows, 0));
        parallel([&](unsigned t, uint32_t b, uint32_t e) {
            doubt[t] = 0;
            for (uint32_t i = b; i < e; ++i) {
                const int r = row_of(i);
                float v0, v1;
                roundings(hi[i], lo[i], out.width[r], v0, v1);
                if (f2u(v0) != f2u(v1)) ++doubt[t];
                const uint32_t w = f2u(host[i]), bit = 1u << (i & 31u);
                if (w == f2u(v0)) out.flip[i >> 5] &= ~bit;
                else if (w == f2u(v1)) out.flip[i >> 5] |= bit;
                else bad[t][r] = 1;
            }
        });
        bool any = false;
        for (int r = 0; r < rows; ++r)
            for (unsigned t = 0; t < nt; ++t)
                if (bad[t][r]) {
                    out.width[r] = out.width[r] * 1.01f + 0x1p-40f;
                    any = true;
                    break;
                }
        if (!any) break;
        if (round == 40) out.error = "libm calibration: no filter width covers the host libm's values";
    }
    for (unsigned t = 0; t < nt; ++t) out.in_doubt += doubt[t];
}

// The two libm expressions the reference evaluates (noiser.rs:470-476).
inline float host_logf_u24(uint32_t i) {
    float u = (float)i / 16777216.0f;
    return logf(fmaxf(u, 1e-9f));
}
inline float host_cosf_u24(uint32_t j) {
    float u = (float)j / 16777216.0f;
    return cosf(6.2831855f * u);
}

}  // namespace hses
