// Counter-style device RNG for the EggRoll noise factors.
//
// The reference draws every factor from a sequential xorshift64 stream
// (hyperscalees-noiser/src/noiser.rs:436-490) seeded by a 64-bit hash of
// (parameter key, epoch bucket, antithetic pair) (noiser.rs:495-506).  Here a
// thread lands anywhere in that stream with a GF(2) jump (the generator is a
// linear map on 64-bit states) and then regenerates normals in registers.
//
// The Box-Muller step calls the platform libm in the reference (Rust
// f32::ln / f32::cos lower to logf / cosf).  Those are not correctly rounded,
// so bit-exactness is obtained in two stages:
//   1. a deterministic fp64 "candidate" for logf(u) and cosf(TAU*u), built
//      from IEEE basic operations only (explicit fma/mul/add, no contraction),
//      rounded to fp32;
//   2. a per-context calibration that compares the candidate with the host
//      libm over all 2^24 possible uniforms and records, one bit per input,
//      where libm rounds to the other neighbour.  A cheap test filters out the
//      inputs that cannot be affected before the bitmap is consulted.
// The kernels run the same scheme on an fp32 candidate (NoiseCal below): a sum
// hi + lo of two fp32 values, 2^-30 and better relative to the result, and two
// roundings of it, hi + (lo +- c*hi), that differ for the few inputs in doubt.
// The functions below compile for host and device so the candidate math can
// be exercised on the CPU as well.
#pragma once

#include <stdint.h>
#include <string.h>
#include <math.h>

#if defined(__CUDACC__)
#define HSES_HD __host__ __device__ __forceinline__
#else
#define HSES_HD static inline
#endif

#if !defined(__CUDACC__)
struct double2 { double x, y; };
struct float4 { float x, y, z, w; };
#endif

namespace hses {

// ---------------------------------------------------------------------------
// bit casts and strictly rounded arithmetic
// ---------------------------------------------------------------------------
HSES_HD uint32_t f2u(float f) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u; memcpy(&u, &f, 4); return u;
#endif
}
HSES_HD float u2f(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f; memcpy(&f, &u, 4); return f;
#endif
}
HSES_HD uint64_t d2u(double d) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t u; memcpy(&u, &d, 8); return u;
#endif
}
HSES_HD double dfma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#else
    return fma(a, b, c);
#endif
}
HSES_HD double dmul(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
HSES_HD double dadd(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
HSES_HD float fmul(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
HSES_HD float fsqrt(float a) {
#if defined(__CUDA_ARCH__)
    return __fsqrt_rn(a);
#else
    return sqrtf(a);
#endif
}
HSES_HD float d2f_rn(double d) {
#if defined(__CUDA_ARCH__)
    return __double2float_rn(d);
#else
    return (float)d;
#endif
}

// ---------------------------------------------------------------------------
// seed hash and generator (noiser.rs:444-455, 495-506)
// ---------------------------------------------------------------------------
HSES_HD uint64_t noise_seed(uint64_t key, int32_t true_epoch, int32_t true_thread) {
    uint64_t h = key ^ 0x9E3779B97F4A7C15ull;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= (uint64_t)(int64_t)true_epoch * 0x94D049BB133111EBull;
    h = ((h << 17) | (h >> 47)) ^ (uint64_t)(int64_t)true_thread;
    h ^= h >> 33;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 29;
    h *= 0x94D049BB133111EBull;
    h ^= h >> 32;
    return h;
}

// One generator step (shifts 13, 7, 17).  On the device every 64-bit shift is
// written as 32x32->64 multiplications by a power of two: the product of a word
// with 2^s holds (word << s) in its low half and (word >> (32 - s)) in its high
// half, and multiplications issue on the FMA pipe, which this code leaves idle,
// instead of the integer pipe that bounds it.
HSES_HD uint64_t xs64_step(uint64_t x) {
#if defined(__CUDA_ARCH__)
    uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
    uint64_t m = (uint64_t)lo * 8192u;                 // x ^= x << 13
    uint32_t h = hi * 8192u;
    lo ^= (uint32_t)m;
    hi ^= h ^ (uint32_t)(m >> 32);
    uint64_t mh = (uint64_t)hi * 33554432u;            // x ^= x >> 7
    uint64_t ml = (uint64_t)lo * 33554432u;
    lo ^= (uint32_t)(ml >> 32) ^ (uint32_t)mh;
    hi ^= (uint32_t)(mh >> 32);
    m = (uint64_t)lo * 131072u;                        // x ^= x << 17
    h = hi * 131072u;
    lo ^= (uint32_t)m;
    hi ^= h ^ (uint32_t)(m >> 32);
    return ((uint64_t)hi << 32) | lo;
#else
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return x;
#endif
}

// eggroll.rs:60-65: noise_reuse==0 pins the epoch bucket to 0; members 2p and
// 2p+1 share the draw of pair p, the odd one with A negated.
HSES_HD int32_t true_epoch_of(int32_t epoch, int32_t noise_reuse) {
    return noise_reuse == 0 ? 0 : epoch / noise_reuse;
}

// ---------------------------------------------------------------------------
// GF(2) jump tables: one 64x64 matrix is stored as 16 nibble tables of 16
// entries (2 KB); applying it costs 16 lookups and xors.
// ---------------------------------------------------------------------------
constexpr int kJumpWords = 256;  // uint64 words per matrix

HSES_HD uint64_t jump_apply(const uint64_t* __restrict__ tab, uint64_t x) {
    uint64_t r = 0;
#pragma unroll
    for (int p = 0; p < 16; ++p) r ^= tab[p * 16 + (int)((x >> (4 * p)) & 15)];
    return r;
}

// Table 16 k + d advances the state by d * 16^k steps: a start state is a chain of dependent tables, one per non-zero
// hexadecimal digit of its position (with one per set bit the chain was twice as long).
HSES_HD uint64_t jump_by(const uint64_t* __restrict__ tabs, uint64_t x, uint64_t n) {
    for (int k = 0; n != 0; ++k, n >>= 4)
        if (n & 15) x = jump_apply(tabs + (size_t)(16 * k + (int)(n & 15)) * kJumpWords, x);
    return x;
}

// The 32 lanes of a warp from one common state to 32 equally spaced positions: the table holds, for every nibble
// value of the common state, the images for all lanes side by side (16 x 16 x 32 words), so that one round of
// coalesced reads does what up to log2(distance) dependent table lookups per lane would.
constexpr int kLaneWords = 16 * 16 * 32;
HSES_HD uint64_t lane_jump(const uint64_t* __restrict__ tab, uint64_t x, int lane) {
    uint64_t r = 0;
#pragma unroll
    for (int p = 0; p < 16; ++p) r ^= tab[(p * 16 + (int)((x >> (4 * p)) & 15)) * 32 + lane];
    return r;
}

// ---------------------------------------------------------------------------
// libm-conformant logf / cosf on the 24-bit uniforms
// ---------------------------------------------------------------------------
struct LibmCal {
    const double2* log_tab;      // 64 x {1/c, log c}
    const uint32_t* log_flip;    // 2^24 bits
    const uint32_t* cos_flip;    // 2^24 bits
    const uint32_t* log_delta;   // 256 thresholds on |low29 - 2^28|, by top byte of the input
    const uint32_t* cos_delta;   // 256 thresholds
    float log_of_zero;           // host logf(1e-9f), used when the uniform is 0
};

constexpr double kLn2 = 0x1.62e42fefa39efp-1;
constexpr double kPio2Hi = 0x1.921fb54442d10p+0;   // pi/2 to 49 bits: n*hi exact for n <= 15
constexpr double kPio2Lo = 0x1.08d313198a2e0p-49;  // pi/2 - hi
constexpr float kTauF = 6.2831855f;                // std::f32::consts::TAU

// fp64 value of log(i * 2^-24), i in [1, 2^24), accurate to ~2^-38 relative.
// z*2^k = u with z in [0.75, 1.5); 64 sub-intervals uniform in the fp32 bit
// pattern, the two that touch 1.0 use c = 1 so r = z - 1 is exact there.
HSES_HD double log_candidate(uint32_t i, const double2* __restrict__ tab) {
    float uf = (float)i * 5.9604644775390625e-08f;  // exact: i < 2^24, scale 2^-24
    uint32_t ix = f2u(uf);
    uint32_t tmp = ix - 0x3f400000u;
    int j = (int)((tmp >> 17) & 63u);
    int k = (int32_t)tmp >> 23;
    float zf = u2f(ix - (tmp & 0xff800000u));
    double2 e = tab[j];
    double r = dfma((double)zf, e.x, -1.0);
    double p = dfma(r, -1.0 / 6.0, 1.0 / 5.0);
    p = dfma(r, p, -1.0 / 4.0);
    p = dfma(r, p, 1.0 / 3.0);
    p = dfma(r, p, -1.0 / 2.0);
    p = dfma(dmul(r, r), p, r);              // r - r^2/2 + ... - r^6/6
    return dfma((double)k, kLn2, dadd(e.y, p));
}

// fp64 value of cos(theta) for an fp32 theta in [0, 2*pi], ~2^-44 relative.
// cos(t) = sin(t + pi/2) = (-1)^q sin(rho), rho = t - (2q-1)*pi/2 in [-pi/2, pi/2].
HSES_HD double cos_candidate(float theta) {
    int q = (int)(fmul(theta, 0.31830987f) + 1.0f);  // any q with |rho| <~ pi/2 + 1e-6 works
    double n = (double)(2 * q - 1);
    double rho = dfma(-n, kPio2Hi, (double)theta);
    rho = dfma(-n, kPio2Lo, rho);
    double s = dmul(rho, rho);
    double p = dfma(s, 1.0 / 355687428096000.0, -1.0 / 1307674368000.0);  // 1/17!, -1/15!
    p = dfma(s, p, 1.0 / 6227020800.0);                                  // 1/13!
    p = dfma(s, p, -1.0 / 39916800.0);                                   // -1/11!
    p = dfma(s, p, 1.0 / 362880.0);                                      // 1/9!
    p = dfma(s, p, -1.0 / 5040.0);                                       // -1/7!
    p = dfma(s, p, 1.0 / 120.0);                                         // 1/5!
    p = dfma(s, p, -1.0 / 6.0);                                          // -1/3!
    double v = dfma(dmul(rho, s), p, rho);
    return (q & 1) ? -v : v;
}

// Round an fp64 candidate to fp32 and report how the rounding went:
// low29 = discarded mantissa bits, alt = the neighbour on the other side of
// the rounding midpoint.
struct Rounded {
    uint32_t bits;   // round-to-nearest result
    uint32_t alt;    // the other bracketing fp32 value: bits + step
    uint32_t dist;   // |low29 - 2^28|: 0 at the midpoint, 2^28 on an fp32 value
    int32_t step;    // +1 or -1
};
HSES_HD Rounded round_candidate(double y) {
    // The rounding itself is the hardware's fp64 -> fp32 conversion (the conversion pipe is nearly idle
    // in this code, the integer pipe is what bounds it).  The other neighbour lies one step up in
    // magnitude when the discarded bits are below the midpoint and one step down otherwise.  An exact
    // midpoint would make that rule name the wrong neighbour for an even mantissa; the candidates
    // (logarithms and cosines of fp32 arguments) never are, and the calibration would refuse a
    // context in which the host's value is neither `bits` nor `alt`.
    Rounded r;
#if defined(__CUDA_ARCH__)
    const uint32_t low = (uint32_t)__double2loint(y) & 0x1fffffffu;
#else
    const uint32_t low = (uint32_t)(d2u(y) & 0x1fffffffull);
#endif
    r.bits = f2u(d2f_rn(y));
    r.step = low >= 0x10000000u ? -1 : 1;
    r.alt = r.bits + (uint32_t)r.step;
    r.dist = low >= 0x10000000u ? low - 0x10000000u : 0x10000000u - low;
    return r;
}

// bit (i mod 32) of a bitmap word
HSES_HD uint32_t bit_of(uint32_t word, uint32_t i) {
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(word, 0u, i) & 1u;   // the funnel shift takes its count modulo 32
#else
    return (word >> (i & 31u)) & 1u;
#endif
}

HSES_HD float apply_flip(const Rounded& r, uint32_t idx, const uint32_t* __restrict__ flip,
                         const uint32_t* __restrict__ delta) {
    uint32_t bits = r.bits;
    if (r.dist < delta[idx >> 16]) {
        if ((flip[idx >> 5] >> (idx & 31u)) & 1u) bits = r.alt;
    }
    return u2f(bits);
}

// logf(max(i*2^-24, 1e-9f)) as the host libm returns it.
HSES_HD float libm_logf_u24(uint32_t i, const LibmCal& cal) {
    if (i == 0) return cal.log_of_zero;
    return apply_flip(round_candidate(log_candidate(i, cal.log_tab)), i, cal.log_flip, cal.log_delta);
}
// cosf(TAU * j*2^-24) as the host libm returns it.
HSES_HD float libm_cosf_u24(uint32_t j, const LibmCal& cal) {
    float theta = fmul(kTauF, (float)j * 5.9604644775390625e-08f);
    return apply_flip(round_candidate(cos_candidate(theta)), j, cal.cos_flip, cal.cos_delta);
}

// noiser.rs:470-477: one standard normal from two consecutive generator outputs.
HSES_HD float normal_from_draws(uint64_t x1, uint64_t x2, const LibmCal& cal) {
    float lg = libm_logf_u24((uint32_t)(x1 >> 40), cal);
    float radius = fsqrt(fmul(-2.0f, lg));
    return fmul(radius, libm_cosf_u24((uint32_t)(x2 >> 40), cal));
}

HSES_HD float next_normal(uint64_t& state, const LibmCal& cal) {
    uint64_t x1 = xs64_step(state);
    uint64_t x2 = xs64_step(x1);
    state = x2;
    return normal_from_draws(x1, x2, cal);
}

// ---------------------------------------------------------------------------
// The kernels' form: fp32 candidates.  fp64 operations and conversions share narrow pipes with each other and
// with the tensor cores; here a normal is some 100 instructions, most of them on the full-rate fp32 pipe.
// ---------------------------------------------------------------------------
HSES_HD float ffma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return fmaf(a, b, c);
#endif
}
HSES_HD float fadd(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
HSES_HD float u2float(uint32_t v) {
#if defined(__CUDA_ARCH__)
    return __uint2float_rn(v);
#else
    return (float)v;
#endif
}
HSES_HD float i2float(int32_t v) {
#if defined(__CUDA_ARCH__)
    return __int2float_rn(v);
#else
    return (float)v;
#endif
}

constexpr int kLogRows = 64, kCosRows = 256;
struct NoiseCal {
    const float4* log_tab;      // kLogRows x {2^-24 / c, -log(1/c) high, low, filter width}
    const float4* cos_tab;      // kCosRows x {t, cos t, sin t, low part of cos t}
    const float* cos_width;     // kCosRows filter widths
    const uint32_t* log_flip;   // 2^24 bits: which of the two roundings the host libm returns
    const uint32_t* cos_flip;
};
// k * ln 2 in two parts; the factor 2^-23 undoes the scale of an exponent field read as an integer.  The high part
// has 18 bits, like the table's, so that their sum is exact.
constexpr float kLn2Hi = (float)(181704.0 / 262144.0 / 8388608.0);
constexpr float kLn2Lo = (float)((0x1.62e42fefa39efp-1 - 181704.0 / 262144.0) / 8388608.0);
constexpr float kUniform0 = 1e-9f * 16777216.0f;   // the reference raises u to 1e-9 (noiser.rs:471)

// row of the log table an input uses
HSES_HD int log_row(uint32_t i) {
    float uf = u2float(i);
    uf = uf > kUniform0 ? uf : kUniform0;
    return (int)(((f2u(uf) - 0x4b400000u) >> 17) & 63u);
}
// log(max(i 2^-24, 1e-9)) = hi + lo.  i = z 2^k with z in [0.75, 1.5) 2^24; the row's c divides z up to
// r = z/c - 1, |r| < 2^-6 (rows 31 and 32 touch 1 and use c = 1: r is exact there).
HSES_HD void log_parts(uint32_t i, const float4& e, float& hi, float& lo) {
    float uf = u2float(i);
    uf = uf > kUniform0 ? uf : kUniform0;
    const uint32_t ix = f2u(uf), kb = (ix - 0x4b400000u) & 0xff800000u;
    const float kf = i2float((int32_t)kb);
    const float r = ffma(u2f(ix - kb), e.x, -1.0f);
    const float th = ffma(kf, kLn2Hi, e.y), tl = ffma(kf, kLn2Lo, e.z);
    hi = fadd(th, r);
    const float er = fadd(r, -fadd(hi, -th));      // what the sum lost
    float p = ffma(r, 0.2f, -0.25f);
    p = ffma(r, p, 1.0f / 3.0f);
    p = ffma(r, p, -0.5f);
    lo = fadd(ffma(fmul(r, r), p, tl), er);
}
// cos of the fp32 product TAU * (j 2^-24) = hi + lo.  d = theta - t is exact, hi = cos t - d sin t rounded once, its
// rounding error is recovered exactly, the rest is of second order.
HSES_HD void cos_parts(uint32_t j, const float4& e, float& hi, float& lo) {
    const float theta = fmul(u2float(j), kTauF * 5.9604644775390625e-08f);
    const float d = fadd(theta, -e.x);
    const float q = fmul(d, d);
    const float inner = ffma(e.z, fmul(d, 1.0f / 6.0f), fmul(e.y, ffma(q, 1.0f / 24.0f, -0.5f)));
    hi = ffma(-e.z, d, e.y);
    const float res = ffma(-e.z, d, fadd(e.y, -hi));
    lo = ffma(q, inner, fadd(res, e.w));
}
// the two roundings; they differ when the true value may lie on either side of a rounding boundary
HSES_HD void roundings(float hi, float lo, float c, float& v0, float& v1) {
    v0 = fadd(hi, ffma(hi, c, lo));
    v1 = fadd(hi, ffma(hi, -c, lo));
}
HSES_HD int cos_row(uint32_t j) { return (int)(j >> 16); }

#if defined(__CUDACC__)
// sqrt of a normal, positive x, correctly rounded: one Newton step with an exact residual from an approximate
// reciprocal root (Markstein, IBM J. Res. Dev. 34, 1990).  The argument is -2 log u, between 1e-7 and 42: none of the
// special cases a general square root has to branch for.
__device__ __forceinline__ float sqrt_residual(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const float s = __fmul_rn(x, y);
    return __fmaf_rn(__fmaf_rn(-s, s, x), __fmul_rn(0.5f, y), s);
}
// N consecutive normals (noiser.rs:470-477).  Laid out as independent chains — generator steps, logarithms, cosines,
// then all bitmap reads together — so that table and bitmap latencies overlap instead of adding up.
// The bitmap word's index i >> 5 is taken as the high half of a product: a shift would go to the integer pipe, which
// bounds this code, the multiplier has room (223 -> 231 G normals/s).  The factor comes out of an opaque move, or the
// compiler turns the product back into a shift.
__device__ __forceinline__ uint32_t opaque(uint32_t v) {
    uint32_t r;
    asm("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
template <int N>
__device__ __forceinline__ void normals(uint64_t& state, const NoiseCal& cal, float (&out)[N]) {
    const uint32_t r5 = opaque(1u << 27);   // >> 5
    uint32_t iu[N], ju[N];
    uint64_t x = state;
#pragma unroll
    for (int n = 0; n < N; ++n) {
        x = xs64_step(x);
        iu[n] = (uint32_t)(x >> 40);
        x = xs64_step(x);
        ju[n] = (uint32_t)(x >> 40);
    }
    state = x;
    float l0[N], l1[N], c0[N], c1[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        float hi, lo;
        const float4 le = cal.log_tab[log_row(iu[n])];
        log_parts(iu[n], le, hi, lo);
        roundings(hi, lo, le.w, l0[n], l1[n]);
        cos_parts(ju[n], cal.cos_tab[cos_row(ju[n])], hi, lo);
        roundings(hi, lo, cal.cos_width[cos_row(ju[n])], c0[n], c1[n]);
    }
    uint32_t wl[N], wc[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        wl[n] = l0[n] != l1[n] ? cal.log_flip[__umulhi(iu[n], r5)] : 0u;
        wc[n] = c0[n] != c1[n] ? cal.cos_flip[__umulhi(ju[n], r5)] : 0u;
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const float lg = (wl[n] & (1u << (iu[n] & 31u))) ? l1[n] : l0[n];
        const float cs = (wc[n] & (1u << (ju[n] & 31u))) ? c1[n] : c0[n];
        out[n] = __fmul_rn(sqrt_residual(__fmul_rn(-2.0f, lg)), cs);
    }
}
__device__ __forceinline__ void normals4(uint64_t& state, const NoiseCal& cal, float (&out)[4]) { normals<4>(state, cal, out); }
__device__ __forceinline__ float normal1(uint64_t& state, const NoiseCal& cal) {
    float z[1];
    normals<1>(state, cal, z);
    return z[0];
}
// The candidate's tables in shared memory (6 KB); the caller synchronises.  Random rows of 16 bytes cost seven or
// eight wavefronts a read, words three or four; with the width in the cosine rows (32-byte rows, half the banks) the
// reads of a normal took 34 wavefronts and the L1 bounded the generator.
struct CalTab {
    float4 log_tab[kLogRows];
    float4 cos_tab[kCosRows];
    float cos_width[kCosRows];
};
__device__ __forceinline__ void stage_cal(NoiseCal& cal, CalTab& tab) {
    for (int i = threadIdx.x; i < kLogRows; i += blockDim.x) tab.log_tab[i] = cal.log_tab[i];
    for (int i = threadIdx.x; i < kCosRows; i += blockDim.x) {
        tab.cos_tab[i] = cal.cos_tab[i];
        tab.cos_width[i] = cal.cos_width[i];
    }
    cal.log_tab = tab.log_tab;
    cal.cos_tab = tab.cos_tab;
    cal.cos_width = tab.cos_width;
}
#endif

}  // namespace hses
