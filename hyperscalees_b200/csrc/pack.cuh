// What the packed tensor-core kernels (linear_pack.cu, snn_layer.cu) share: the fp16 hi/lo split of fp32 rows, the
// operand layouts of a pair's factors and how they are made.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "tc_common.cuh"

namespace hses {
namespace pack {

constexpr int PK_EXP_B = 11;       // B * 2^11: |normal| < 6 keeps it below 2^14
constexpr int PK_SEG = 8192;       // normals of a factor segment, at most

// two values as three bf16 pairs whose sums are the values (24 bits)
struct Parts {
    uint32_t p[3];
};
__device__ __forceinline__ Parts split2(float a, float b) {
    Parts r;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        r.p[i] = *reinterpret_cast<const uint32_t*>(&h);
        a -= __uint_as_float(r.p[i] << 16);
        b -= __uint_as_float(r.p[i] & 0xffff0000u);
    }
    return r;
}

// Which row of the call a packed row is.
struct RowMap {
    int packed;          // 0: row p is row p; 2: p = sample * t_steps + step is row step * n_pop + sample; 1: pairs, see below
    int rp;              // padded rows per pair
    int t_steps, bm;
    int64_t n_pop;
    int32_t first_thread, first_pair;
    int64_t rows;        // packed rows in total
};
__device__ __forceinline__ bool map_row(const RowMap& m, int64_t p, int64_t& R, bool& odd) {
    odd = false;
    R = p;
    if (p >= m.rows) return false;
    if (!m.packed) return true;
    if (m.packed == 2) {
        const int64_t sample = p / m.t_steps;
        R = (p - sample * m.t_steps) * m.n_pop + sample;
        return true;
    }
    const int32_t pair = (int32_t)(p / m.rp);
    const int lr = (int)(p - (int64_t)pair * m.rp);
    int64_t m_lo = (int64_t)(m.first_pair + pair) * 2 - m.first_thread, m_hi = m_lo + 2;
    if (m_lo < 0) m_lo = 0;
    if (m_hi > m.n_pop) m_hi = m.n_pop;
    const int rps = (int)(m_hi - m_lo) * m.bm;
    const int step = lr / rps, rr = lr - step * rps;
    if (step >= m.t_steps) return false;
    R = ((int64_t)step * m.n_pop + m_lo) * m.bm + rr;
    odd = ((m.first_thread + m_lo + rr / m.bm) & 1) != 0;
    return true;
}

// ------------------------------------------------------------------ operand preparation
struct SplitJob {
    const float* src;
    int64_t stride;
    int64_t rows;
    int k, kp;           // values per row, of the operand (multiple of 8, padded with zeros)
    int vec;             // rows are 16-byte aligned
    __half *hi, *lo;
    float* inv_scale;
    int* lo_flag;
    int fixed;           // hi: multiples of 8 (11 bits of the row's largest value): sums over spikes are exact
    int pitch;           // values from one row of the operand to the next; 0: kp
};

// values e .. e+3 of a row of k values; past the end: 0
__device__ __forceinline__ float4 load4(const float* row, int e, int k, int vec) {
    if (vec && e + 4 <= k) return __ldg(reinterpret_cast<const float4*>(row + e));
    float4 v;
    v.x = e < k ? __ldg(row + e) : 0.0f;
    v.y = e + 1 < k ? __ldg(row + e + 1) : 0.0f;
    v.z = e + 2 < k ? __ldg(row + e + 2) : 0.0f;
    v.w = e + 3 < k ? __ldg(row + e + 3) : 0.0f;
    return v;
}
// power of two that brings the largest magnitude m of a row into [2^13, 2^14); 1 for rows without one
__device__ __forceinline__ int scale_exponent(float m) {
    const int ex = (int)((__float_as_uint(m) >> 23) & 0xffu) - 127;
    int e = 13 - ex;
    if (ex <= -127 || ex >= 128) e = 0;
    return max(-100, min(100, e));
}
__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    return m;
}
__device__ __forceinline__ float max4(float m, float4 v) {
    return fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
}
__device__ __forceinline__ void split4(float4 v, float s, uint2& h2, uint2& l2, uint32_t& nz, bool fixed = false) {
    const float x0 = v.x * s, x1 = v.y * s, x2 = v.z * s, x3 = v.w * s;
    const auto grid = [&](float x) { return fixed ? rintf(x * 0.125f) * 8.0f : x; };
    const __half2 h01 = __floats2half2_rn(grid(x0), grid(x1)), h23 = __floats2half2_rn(grid(x2), grid(x3));
    const float2 b01 = __half22float2(h01), b23 = __half22float2(h23);
    const __half2 l01 = __floats2half2_rn(x0 - b01.x, x1 - b01.y), l23 = __floats2half2_rn(x2 - b23.x, x3 - b23.y);
    h2 = make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
    l2 = make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
    nz |= (l2.x | l2.y) & 0x7fff7fffu;   // a lo half of -0 is still zero
}

// One warp takes RPW rows at a time, NJ pieces of 128 values each in registers (NJ = 0: rows of any length,
// read twice, the second time from L1 or L2).
template <int NJ, int RPW>
__device__ __forceinline__ void split_rows(const SplitJob& j, const RowMap& map, int64_t block) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t p0 = (block * (blockDim.x >> 5) + warp) * RPW;
    uint32_t nz = 0;
    const int n4 = j.kp >> 2, pitch = j.pitch ? j.pitch : j.kp;
    if (NJ > 0) {
        float4 v[RPW][NJ > 0 ? NJ : 1];
        bool valid[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            int64_t R;
            bool odd;
            valid[r] = p0 + r < j.rows && map_row(map, p0 + r, R, odd);   // warp-uniform
            const float* row = j.src + (size_t)(valid[r] ? R : 0) * j.stride;
#pragma unroll
            for (int i = 0; i < NJ; ++i)
                v[r][i] = valid[r] ? load4(row, 4 * (lane + 32 * i), j.k, j.vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            if (!valid[r]) continue;
            float m = 0.0f;
#pragma unroll
            for (int i = 0; i < NJ; ++i) m = max4(m, v[r][i]);
            const int e = scale_exponent(warp_max(m));
            const float s = __uint_as_float((uint32_t)(127 + e) << 23);
            if (lane == 0) j.inv_scale[p0 + r] = __uint_as_float((uint32_t)(127 - e) << 23);
            uint2* dh = reinterpret_cast<uint2*>(j.hi + (size_t)(p0 + r) * pitch);
            uint2* dl = reinterpret_cast<uint2*>(j.lo + (size_t)(p0 + r) * pitch);
#pragma unroll
            for (int i = 0; i < NJ; ++i) {
                const int c = lane + 32 * i;
                if (c < n4) {
                    uint2 h2, l2;
                    split4(v[r][i], s, h2, l2, nz, j.fixed);
                    dh[c] = h2;
                    dl[c] = l2;
                }
            }
        }
    } else {
        int64_t R;
        bool odd;
        if (p0 >= j.rows || !map_row(map, p0, R, odd)) return;
        const float* row = j.src + (size_t)R * j.stride;
        float m = 0.0f;
        for (int c = lane; c < n4; c += 32) m = max4(m, load4(row, 4 * c, j.k, j.vec));
        const int e = scale_exponent(warp_max(m));
        const float s = __uint_as_float((uint32_t)(127 + e) << 23);
        if (lane == 0) j.inv_scale[p0] = __uint_as_float((uint32_t)(127 - e) << 23);
        uint2* dh = reinterpret_cast<uint2*>(j.hi + (size_t)p0 * pitch);
        uint2* dl = reinterpret_cast<uint2*>(j.lo + (size_t)p0 * pitch);
        for (int c = lane; c < n4; c += 32) {
            uint2 h2, l2;
            split4(load4(row, 4 * c, j.k, j.vec), s, h2, l2, nz, j.fixed);
            dh[c] = h2;
            dl[c] = l2;
        }
    }
    // one flag per call tells the product whether any lo half is non-zero (a set flag is not set again)
    if (j.lo_flag && __any_sync(0xffffffffu, nz != 0) && lane == 0 && *reinterpret_cast<volatile int*>(j.lo_flag) == 0)
        atomicOr(j.lo_flag, 1);
}
struct FactorJob {
    const float *cache_a, *cache_b;   // raw (pairs, a, r) and (pairs, k, r), or NULL: regenerate
    const uint64_t *jump, *lane4, *lane16;
    NoiseCal cal;
    uint64_t key;
    int32_t true_epoch, first_pair;
    int64_t pairs;
    int r, r16, k, kp, a;
    int row_a0, row_b0;               // first output-side and input-side row of a pair's stream block
    int seg;                          // rows per segment (a multiple of 8)
    int bn, n_chunks, kb;             // output columns per chunk, chunks, rank values per block of A's image
    float base_sigma;
    const float* col_scale;           // 2^-e of W's rows
    __half *bhi, *blo;                // (pairs, r16, kp), rows pitch values apart (0: kp)
    int pitch;
    __nv_bfloat16* aimg;              // (pairs, chunk, r16 / kb, part 3, kb / 8, bn, 8)
};

// Segments of a pair's k + a rows of normals: as long as shared memory allows (a segment's start is a chain of tables that
// its block waits for), shorter where that leaves SMs without four of them.  In stream order a segment may hold the end of
// B and the start of A; else B's segments come first, then A's.  1000 members of 784-300-100, rank 6: 49 us; 512 rows of
// one factor at a time, four normals to a thread 64 us; 16 pairs are fastest in short segments.
inline int plan_segments(FactorJob& f, int sms) {
    const int64_t normals = f.pairs * (int64_t)(f.k + f.a) * f.r;
    const int want = (int)std::max<int64_t>(512, std::min<int64_t>(PK_SEG, normals / (4 * (int64_t)sms)));
    f.seg = std::max(8, std::min(2048, (want / f.r) & ~7));
    return f.row_b0 == 0 ? (f.k + f.a + f.seg - 1) / f.seg : (f.k + f.seg - 1) / f.seg + (f.a + f.seg - 1) / f.seg;
}
// Segment `seg` of pair `p`: its normals into shared memory (from the cache, or stream_fill), then to the operand layout.
__device__ __forceinline__ void factor_segment(const FactorJob& f, int64_t p, int seg, float* buf, CalTab& tab, uint64_t* state_s) {
    const int tid = threadIdx.x, step = f.seg;
    int b0, nb, a0, na;                                       // first row and rows of B and of A in this segment
    if (f.row_b0 == 0) {
        const int c0 = seg * step, c1 = min(c0 + step, f.k + f.a);
        b0 = min(c0, f.k), nb = min(c1, f.k) - b0;
        a0 = max(c0 - f.k, 0), na = max(c1 - f.k, 0) - a0;
    } else {
        const int nseg_b = (f.k + step - 1) / step;
        const bool is_b = seg < nseg_b;
        b0 = is_b ? seg * step : f.k, nb = is_b ? min(step, f.k - b0) : 0;
        a0 = is_b ? 0 : (seg - nseg_b) * step, na = is_b ? 0 : min(step, f.a - a0);
    }
    if (f.cache_b) {
        chain_wait();
        auto fetch = [&](float* dst, const float* src, int cnt) {
            if (((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(4 * (dst - buf))) & 15) == 0) {
                for (int i = tid; i < cnt / 4; i += blockDim.x)
                    *reinterpret_cast<float4*>(dst + 4 * i) = __ldg(reinterpret_cast<const float4*>(src) + i);
                for (int i = (cnt & ~3) + tid; i < cnt; i += blockDim.x) dst[i] = __ldg(src + i);
            } else {
                for (int i = tid; i < cnt; i += blockDim.x) dst[i] = __ldg(src + i);
            }
        };
        fetch(buf, f.cache_b + ((size_t)p * f.k + b0) * f.r, nb * f.r);
        fetch(buf + nb * f.r, f.cache_a + ((size_t)p * f.a + a0) * f.r, na * f.r);
    } else {
        NoiseCal cal = f.cal;
        stage_cal(cal, tab);
        const uint64_t first = (uint64_t)f.r * (uint64_t)(nb ? b0 + f.row_b0 : a0 + f.row_a0);
        stream_fill(cal, f.jump, f.lane4, f.lane16, noise_seed(f.key, f.true_epoch, f.first_pair + (int32_t)p) | 1ull, first,
                    (nb + na) * f.r, state_s, [&](int off, float (&z)[4]) {
                        *reinterpret_cast<float4*>(buf + off) = make_float4(z[0], z[1], z[2], z[3]);
                    });
        chain_wait();   // the normals need nothing of the kernels before
    }
    __syncthreads();
    if (nb) {
        // eight consecutive k of one rank column per thread: 4 such pieces x 8 columns per warp
        const int kend = b0 + nb == f.k ? f.kp - b0 : nb;     // the padding of the last segment's rows is zero
        const int ng = (kend + 7) >> 3, qb = f.r16 >> 3;
        const float sc = (float)(1 << PK_EXP_B);
        for (int idx = tid; idx < ((ng + 3) & ~3) * f.r16; idx += blockDim.x) {
            const int blk = idx >> 5, l = idx & 31;
            const int q = (blk % qb) * 8 + (l & 7), g = (blk / qb) * 4 + (l >> 3);
            if (g >= ng) continue;
            uint2 h0 = make_uint2(0, 0), h1 = h0, l0 = h0, l1 = h0;
            if (q < f.r) {
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = g * 8 + j < nb ? buf[(g * 8 + j) * f.r + q] : 0.0f;
                uint32_t nz = 0;
                split4(make_float4(v[0], v[1], v[2], v[3]), sc, h0, l0, nz);
                split4(make_float4(v[4], v[5], v[6], v[7]), sc, h1, l1, nz);
            }
            const size_t o = ((size_t)p * f.r16 + q) * (f.pitch ? f.pitch : f.kp) + b0 + g * 8;
            *reinterpret_cast<uint4*>(f.bhi + o) = make_uint4(h0.x, h0.y, h1.x, h1.y);
            *reinterpret_cast<uint4*>(f.blo + o) = make_uint4(l0.x, l0.y, l1.x, l1.y);
        }
    }
    if (na) {
        const float* src = buf + nb * f.r;
        for (int idx = tid; idx < na * (f.r16 >> 3); idx += blockDim.x) {
            const int g = idx / na, i = idx - g * na;         // rank piece, row of the segment
            const int n = a0 + i, c = n / f.bn, nn = n - c * f.bn;
            uint32_t w[3][4] = {};
            if (g * 8 < f.r) {
                const uint32_t e = 254u - (__float_as_uint(__ldg(f.col_scale + n)) >> 23);   // exponent field of 2^+e
                const float sc = __fmul_rn(f.base_sigma, __uint_as_float(e << 23)) * (1.0f / (1 << PK_EXP_B));
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    float v[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int q = g * 8 + j + h;
                        v[h] = q < f.r ? __fmul_rn(src[i * f.r + q], sc) : 0.0f;
                    }
#pragma unroll
                    for (int part = 0; part < 3; ++part) {
                        const __nv_bfloat162 b = __floats2bfloat162_rn(v[0], v[1]);
                        w[part][j >> 1] = *reinterpret_cast<const uint32_t*>(&b);
                        v[0] -= __bfloat162float(b.x);
                        v[1] -= __bfloat162float(b.y);
                    }
                }
            }
            const int kblk = (g * 8) / f.kb, gi = g - kblk * (f.kb >> 3);
            __nv_bfloat16* img = f.aimg + ((((size_t)p * f.n_chunks + c) * (f.r16 / f.kb) + kblk) * 3) * f.kb * f.bn;
#pragma unroll
            for (int part = 0; part < 3; ++part)
                *reinterpret_cast<uint4*>(img + (size_t)part * f.kb * f.bn + ((size_t)gi * f.bn + nn) * 8) =
                    make_uint4(w[part][0], w[part][1], w[part][2], w[part][3]);
        }
    }
}

}  // namespace pack
}  // namespace hses
