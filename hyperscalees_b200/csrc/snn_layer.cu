// Forward pass of the spiking MLP (SnnModel::forward, hyperscalees-models/src/snn.rs:253-282, any number of hidden
// layers) in one kernel per layer: spikes travel between the layers as fp16, the LIF scan over the T steps runs behind
// the product, and nothing but spikes (or, behind the last hidden layer, their counts) is written to memory.
//
//   launch 1  encode_half       Poisson spikes as fp16 (or: f32 input spikes converted)
//   launch 2  snn_split_w       W of every hidden layer as fp16 hi + lo
//   launch 3  snn_factors       every hidden layer's factors in operand layout (see linear_pack.cu), noise only
//   launch 4. snn_layer         per hidden layer
//   last      snn_readout       rates -> logits -> score, one CTA per antithetic pair
// snn_layer: a tile is `spt` samples x all T steps (at most 128 rows), fetched by one 3-D TMA box per k-block, so that
// the scan of a neuron never leaves the CTA.  Inputs that are exact in fp16 need two MMA passes (x * W_hi + x * W_lo).
// With noise a tile holds whole antithetic pairs or lies inside one; t = x·B and t·(sA)ᵀ are tensor-core products as in
// linear_pack.cu.  Two groups of four epilogue warps turn 16 columns at a time into currents in shared memory, scan
// them and store the spikes.  No multicast, no cluster launch, bounded waits only.
#include <cuda.h>

#include <algorithm>
#include <array>
#include <vector>

#include "linear.cuh"
#include "pack.cuh"
#include "snn_layer.cuh"

namespace hses {

namespace {

using namespace tc;
using namespace pack;

constexpr int SL_THREADS = 320;          // warp 0 TMA, warp 1 MMA, warps 2-9 scan; with noise also
constexpr int SL_THREADS_T = 576;        // warps 10-17: t to operand layout
constexpr int SL_MAX_STAGES = 6;
constexpr int SL_SMEM_LIMIT = 232448;
constexpr int kSnnMaxLayers = 8;         // hidden layers

// ------------------------------------------------------------------------------- input
// poisson_encode_fused_oxide.rs:36-105 (see poisson_kernel in elementwise.cu for the threshold), eight neighbouring
// inputs of a row per thread, spikes as fp16 rows of kp values (the padding is zero), row sample * T + step.  Bound by the
// generator's integer work (8 steps of 784 inputs: 12 instructions a step).
__global__ void __launch_bounds__(256)
encode_half_kernel(const float* __restrict__ probs, int64_t batch, int in_dim, int64_t stride, int T, uint32_t mix,
                   __half* __restrict__ out, int kp) {
    chain_begin();
    const int groups = kp >> 3;
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x, srow = v / (uint32_t)groups;   // batch * in_dim < 2^32
    if (srow >= batch) return;
    const int64_t row = srow;
    const int col = (int)(v - srow * groups) * 8;
    PoissonCell c[8];
    const bool vec = (reinterpret_cast<uintptr_t>(probs) & 15) == 0 && (stride & 3) == 0 && col + 8 <= in_dim;
    float p[8];
    if (vec) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(probs + row * stride + col));
        const float4 b = __ldg(reinterpret_cast<const float4*>(probs + row * stride + col + 4));
        p[0] = a.x; p[1] = a.y; p[2] = a.z; p[3] = a.w; p[4] = b.x; p[5] = b.y; p[6] = b.z; p[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = col + i < in_dim ? __ldg(probs + row * stride + col + i) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = poisson_cell(p[i], poisson_seed((uint32_t)(row * in_dim + col + i), mix));
    for (int t = 0; t < T; ++t) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            c[i].x = xs32(c[i].x);
            c[i + 1].x = xs32(c[i + 1].x);
            w[i >> 1] = (c[i].x <= c[i].last ? 0x3C00u : 0u) | (c[i + 1].x <= c[i + 1].last ? 0x3C000000u : 0u);
        }
        *reinterpret_cast<uint4*>(out + ((size_t)row * T + t) * kp + col) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// f32 spikes (T, n, k) as fp16 with no scale, rows sample * T + step; sets the flag when a value is not exact there
__global__ void __launch_bounds__(256)
spikes_half_kernel(const float* __restrict__ src, int64_t n, int T, int k, int64_t stride, __half* __restrict__ out, int kp,
                   int* __restrict__ inexact) {
    chain_begin();
    const int groups = kp >> 3;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n * T * groups) return;
    const int64_t row = v / groups;
    const int col = (int)(v - row * groups) * 8;
    const int64_t t = row / n, sample = row - t * n;
    const int vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && (stride & 3) == 0;
    const float4 a = load4(src + row * stride, col, k, vec), b = load4(src + row * stride, col + 4, k, vec);
    uint2 h0, h1, l0, l1;
    uint32_t nz = 0;
    split4(a, 1.0f, h0, l0, nz);
    split4(b, 1.0f, h1, l1, nz);
    // an infinite or NaN half is not the value either (its remainder is NaN, so nz is set)
    if (nz && *reinterpret_cast<volatile int*>(inexact) == 0) atomicOr(inexact, 1);
    *reinterpret_cast<uint4*>(out + (size_t)(sample * T + t) * kp + col) = make_uint4(h0.x, h0.y, h1.x, h1.y);
}
// only when the flag is set: the input once more, every row scaled and split into hi + lo
template <int NJ, int RPW>
__global__ void __launch_bounds__(256) split_if_inexact_kernel(SplitJob j, RowMap map) {
    chain_begin();
    if (*j.lo_flag == 0) return;
    for (int64_t b = blockIdx.x; b * (blockDim.x >> 5) * RPW < j.rows; b += gridDim.x) split_rows<NJ, RPW>(j, map, b);
}

struct SplitJobs {
    int n;
    SplitJob j[kSnnMaxLayers];
    int block0[kSnnMaxLayers + 1];
    int* clear;              // the input's flag, or NULL
};
template <int NJ, int RPW>
__global__ void __launch_bounds__(256) snn_split_w_kernel(const __grid_constant__ SplitJobs jobs) {
    chain_begin();
    if (jobs.clear && blockIdx.x == 0 && threadIdx.x == 0) *jobs.clear = 0;
    int i = 0;
    while (i + 1 < jobs.n && (int)blockIdx.x >= jobs.block0[i + 1]) ++i;
    RowMap map{};
    map.rows = jobs.j[i].rows;
    split_rows<NJ, RPW>(jobs.j[i], map, blockIdx.x - jobs.block0[i]);
}

struct FactorJobs {
    int n;
    FactorJob j[kSnnMaxLayers];
    int segs[kSnnMaxLayers];
    int64_t block0[kSnnMaxLayers + 1];
};
__global__ void __launch_bounds__(256) snn_factors_kernel(const __grid_constant__ FactorJobs jobs) {
    __shared__ __align__(16) float buf[PK_SEG];
    __shared__ CalTab tab;
    __shared__ uint64_t state_s[32];
    chain_next();                                             // factor_segment waits
    int i = 0;
    while (i + 1 < jobs.n && (int64_t)blockIdx.x >= jobs.block0[i + 1]) ++i;
    const int64_t rel = blockIdx.x - jobs.block0[i];
    factor_segment(jobs.j[i], rel / jobs.segs[i], (int)(rel % jobs.segs[i]), buf, tab, state_s);
}

// ------------------------------------------------------------------------- hidden layer
struct LayerArgs {
    int T, spt;              // steps, samples per tile; (T - 1) * spt and spt rounded up to 8 fit `rows`
    int exact;               // 128 rows: the products with W's lo half in an accumulator of their own (see make_plan)
    int rows;                // 128: two accumulators in turn; 192, 256: one, W and the factors read less often
    int64_t n;               // samples
    int64_t tiles;
    int ppt;                 // whole pairs per tile, or 0: tpp tiles inside a pair
    int tpp;
    int spp;                 // samples per pair
    int bm;
    int groups, n_chunks, bn, a, k_blocks;
    int nt, r16;
    int t_chains;            // sums of t over k, 2 nt columns each (B hi, B lo)
    int64_t pairs;
    const __nv_bfloat16* aimg;
    const float *row_scale, *col_scale;
    const int* inexact;      // NULL or the flag of spikes_half: x has a lo half and row scales
    float leak, v_th;
    int reset;
    __half* out_half;        // spikes (n, T, out_pitch), or NULL
    int out_pitch;
    float* count;            // spikes over the T steps (n, a), or NULL
    int stages, stage_bytes;
    int* status;
};
constexpr int SL_OPERAND = 128 * 128;    // bytes of 128 rows x 64 values: x, W hi, W lo

struct Scan {
    uint32_t lo;             // accumulator of the lo products, or 0: in y
    uint32_t y, u;           // TMEM address of sample 0's first step in the accumulators of the product and of the rank term
    int T, spt, cnt;         // samples of the tile
    bool live;
    float cs, leak, v_th;
    const float* row_scale;  // of sample 0, step 0, or NULL
    __half* out;             // of sample 0, step 0, or NULL
    int out_pitch;
    float* count;            // of sample 0, or NULL
    int a;
};
// run_lif (snn.rs:73-97) of one neuron per thread for the samples sb .. sb+7: their currents of all steps are columns of
// this thread's TMEM lane, so the membranes never leave registers.  Eight chains side by side, since a scheduler has two of
// these warps, and a loop over the steps: unrolled for a known T the same work was bound by fetching instructions.
template <bool PERT, bool HARD>
__device__ __forceinline__ void scan8(const Scan& c, int sb) {
    uint32_t ny[8], nu[8], nl[8] = {};
    float v[8], sum[8];
    const int left = c.cnt - sb;                                // samples of this block, uniform
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = sum[s] = 0.0f;
    auto load = [&](int t) {
        tmem_ld8_issue(c.y + t * c.spt + sb, ny);
        if (c.lo) tmem_ld8_issue(c.lo + t * c.spt + sb, nl);
        if (PERT) tmem_ld8_issue(c.u + t * c.spt + sb, nu);
    };
    load(0);
    unsigned short* out = c.out ? reinterpret_cast<unsigned short*>(c.out) + (int64_t)sb * c.T * c.out_pitch : nullptr;
    const int64_t sample_pitch = (int64_t)c.T * c.out_pitch;
#pragma unroll 1
    for (int t = 0; t < c.T; ++t) {
        float cur[8];
        tmem_ld_wait();
#pragma unroll
        for (int s = 0; s < 8; ++s) {                           // the scales are powers of two: exact
            float y = __uint_as_float(ny[s]);
            if (c.lo) y = __fadd_rn(y, __uint_as_float(nl[s]));
            cur[s] = __fmul_rn(PERT ? __fadd_rn(y, __uint_as_float(nu[s])) : y, c.cs);
        }
        load(min(t + 1, c.T - 1));
        if (c.row_scale) {
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (s < left) cur[s] = __fmul_rn(cur[s], __ldg(c.row_scale + (sb + s) * c.T + t));
        }
        unsigned short half[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const float sp = lif_update(v[s], cur[s], c.leak, c.v_th, HARD ? HSES_RESET_HARD : HSES_RESET_SUBTRACT);
            sum[s] = __fadd_rn(sum[s], sp);
            half[s] = sp != 0.0f ? 0x3C00 : 0;                  // 1.0 as fp16
        }
        if (out) {
            if (c.live) {
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    if (s < left) out[s * sample_pitch] = half[s];
            }
            out += c.out_pitch;
        }
    }
    tmem_ld_wait();
    if (c.count && c.live) {
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s < left) c.count[(int64_t)(sb + s) * c.a] = sum[s];
    }
}

template <bool PERT>
__global__ void __launch_bounds__(PERT ? SL_THREADS_T : SL_THREADS, 1)
snn_layer_kernel(const __grid_constant__ CUtensorMap tm_xhi, const __grid_constant__ CUtensorMap tm_xlo,
                 const __grid_constant__ CUtensorMap tm_whi, const __grid_constant__ CUtensorMap tm_wlo,
                 const __grid_constant__ CUtensorMap tm_bhi, const __grid_constant__ CUtensorMap tm_blo,
                 const LayerArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t x_tx = (uint32_t)(g.spt * g.T) * 128;      // bytes a box of x brings
    const uint32_t w_tx = (uint32_t)g.bn * 128, b_bytes = (uint32_t)g.nt * 128;
    const int W_HI = g.rows * 128, W_LO = W_HI + SL_OPERAND, B_HI = W_LO + SL_OPERAND;
    uint8_t* tparts = smem + (size_t)g.stages * g.stage_bytes;   // t: [part 3][nt / 8][rows][8] bf16
    const int part_bytes = g.nt * g.rows * 2, bufs = !PERT || (g.rows == 128 && !g.exact) ? 2 : 1;
    __shared__ uint64_t full[SL_MAX_STAGES], empty[SL_MAX_STAGES], tfull[2], tempty[2], tacc, tready;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag_s;
    volatile int* abort_flag = &abort_flag_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_flag_s = 0;
        for (int s = 0; s < g.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 256);
        }
        mbar_init(&tacc, 1);
        mbar_init(&tready, 256);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    chain_wait();                                             // before the allocation: a waiting block holds no tensor memory
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_next();
    // exact: the product at 0, its lo part 128 (without noise 256) further, the rank term at 256, t at 384.  Else:
    // Columns 0-255: accumulators of the product, `rows` each (without noise up to 511).  The same from 256: the rank term,
    // whose columns hold t (a part of 128 columns per 128 rows) until it has been read.
    const uint32_t tmem = tmem_slot;
    const int64_t units = g.tiles * g.groups;
    const bool x_lo = g.inexact != nullptr && *g.inexact != 0;
    const int x_parts = x_lo ? 2 : 1;                         // stages per k-block: (x_hi, W_hi, W_lo), then (x_lo, W_hi)
    // samples of tile mt: first one and count; its pairs
    auto tile_of = [&](int64_t mt, int64_t& s0, int& cnt, int64_t& p0, int& nd) {
        p0 = 0;
        nd = 0;
        if (!PERT) {
            s0 = mt * g.spt;
            cnt = (int)min((int64_t)g.spt, g.n - s0);
        } else if (g.ppt) {
            s0 = mt * g.ppt * g.spp;
            p0 = mt * g.ppt;
            nd = (int)min((int64_t)g.ppt, g.pairs - p0);
            cnt = nd * g.spp;
        } else {
            p0 = mt / g.tpp;
            const int sub = (int)(mt - p0 * g.tpp);
            s0 = p0 * g.spp + (int64_t)sub * g.spt;
            cnt = min(g.spt, g.spp - sub * g.spt);
            nd = 1;
        }
    };

    if (warp == 0) {
        if (lane == 0) {
            Ring ring{0, 0};
            bool ok = true;
            auto slot = [&](uint32_t bytes) -> uint8_t* {
                ok = mbar_wait(&empty[ring.s], ring.ph ^ 1, abort_flag, g.status, 1);
                if (!ok) return nullptr;
                mbar_expect_tx(&full[ring.s], bytes);
                return smem + (size_t)ring.s * g.stage_bytes;
            };
            for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                const int64_t mt = u / g.groups;
                const int grp = (int)(u - mt * g.groups);
                const int c0 = g.n_chunks * grp / g.groups, c1 = g.n_chunks * (grp + 1) / g.groups;
                int64_t s0, p0;
                int cnt, nd;
                tile_of(mt, s0, cnt, p0, nd);
                for (int c = c0; c < c1 && ok; ++c) {
                    const bool with_t = PERT && c == c0;
                    for (int kb = 0; kb < g.k_blocks && ok; ++kb)
                        for (int part = 0; part < x_parts; ++part, ring.next(g.stages)) {
                            uint8_t* st = slot(x_tx + (2 - part) * (w_tx + (with_t ? b_bytes : 0)));
                            if (!ok) break;
                            uint64_t* bar = &full[ring.s];
                            tma_load_3d(st, part ? &tm_xlo : &tm_xhi, kb * 64, (int)s0, 0, bar);
                            tma_load_2d(st + W_HI, &tm_whi, kb * 64, c * g.bn, bar);
                            if (!part) tma_load_2d(st + W_LO, &tm_wlo, kb * 64, c * g.bn, bar);
                            if (with_t) {
                                tma_load_2d(st + B_HI, &tm_bhi, kb * 64, (int)(p0 * g.r16), bar);
                                if (!part) tma_load_2d(st + B_HI + b_bytes, &tm_blo, kb * 64, (int)(p0 * g.r16), bar);
                            }
                        }
                    if (PERT) {
                        const uint32_t bytes = 3u * g.r16 * g.bn * 2;
                        for (int i = 0; i < nd && ok; ++i, ring.next(g.stages)) {
                            uint8_t* st = slot(bytes);
                            if (!ok) break;
                            bulk_load(st, g.aimg + ((size_t)(p0 + i) * g.n_chunks + c) * 3 * g.r16 * g.bn, bytes,
                                      &full[ring.s]);
                        }
                    }
                }
            }
            if (!ok) {
                // copies already issued still land in this CTA's shared memory: give them a bounded moment
                for (int s = 0; s < g.stages; ++s)
                    for (uint32_t i = 0; i < 4096; ++i) {
                        if (mbar_try(&full[s], 0) || mbar_try(&full[s], 1)) break;
                        __nanosleep(256);
                    }
            }
        }
    } else if (warp == 1) {
        // the whole warp runs the loop, so that addresses and descriptors are uniform; one lane issues
        const int n16 = (g.spt * g.T + 15) & ~15, t_halves = n16 > 128 ? 2 : 1;
        const uint32_t idesc = make_idesc(n16), idesc_u = make_idesc_bf16(n16);
        const uint32_t idesc_t = make_idesc(PERT ? 2 * g.nt : 16), idesc_tl = make_idesc(PERT ? g.nt : 16);
        const int tc_len = PERT ? (g.k_blocks + g.t_chains - 1) / g.t_chains : 1;
        const uint64_t desc0 = make_smem_desc(smem), desc_step = (uint64_t)(g.stage_bytes >> 4);
        const uint64_t plain0 = make_plain_desc(smem, g.bn * 16), plain_t = make_plain_desc(tparts, g.rows * 16);
        const uint32_t abytes = (uint32_t)g.r16 * g.bn * 2;       // one part of an image
        uint32_t acc_it = 0, unit_no = 0;
        Ring ring{0, 0};
        bool ok = true;
        for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x, ++unit_no) {
            const int64_t mt = u / g.groups;
            const int grp = (int)(u - mt * g.groups);
            const int c0 = g.n_chunks * grp / g.groups, c1 = g.n_chunks * (grp + 1) / g.groups;
            int64_t s0, p0;
            int cnt, nd;
            tile_of(mt, s0, cnt, p0, nd);
            for (int c = c0; c < c1 && ok; ++c, ++acc_it) {
                const bool with_t = PERT && c == c0;
                const int b = bufs == 2 ? (int)(acc_it & 1) : 0;
                const uint32_t ph = (bufs == 2 ? acc_it >> 1 : acc_it) & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(&tempty[b], ph ^ 1, abort_flag, g.status, 2));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(b * g.rows), dl = !g.exact ? d : d + (PERT ? 128 : 256);
                const uint32_t tmem_u = d + 256;
                uint32_t tc_col = g.exact ? tmem + 384 : tmem_u;                     // accumulator and k-blocks left of t's current sum
                int tc_left = tc_len;
                for (int kb = 0; kb < g.k_blocks && ok; ++kb)
                    for (int part = 0; part < x_parts; ++part, ring.next(g.stages)) {
                        ok = __all_sync(0xffffffffu, mbar_wait(&full[ring.s], ring.ph, abort_flag, g.status, 3));
                        if (!ok) break;
                        tc_fence_after();
                        // part 0: x_hi against both halves of the other operand; part 1: x_lo against its hi half
                        const uint64_t dx = desc0 + __shfl_sync(0xffffffffu, ring.s, 0) * desc_step;
                        const uint64_t dwh = dx + (W_HI >> 4), dwl = dx + (W_LO >> 4), db = dx + (B_HI >> 4);
                        const uint32_t more = (kb | part) != 0;
                        {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {       // 16 fp16 = 32 bytes along k
                                if (!part) umma_f16_warp(dl, dwl + 2 * ks, dx + 2 * ks, idesc, ks ? 1u : more);
                                umma_f16_warp(part ? dl : d, dwh + 2 * ks, dx + 2 * ks, idesc, !g.exact || part || kb || ks);
                            }
                            if (with_t) {
                                // t: B's halves side by side, in sums of a few k-blocks each
                                for (int h = 0; h < t_halves; ++h) {
                                    const uint32_t col = tc_col + h * 128;
                                    const uint64_t dxh = dx + h * (SL_OPERAND >> 4);
#pragma unroll
                                    for (int ks = 0; ks < 4; ++ks)
                                        umma_f16_warp(part ? col + g.nt : col, dxh + 2 * ks, db + 2 * ks, part ? idesc_tl : idesc_t,
                                                      ks || part || tc_left != tc_len);
                                }
                            }
                            umma_commit_warp(&empty[ring.s]);
                        }
                        if (with_t && part + 1 == x_parts && --tc_left == 0) {
                            tc_col += 2 * g.nt;
                            tc_left = tc_len;
                        }
                    }
                if (!ok) break;
                if (PERT) {
                    if (with_t) {
                        umma_commit_warp(&tacc);
                        ok = __all_sync(0xffffffffu, mbar_wait(&tready, unit_no & 1, abort_flag, g.status, 4));
                        if (!ok) break;
                    }
                    tc_fence_after();
                    for (int dd = 0; dd < nd; ++dd, ring.next(g.stages)) {
                        ok = __all_sync(0xffffffffu, mbar_wait(&full[ring.s], ring.ph, abort_flag, g.status, 3));
                        if (!ok) break;
                        tc_fence_after();
                        for (int ks = 0; ks < g.r16 / 16; ++ks) {
                            const uint64_t dt = plain_t + (uint64_t)(((dd * g.r16 + ks * 16) >> 3) * g.rows);
                            const uint64_t da = plain0 + ring.s * desc_step + (uint64_t)(ks * 2 * g.bn);
                            const uint32_t t1 = part_bytes >> 4, t2 = 2 * t1, a1 = abytes >> 4, a2 = 2 * a1;
                            {
                                umma_f16_warp(tmem_u, da, dt + t2, idesc_u, (dd | ks) != 0);
                                umma_f16_warp(tmem_u, da + a2, dt, idesc_u, 1);
                                umma_f16_warp(tmem_u, da + a1, dt + t1, idesc_u, 1);
                                umma_f16_warp(tmem_u, da, dt + t1, idesc_u, 1);
                                umma_f16_warp(tmem_u, da + a1, dt, idesc_u, 1);
                                umma_f16_warp(tmem_u, da, dt, idesc_u, 1);
                            }
                        }
                        umma_commit_warp(&empty[ring.s]);
                    }
                    if (!ok) break;
                }
                umma_commit_warp(&tfull[b]);
                __syncwarp();
            }
        }
    } else if (PERT && warp >= 10) {
        // ------------------------------------------------------- t to bf16 parts in shared memory
        // more than 128 rows: each four warps take 128 of them; else every second piece of eight columns
        const int q4 = warp & 3, eh = (warp - 10) >> 2;
        const bool tall = g.spt * g.T > 128;
        const int row = q4 * 32 + lane + (tall ? eh * 128 : 0), step = row / g.spt, sm = row - step * g.spt;
        uint32_t acc_it = 0, unit_no = 0;
        for (int64_t u = blockIdx.x; u < units; u += gridDim.x, ++unit_no) {
            const int64_t mt = u / g.groups;
            const int grp = (int)(u - mt * g.groups);
            int64_t s0, p0;
            int cnt, nd;
            tile_of(mt, s0, cnt, p0, nd);
            const int b = bufs == 2 ? (int)(acc_it & 1) : 0;
            acc_it += g.n_chunks * (grp + 1) / g.groups - g.n_chunks * grp / g.groups;
            const uint32_t t0 = tmem + ((uint32_t)(q4 * 32) << 16) + (g.exact ? 384 : 256 + b * g.rows) + (tall ? eh * 128 : 0);
            const int64_t s = s0 + sm;
            const bool odd = ((s / g.bm) & 1) != 0;           // the odd member of a pair has A negated
            const int d = step < g.T && sm < cnt ? (int)(s / g.spp - p0) : -1;
            if (!__all_sync(0xffffffffu, mbar_wait(&tacc, unit_no & 1, abort_flag, g.status, 5))) break;
            tc_fence_after();
            for (int c8 = tall ? 0 : eh; c8 < g.nt / 8; c8 += tall ? 1 : 2) {
                uint32_t w[3][4];
                float tv[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) tv[j] = 0.0f;
                for (int half = 1; half >= 0; --half)         // what B's lo half gave, then the rest
                    for (int ch = 0; ch < g.t_chains; ++ch) {
                        uint32_t v[8];
                        tmem_ld8(t0 + (2 * ch + half) * g.nt + c8 * 8, v);
#pragma unroll
                        for (int j = 0; j < 8; ++j) tv[j] = __fadd_rn(tv[j], __uint_as_float(v[j]));
                    }
                const bool mine = c8 * 8 / g.r16 == d;        // only the columns of the row's own pair are not zero
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    float v0 = mine ? tv[j] : 0.0f, v1 = mine ? tv[j + 1] : 0.0f;
                    if (odd) v0 = -v0, v1 = -v1;
#pragma unroll
                    for (int part = 0; part < 3; ++part) {
                        const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
                        w[part][j >> 1] = *reinterpret_cast<const uint32_t*>(&h);
                        v0 -= __bfloat162float(h.x);
                        v1 -= __bfloat162float(h.y);
                    }
                }
#pragma unroll
                for (int part = 0; part < 3; ++part)
                    if (row < g.rows) *reinterpret_cast<uint4*>(tparts + part * part_bytes + (c8 * g.rows + row) * 16) =
                        make_uint4(w[part][0], w[part][1], w[part][2], w[part][3]);
            }
            fence_proxy_async();
            tc_fence_before();
            mbar_arrive(&tready);
        }
    } else {
        // ----------------------------------------------------------------------------- scan
        const int q4 = warp & 3, eh = (warp - 2) >> 2;        // TMEM quadrant; group: sample blocks eh, eh + 2, ..
        const int gt = q4 * 32 + lane;                        // TMEM lane: a neuron of the chunk
        const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16);
        uint32_t acc_it = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const int64_t mt = u / g.groups;
            const int grp = (int)(u - mt * g.groups);
            const int c0 = g.n_chunks * grp / g.groups, c1 = g.n_chunks * (grp + 1) / g.groups;
            int64_t s0, p0;
            int cnt, nd;
            tile_of(mt, s0, cnt, p0, nd);
            for (int c = c0; c < c1; ++c, ++acc_it) {
                const int b = bufs == 2 ? (int)(acc_it & 1) : 0;
                ok = __all_sync(0xffffffffu, mbar_wait(&tfull[b], (bufs == 2 ? acc_it >> 1 : acc_it) & 1, abort_flag, g.status, 6));
                if (!ok) break;
                tc_fence_after();
                const int n = c * g.bn + gt;
                const bool live = gt < g.bn && n < g.a;
                if (c * g.bn + q4 * 32 < g.a && q4 * 32 < g.bn) {
                    const Scan sc{g.exact ? lane_base + b * g.rows + (PERT ? 128 : 256) : 0, lane_base + b * g.rows, lane_base + 256 + b * g.rows, g.T, g.spt, cnt, live, live ? __ldg(g.col_scale + n) : 0.0f,
                                  g.leak, g.v_th, x_lo ? g.row_scale + s0 * g.T : nullptr,
                                  g.out_half ? g.out_half + (size_t)s0 * g.T * g.out_pitch + n : nullptr, g.out_pitch,
                                  g.count ? g.count + (size_t)s0 * g.a + n : nullptr, g.a};
                    for (int sb = eh * 8; sb < cnt; sb += 16) {
                        if (g.reset == HSES_RESET_HARD) scan8<PERT, true>(sc, sb);
                        else scan8<PERT, false>(sc, sb);
                    }
                }
                tc_fence_before();
                mbar_arrive(&tempty[b]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ------------------------------------------------------------------------------ readout
struct ReadoutArgs {
    const float* count;          // spikes over the T steps (n, h)
    int T;
    const float* w;              // (classes, h)
    int64_t w_stride;
    int h, classes, r, bm;
    int64_t n, n_pop;            // samples, members
    int spb, slices, rows;       // samples per block, blocks per pair (noise: a block lies inside one pair), samples staged
    int32_t first_pair;
    const float *cache_a, *cache_b;
    NoiseCal cal;
    const uint64_t *jump, *lane4, *lane16;
    uint64_t key;
    int32_t true_epoch;
    float base_sigma, gain;
    const float* gain_ptr;
    float* logits;               // or NULL
    const int32_t* labels;       // or NULL
    int reward;
    float* per_sample;           // scores of single samples, when a block does not hold whole members
    float* raw_fitness;
};
// [Wᵀ | B] as one matrix of h rows, classes + r columns: the pitch is a multiple of four (16-byte broadcasts) and of no eight
__host__ __device__ inline int ro_pitch(int classes, int r) {
    const int j = (classes + r + 3) & ~3;
    return j % 8 ? j : j + 4;
}
__host__ __device__ inline size_t ro_floats(int h, int classes, int r, int rows) {
    const int j = ro_pitch(classes, r);
    return (size_t)h * j + (((size_t)r * classes + 3) & ~(size_t)3) + (size_t)rows * ((h | 1) + j + 1) + rows;
}

// The blocks of an antithetic pair (or, without noise, a slice of the samples each): W and the pair's factors in shared
// memory, [y | t] = counts·[Wᵀ | B] / T, logits = gain * (y ± t·(sA)ᵀ), then the score of every sample (snn_mnist.rs:180-201)
// and each member's mean.  A lane is a sample, a warp takes four columns at a time.  The whole is a chain of short phases,
// so its time is their latencies: 24 us with a thread per sample and column, a divide per rate and a block per pair of 128
// samples took 61.
__global__ void __launch_bounds__(256, 4) snn_readout_kernel(const __grid_constant__ ReadoutArgs g) {
    extern __shared__ __align__(16) float sm[];
    __shared__ CalTab tab;
    __shared__ uint64_t state_s[64];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = g.h, C = g.classes, r = g.r;
    const int J = ro_pitch(C, r), hp = h | 1, jp = J + 1;
    float* ms = sm;                                           // [h][J]
    float* as = ms + (size_t)h * J;                           // [r][C], scaled
    float* xs = as + ((r * C + 3) & ~3);                      // [rows][hp]
    float* ys = xs + g.rows * hp;                             // [rows][jp]
    float* fs = ys + g.rows * jp;                             // [rows]
    chain_begin();
    const int64_t p = r ? blockIdx.x / g.slices : 0;
    const int64_t s_lo = r ? p * 2 * g.bm + (int64_t)(blockIdx.x - p * g.slices) * g.spb : (int64_t)blockIdx.x * g.spb;
    const int64_t s_hi = min(s_lo + g.spb, r ? (p + 1) * 2 * g.bm : g.n);
    for (int c = warp; c < C; c += 8)
        for (int k = lane; k < h; k += 32) ms[(size_t)k * J + c] = __ldg(g.w + (int64_t)c * g.w_stride + k);
    for (int k = tid; k < h; k += 256)
        for (int j = C + r; j < ((C + r + 3) & ~3); ++j) ms[(size_t)k * J + j] = 0.0f;
    if (r) {
        const int nb = h * r, na = C * r;
        auto put = [&](int e, float z) {                      // value e of the pair's stream: B's rows, then A's
            if (e < nb) ms[(size_t)(e / r) * J + C + e % r] = z;
            else if (e < nb + na) as[(e - nb) % r * C + (e - nb) / r] = __fmul_rn(z, g.base_sigma);
        };
        if (g.cache_a) {
            for (int i = tid; i < nb; i += 256) put(i, __ldg(g.cache_b + p * nb + i));
            for (int i = tid; i < na; i += 256) put(nb + i, __ldg(g.cache_a + p * na + i));
        } else {
            NoiseCal cal = g.cal;
            stage_cal(cal, tab);
            const int cnt = nb + na;
            for (int base = 0; base < cnt; base += 32768) {
                __syncthreads();
                stream_fill(cal, g.jump, g.lane4, g.lane16,
                            noise_seed(g.key, g.true_epoch, g.first_pair + (int32_t)p) | 1ull, (uint64_t)base,
                            min(32768, cnt - base), state_s, [&](int off, float (&z)[4]) {
#pragma unroll
                                for (int j = 0; j < 4; ++j) put(base + off + j, z[j]);
                            });
            }
        }
    }
    const float gain = g.gain_ptr ? *g.gain_ptr : g.gain, steps = (float)g.T;
    float mean_sum = 0.0f;                                    // thread m: the running sum of the block's member m
    for (int64_t s0 = s_lo; s0 < s_hi; s0 += g.rows) {
        const int cnt = (int)min((int64_t)g.rows, s_hi - s0);
        for (int k = lane; k < h; k += 32)
            for (int s = warp; s < cnt; s += 64) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = s + 8 * i < cnt ? __ldg(g.count + (s0 + s + 8 * i) * h + k) : 0.0f;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (s + 8 * i < cnt) xs[(s + 8 * i) * hp + k] = v[i];
            }
        __syncthreads();
        const int cols = (C + r + 3) >> 2, blocks = (cnt + 31) >> 5;
        for (int i = warp; i < cols * blocks; i += 8) {
            const int rb = i / cols, j = (i - rb * cols) * 4, s = rb * 32 + lane;
            const float* x = xs + min(s, cnt - 1) * hp;
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
            for (int k = 0; k < h; ++k) {
                const float4 m = *reinterpret_cast<const float4*>(ms + (size_t)k * J + j);
                const float v = x[k];
                acc[0] = fmaf(v, m.x, acc[0]);
                acc[1] = fmaf(v, m.y, acc[1]);
                acc[2] = fmaf(v, m.z, acc[2]);
                acc[3] = fmaf(v, m.w, acc[3]);
            }
            if (s < cnt) {
#pragma unroll
                for (int q = 0; q < 4; ++q) ys[s * jp + j + q] = __fdiv_rn(acc[q], steps);   // the mean over T (snn.rs:278)
            }
        }
        __syncthreads();
        for (int i = warp; i < C * blocks; i += 8) {
            const int rb = i / C, c = i - rb * C, s = rb * 32 + lane;
            if (s >= cnt) continue;
            float y = ys[s * jp + c];
            if (r) {
                float u = 0.0f;
#pragma unroll 4
                for (int q = 0; q < r; ++q) u = fmaf(ys[s * jp + C + q], as[q * C + c], u);
                y = __fadd_rn(y, (((s0 + s) / g.bm) & 1) ? -u : u);
            }
            ys[s * jp + c] = __fmul_rn(y, gain);
        }
        __syncthreads();
        if (g.logits)
            for (int i = tid; i < cnt * C; i += 256) g.logits[s0 * C + i] = ys[i / C * jp + i % C];
        if (g.labels) {
            for (int s = tid; s < cnt; s += 256) {
                const float f = sample_fitness(ys + s * jp, C, g.labels[s0 + s], g.reward);
                fs[s] = f;
                if (g.per_sample) g.per_sample[s0 + s] = f;
            }
            __syncthreads();
            const int64_t m_lo = s_lo + (int64_t)tid * g.bm;  // samples in order, like member_mean
            if (!g.per_sample && m_lo < s_hi) {
                const int lo = (int)max((int64_t)0, m_lo - s0), hi = (int)min((int64_t)cnt, m_lo + g.bm - s0);
#pragma unroll 8
                for (int s = lo; s < hi; ++s) mean_sum = __fadd_rn(mean_sum, fs[s]);
                if (hi > lo && s0 + hi == m_lo + g.bm) g.raw_fitness[m_lo / g.bm] = __fdiv_rn(mean_sum, (float)g.bm);
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------- host side
struct LayerPlan {
    int exact, rows, spt, ppt, tpp, nt, r16, bn, n_chunks, groups, kp, ap, stages, stage_bytes, smem;
    int64_t tiles;
    size_t o_whi, o_wlo, o_cs, o_bhi, o_blo, o_aimg;
};
struct SnnPlan {
    bool ok;
    std::vector<LayerPlan> l;
    int64_t n, pairs;
    int ro_spb, ro_slices, ro_rows, ro_smem;
    bool ro_members;                 // the readout's blocks hold whole members
    size_t o_x, o_xlo, o_rs, o_h[2], o_rate, o_flag, o_per, bytes;
};

// would the layer's product run on linear_tc?
bool on_linear_tc(const hses_snn_model* m, const hses_pop_args* p, int l) {
    hses_linear_args g{};
    g.x = g.param = reinterpret_cast<const float*>(0x100);
    g.out = reinterpret_cast<float*>(0x100);
    g.t_steps = p->T;
    g.n_pop = p->n_pop;
    g.bm = p->bm;
    g.k = m->dims[l];
    g.a = m->dims[l + 1];
    g.x_row_stride = g.param_row_stride = g.k;
    g.out_row_stride = g.a;
    g.rank = p->rank;
    g.first_thread = p->first_thread;
    g.perturb = p->perturb;
    g.out_scale = 1.0f;
    return tensor_path_supports(g);
}

SnnPlan make_plan(const hses_snn_model* m, const hses_pop_args* p) {
    SnnPlan s{};
    const int hidden = m->n_layers - 1;
    if (hidden < 1 || hidden > kSnnMaxLayers || p->T < 1 || p->T > 128) return s;
    s.n = p->n_pop * p->bm;
    if (s.n >= (1ll << 31) || (double)s.n * p->T >= 2147483648.0) return s;
    const bool pert = p->perturb != 0;
    const int r = pert ? p->rank : 0;
    if (pert) {
        if (p->first_thread % 2 != 0 || p->n_pop % 2 != 0 || r < 1 || r > 64 || (int64_t)p->bm * 2 > (1 << 30)) return s;
        s.pairs = p->n_pop / 2;
        // one sample of each member against wide factors: bound by the factors' bytes, the per-pair kernel reads them
        // as they are in the cache and writes nothing back
        if ((int64_t)2 * p->bm * p->T <= 32 && r % 8 == 0 && r >= 32) return s;
    }
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 255) / 256 * 256;
        return at;
    };
    const int sms = plan_sm_count();
    for (int l = 0; l < hidden; ++l) {
        LayerPlan q{};
        const int k = m->dims[l], a = m->dims[l + 1];
        if (k > 65536 || a > 65536) return s;
        q.kp = (k + 7) & ~7;
        q.ap = (a + 7) & ~7;
        q.n_chunks = (a + 127) / 128;
        q.bn = ((a + q.n_chunks - 1) / q.n_chunks + 15) & ~15;
        if (pert) q.r16 = (r + 15) & ~15;
        // The tensor core truncates as it adds up; from the second block of k on a neuron near its threshold may decide otherwise.  Shapes
        // that linear_tc has no tile for were always fp32 multiply-adds and keep that accuracy: W's hi half on a fixed
        // grid, whose sums over spikes are exact, its lo half in an accumulator of its own.
        q.exact = k > 64 && !on_linear_tc(m, p, l);
        // Samples per tile and groups of chunks: the cheapest by a model of the kernel in cycles (measured at 784 -> 128 and
        // 128 -> 128, T = 8, rank 4).  Loads: 35 bytes per cycle reach an SM when all of them load; products: 8192 flop per
        // cycle; the rank term's way through shared memory and back: 2600; scan: 20 per row.  Tiles of 128 rows overlap the
        // scan with the next tile's products, taller ones read W less often.
        int64_t best = -1;
        for (int rows = q.exact ? 128 : 256; rows >= 128; rows -= 64)
            for (int cap = rows / p->T; cap >= 1; cap -= std::max(1, cap / 16)) {
                if ((p->T - 1) * cap + ((cap + 7) & ~7) > rows) continue;   // the scan reads eight columns at a time
                LayerPlan t = q;
                t.rows = rows;
                t.tpp = 1;
                t.ppt = 0;
                if (pert) {
                    const int spp = 2 * p->bm;
                    if (spp <= cap) {
                        t.ppt = (int)std::min<int64_t>({cap / spp, 64 / q.r16, s.pairs});
                        t.spt = t.ppt * spp;
                        t.tiles = (s.pairs + t.ppt - 1) / t.ppt;
                    } else {
                        t.tpp = (spp + cap - 1) / cap;
                        t.spt = (spp + t.tpp - 1) / t.tpp;
                        t.tiles = s.pairs * t.tpp;
                    }
                    t.nt = std::max(t.ppt, 1) * q.r16;
                } else {
                    t.spt = cap;
                    t.tiles = (s.n + cap - 1) / cap;
                }
                const int used = t.spt * p->T;
                if (used <= rows - 64 && rows > 128) continue;
                t.stage_bytes = rows * 128 + 2 * SL_OPERAND + t.nt * 256;
                const int fixed = 1024 + 3 * t.nt * rows * 2;
                t.stages = std::min(SL_MAX_STAGES, (SL_SMEM_LIMIT - 1024 - fixed) / t.stage_bytes);
                t.smem = fixed + t.stages * t.stage_bytes;
                if (t.stages < 2) continue;
                const int64_t load = ((int64_t)used * 128 + 2 * q.bn * 128 + t.nt * 256) / 35;
                const int64_t mma = 4 * ((int64_t)used + (pert ? (used + 127) / 128 * std::max(32, t.nt) : 0));
                const int64_t rank = pert ? 2600 + (int64_t)std::max(1, t.ppt) * q.r16 / 16 * 6 * used / 2 : 0;
                const int64_t block = std::max(load, mma) + (t.stages == 2 ? std::min(load, mma) / 2 : 0);   // two hide less
                const int64_t front = (k + 63) / 64 * block + rank, scan = 600 + 20 * (int64_t)used;
                const int64_t chunk = pert && (rows > 128 || q.exact) ? front + scan : std::max(front, scan);
                for (int gr = 1; gr <= q.n_chunks; ++gr) {
                    const int64_t waves = (t.tiles * gr + sms - 1) / sms;
                    const int64_t cost = waves * ((q.n_chunks + gr - 1) / gr) * chunk + front + scan - chunk;
                    if (best < 0 || cost < best) {
                        best = cost;
                        t.groups = gr;
                        q = t;
                    }
                }
            }
        if (best < 0) return s;
        q.o_whi = take((size_t)a * q.kp * 2);
        q.o_wlo = take((size_t)a * q.kp * 2);
        q.o_cs = take((size_t)a * 4);
        if (pert) {
            q.o_bhi = take((size_t)s.pairs * q.r16 * q.kp * 2);
            q.o_blo = take((size_t)s.pairs * q.r16 * q.kp * 2);
            q.o_aimg = take((size_t)s.pairs * q.n_chunks * q.r16 * 3 * q.bn * 2);
        }
        s.l.push_back(q);
    }
    // readout: everything of a block in shared memory
    const int h = m->dims[hidden], C = m->dims[hidden + 1];
    // Blocks of whole members take their means themselves: a pair, or a member from 33 samples on.
    s.ro_slices = 1;
    if (pert) {
        s.ro_members = p->bm <= 128;
        s.ro_spb = 2 * p->bm <= 64 ? 2 * p->bm : s.ro_members ? p->bm : 64;
        s.ro_slices = (2 * p->bm + s.ro_spb - 1) / s.ro_spb;
    } else {
        s.ro_members = p->bm <= 64;
        s.ro_spb = s.ro_members ? p->bm * (64 / p->bm) : 64;
    }
    s.ro_rows = std::min(64, (s.ro_spb + 31) & ~31);
    while (s.ro_rows > 8 && ro_floats(h, C, r, s.ro_rows) * 4 > 100 * 1024) s.ro_rows /= 2;
    if (ro_floats(h, C, r, s.ro_rows) * 4 > 200 * 1024) return s;
    s.ro_smem = (int)(ro_floats(h, C, r, s.ro_rows) * 4);
    const size_t rows = (size_t)p->T * s.n;
    s.o_x = take(rows * s.l[0].kp * 2);
    s.o_xlo = take(rows * s.l[0].kp * 2);
    s.o_rs = take(rows * 4);
    for (int i = 0; i < 2; ++i) {
        size_t w = 0;
        for (int l = i; l + 1 < hidden; l += 2) w = std::max(w, (size_t)s.l[l].ap);
        s.o_h[i] = take(rows * w * 2);
    }
    s.o_rate = take((size_t)s.n * h * 4);
    s.o_per = take((size_t)s.n * 4);
    s.o_flag = take(4);
    s.bytes = o + 256;
    s.ok = s.bytes <= (24ull << 30);
    return s;
}

// A step asks for its plan four times (the choice of path, sizes, the run): each thread keeps its last one.
const SnnPlan& plan_snn(const hses_snn_model* m, const hses_pop_args* p) {
    using Key = std::array<int64_t, kSnnMaxLayers + 12>;
    thread_local Key last{};
    thread_local SnnPlan plan{};
    Key key{};
    key[0] = m->n_layers;
    for (int l = 0; l <= m->n_layers && l < kSnnMaxLayers + 3; ++l) key[1 + l] = m->dims[l];
    int64_t* k = key.data() + kSnnMaxLayers + 4;
    k[0] = p->T;
    k[1] = p->n_pop;
    k[2] = p->bm;
    k[3] = p->perturb;
    k[4] = p->rank;
    k[5] = p->first_thread % 2;
    k[6] = plan_sm_count();
    if (key != last) {
        plan = make_plan(m, p);
        last = key;
    }
    return plan;
}

int encode_2d(CUtensorMap* map, const void* base, int64_t rows, int cols, int pitch, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return HSES_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)pitch * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
        return HSES_ERR_CUDA;
    }
    return HSES_OK;
}
// spikes (n, T, k) with rows of `pitch` values; a box is 64 inputs of spt samples x T steps, step by step
int encode_spikes(CUtensorMap* map, const void* base, int64_t n, int T, int k, int pitch, int spt) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return HSES_ERR_CUDA;
    }
    cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)n, (cuuint64_t)T};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 2 * (cuuint64_t)T, (cuuint64_t)pitch * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)spt, (cuuint32_t)T};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (spikes) failed with code " + std::to_string((int)r));
        return HSES_ERR_CUDA;
    }
    return HSES_OK;
}
}  // namespace

bool snn_fused_supports(const hses_snn_model* m, const hses_pop_args* p) { return plan_snn(m, p).ok; }

size_t snn_fused_workspace_bytes(const hses_snn_model* m, const hses_pop_args* p) { return plan_snn(m, p).bytes; }

int run_snn_fused(hses_ctx* ctx, cudaStream_t st, const hses_snn_model* m, const hses_pop_args* p, const SnnInput& in,
                  float* logits, const SnnScore& score, void* workspace, size_t workspace_bytes) {
    const SnnPlan& s = plan_snn(m, p);
    HSES_REQUIRE(s.ok, "shape not covered");
    HSES_REQUIRE(workspace != nullptr && workspace_bytes >= s.bytes, "workspace too small");
    HSES_REQUIRE(p->noise_reuse >= 0 && p->first_thread >= 0, "negative thread id or noise_reuse");
    uint8_t* ws = reinterpret_cast<uint8_t*>(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    auto half_at = [&](size_t o) { return reinterpret_cast<__half*>(ws + o); };
    auto float_at = [&](size_t o) { return reinterpret_cast<float*>(ws + o); };
    const int hidden = m->n_layers - 1;
    const bool pert = p->perturb != 0;
    const int64_t rows = (int64_t)p->T * s.n;
    const int32_t te = true_epoch_of(p->epoch, p->noise_reuse);
    int* flag = reinterpret_cast<int*>(ws + s.o_flag);

    const int k0 = m->dims[0], kp0 = s.l[0].kp;
    // ---- weights of every hidden layer ----
    {
        SplitJobs jobs{};
        jobs.n = hidden;
        jobs.clear = in.images ? nullptr : flag;
        int widest = 0, blocks = 0;
        for (int l = 0; l < hidden; ++l) widest = std::max(widest, s.l[l].kp);
        const int rpb = widest <= 1024 ? 16 : 8;   // rows per block
        for (int l = 0; l < hidden; ++l) {
            const LayerPlan& q = s.l[l];
            const int vec = ((uintptr_t)m->weights[l] & 15u) == 0 && m->weight_strides[l] % 4 == 0;
            jobs.j[l] = SplitJob{m->weights[l], m->weight_strides[l], m->dims[l + 1], m->dims[l], q.kp, vec, half_at(q.o_whi),
                                 half_at(q.o_wlo), float_at(q.o_cs), nullptr, q.exact};
            jobs.block0[l] = blocks;
            blocks += (m->dims[l + 1] + rpb - 1) / rpb;
        }
        HSES_KERNEL(ctx, st, "snn_split_w");
        if (widest <= 1024)
            chain_launch(snn_split_w_kernel<8, 2>, (unsigned)blocks, 256, 0, st, jobs);
        else
            chain_launch(snn_split_w_kernel<0, 1>, (unsigned)blocks, 256, 0, st, jobs);
        HSES_LAUNCH_CHECK();
    }
    // ---- input spikes ----
    if (in.images) {
        HSES_REQUIRE((double)s.n * k0 < 4294967296.0, "batch*in_dim must fit the 32-bit element index of the reference stream");
        const uint32_t mix = in.seeds[0] ^ in.seeds[1] ^ in.seeds[2] ^ in.seeds[3];
        const int64_t total = s.n * (kp0 / 8);
        HSES_KERNEL(ctx, st, "encode_half");
        chain_launch(encode_half_kernel, (unsigned)((total + 255) / 256), 256, 0, st, in.images, s.n, k0, in.stride, p->T, mix, half_at(s.o_x),
                                                                           kp0);
        HSES_LAUNCH_CHECK();
    } else {
        const int64_t total = rows * (kp0 / 8);
        {
            HSES_KERNEL(ctx, st, "spikes_half");
            chain_launch(spikes_half_kernel, (unsigned)((total + 255) / 256), 256, 0, st, in.spikes, s.n, p->T, k0, in.stride, half_at(s.o_x), kp0,
                                                                               flag);
            HSES_LAUNCH_CHECK();
        }
        RowMap map{};
        map.rows = rows;
        map.packed = 2;
        map.t_steps = p->T;
        map.n_pop = s.n;
        const int vec = ((uintptr_t)in.spikes & 15u) == 0 && in.stride % 4 == 0;
        const SplitJob j{in.spikes, in.stride, rows, k0, kp0, vec, half_at(s.o_x), half_at(s.o_xlo), float_at(s.o_rs), flag};
        HSES_KERNEL(ctx, st, "split_if_inexact");
        if (kp0 <= 1024)
            chain_launch(split_if_inexact_kernel<8, 2>, 4 * ctx->sm_count, 256, 0, st, j, map);
        else
            chain_launch(split_if_inexact_kernel<0, 1>, 4 * ctx->sm_count, 256, 0, st, j, map);
        HSES_LAUNCH_CHECK();
    }

    // ---- factors of every hidden layer ----
    if (pert) {
        FactorJobs jobs{};
        jobs.n = hidden;
        int64_t blocks = 0;
        for (int l = 0; l < hidden; ++l) {
            const LayerPlan& q = s.l[l];
            FactorJob& f = jobs.j[l];
            const hses_factor_cache* c = m->caches ? m->caches[l] : nullptr;
            if (c) {
                hses_linear_args la{};
                la.cache = c;
                la.key = m->keys[l];
                la.epoch = p->epoch;
                la.noise_reuse = p->noise_reuse;
                la.rank = p->rank;
                la.a = m->dims[l + 1];
                la.k = m->dims[l];
                la.first_thread = p->first_thread;
                la.n_pop = p->n_pop;
                int rc = resolve_factor_cache(la, &f.cache_a, &f.cache_b);
                if (rc != HSES_OK) return rc;
            }
            f.jump = ctx->t.jump_tabs;
            f.lane4 = ctx->t.jump_lane4;
            f.lane16 = ctx->t.jump_lane16;
            f.cal = ctx->cal();
            f.key = m->keys[l];
            f.true_epoch = te;
            f.first_pair = p->first_thread / 2;
            f.pairs = s.pairs;
            f.r = p->rank;
            f.r16 = q.r16;
            f.k = m->dims[l];
            f.kp = q.kp;
            f.a = m->dims[l + 1];
            f.row_a0 = f.k;
            f.row_b0 = 0;
            f.bn = q.bn;
            f.n_chunks = q.n_chunks;
            f.kb = q.r16;
            f.base_sigma = p->sigma / sqrtf((float)p->rank);
            f.col_scale = float_at(q.o_cs);
            f.bhi = half_at(q.o_bhi);
            f.blo = half_at(q.o_blo);
            f.aimg = reinterpret_cast<__nv_bfloat16*>(ws + q.o_aimg);
            jobs.segs[l] = plan_segments(f, ctx->sm_count);
            jobs.block0[l] = blocks;
            blocks += s.pairs * jobs.segs[l];
        }
        HSES_REQUIRE(blocks < (1ll << 31), "too many pairs");
        HSES_KERNEL(ctx, st, "snn_factors");
        chain_launch(snn_factors_kernel, (unsigned)blocks, 256, 0, st, jobs);
        HSES_LAUNCH_CHECK();
    }

    // ---- hidden layers ----
    for (int l = 0; l < hidden; ++l) {
        const LayerPlan& q = s.l[l];
        const bool last = l + 1 == hidden;
        LayerArgs a{};
        a.T = p->T;
        a.spt = q.spt;
        a.rows = q.rows;
        a.exact = q.exact;
        a.k_blocks = (m->dims[l] + 63) / 64;
        a.nt = q.nt;
        if (pert) {
            const int most = 64 / q.nt, len = (a.k_blocks + most - 1) / most;   // k-blocks per sum of t, see the kernel
            a.t_chains = (a.k_blocks + len - 1) / len;
        }
        a.n = s.n;
        a.tiles = q.tiles;
        a.ppt = q.ppt;
        a.tpp = q.tpp;
        a.spp = 2 * p->bm;
        a.bm = p->bm;
        a.groups = q.groups;
        a.n_chunks = q.n_chunks;
        a.bn = q.bn;
        a.a = m->dims[l + 1];
        a.r16 = q.r16;
        a.pairs = s.pairs;
        a.aimg = reinterpret_cast<const __nv_bfloat16*>(ws + q.o_aimg);
        a.row_scale = float_at(s.o_rs);
        a.col_scale = float_at(q.o_cs);
        a.inexact = l == 0 && !in.images ? flag : nullptr;
        a.leak = 1.0f / m->tau_m;
        a.v_th = m->v_th[l];
        a.reset = m->reset_mode;
        a.out_half = last ? nullptr : half_at(s.o_h[l & 1]);
        a.out_pitch = q.ap;
        a.count = last ? float_at(s.o_rate) : nullptr;
        a.stages = q.stages;
        a.stage_bytes = q.stage_bytes;
        a.status = ctx->t.status_word;
        const void* x = l == 0 ? half_at(s.o_x) : half_at(s.o_h[(l - 1) & 1]);
        const int pitch = l == 0 ? kp0 : s.l[l - 1].ap;
        CUtensorMap mx, mxl, mw, mwl, mb, mbl;
        int rc = encode_spikes(&mx, x, s.n, p->T, m->dims[l], pitch, q.spt);
        if (rc == HSES_OK) rc = encode_spikes(&mxl, l == 0 ? half_at(s.o_xlo) : x, s.n, p->T, m->dims[l], pitch, q.spt);
        if (rc == HSES_OK) rc = encode_2d(&mw, half_at(q.o_whi), a.a, q.kp, q.kp, q.bn);
        if (rc == HSES_OK) rc = encode_2d(&mwl, half_at(q.o_wlo), a.a, q.kp, q.kp, q.bn);
        mb = mw;
        mbl = mwl;
        if (rc == HSES_OK && pert) rc = encode_2d(&mb, half_at(q.o_bhi), s.pairs * q.r16, q.kp, q.kp, q.nt);
        if (rc == HSES_OK && pert)
            rc = encode_2d(&mbl, half_at(q.o_blo), s.pairs * q.r16, q.kp, q.kp, q.nt);
        if (rc != HSES_OK) return rc;
        const unsigned grid = (unsigned)std::min<int64_t>(q.tiles * q.groups, ctx->sm_count);
        auto kernel = pert ? snn_layer_kernel<true> : snn_layer_kernel<false>;
        HSES_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, q.smem));
        HSES_KERNEL(ctx, st, "snn_layer");
        chain_launch(kernel, grid, pert ? SL_THREADS_T : SL_THREADS, q.smem, st, mx, mxl, mw, mwl, mb, mbl, a);
        HSES_LAUNCH_CHECK();
    }

    // ---- readout and score ----
    ReadoutArgs o{};
    o.count = float_at(s.o_rate);
    o.T = p->T;
    o.w = m->weights[hidden];
    o.w_stride = m->weight_strides[hidden];
    o.h = m->dims[hidden];
    o.classes = m->dims[hidden + 1];
    o.r = pert ? p->rank : 0;
    o.bm = p->bm;
    o.n = s.n;
    o.n_pop = p->n_pop;
    o.spb = s.ro_spb;
    o.slices = s.ro_slices;
    o.rows = s.ro_rows;
    o.first_pair = p->first_thread / 2;
    if (pert) {
        o.cal = ctx->cal();
        o.jump = ctx->t.jump_tabs;
        o.lane4 = ctx->t.jump_lane4;
        o.lane16 = ctx->t.jump_lane16;
        o.key = m->keys[hidden];
        o.true_epoch = te;
        o.base_sigma = p->sigma / sqrtf((float)p->rank);
        const hses_factor_cache* c = m->caches ? m->caches[hidden] : nullptr;
        if (c) {
            hses_linear_args la{};
            la.cache = c;
            la.key = m->keys[hidden];
            la.epoch = p->epoch;
            la.noise_reuse = p->noise_reuse;
            la.rank = p->rank;
            la.a = o.classes;
            la.k = o.h;
            la.first_thread = p->first_thread;
            la.n_pop = p->n_pop;
            int rc = resolve_factor_cache(la, &o.cache_a, &o.cache_b);
            if (rc != HSES_OK) return rc;
        }
    }
    o.gain = m->out_gain;
    o.gain_ptr = m->out_gain_dev;
    o.logits = logits;
    o.labels = score.labels;
    o.reward = score.reward;
    o.raw_fitness = score.raw_fitness;
    o.per_sample = score.labels && !s.ro_members ? float_at(s.o_per) : nullptr;
    {
        const int64_t blocks = pert ? s.pairs * s.ro_slices : (s.n + s.ro_spb - 1) / s.ro_spb;
        HSES_CUDA(cudaFuncSetAttribute(snn_readout_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, s.ro_smem));
        HSES_KERNEL(ctx, st, "snn_readout");
        chain_launch(snn_readout_kernel, (unsigned)blocks, 256, s.ro_smem, st, o);
        HSES_LAUNCH_CHECK();
    }
    if (o.per_sample) return hses_member_mean(ctx, reinterpret_cast<hses_stream>(st), o.per_sample, p->n_pop, p->bm, score.raw_fitness);
    return HSES_OK;
}

}  // namespace hses
