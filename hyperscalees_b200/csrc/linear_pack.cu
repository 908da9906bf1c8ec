// Tensor-core path of the perturbed linear layer (do_mm, hyperscalees-noiser/src/eggroll.rs:419-446,
// + lif_step, snn.rs:53-65) for shapes that fit no tile: any number of rows, samples per member, inputs
// and outputs, any pitch, ranks up to 128.  linear_tc.cu keeps the tile-aligned shapes.
//
// The rows of an antithetic pair (both members, all time steps) are packed next to each other and padded
// to a multiple of 32 (64 or 128 for wide ranks), so that a 32-row slice of a 128-row tile always belongs
// to one pair.  Both products of the rank-r term then run on the tensor cores as well: t = x·B is a
// second, narrow product over the same x tiles (the B blocks of the tile's pairs side by side), and
// t·(sA)ᵀ extends the K dimension of the main product (t in the columns of its own pair, zeros elsewhere),
// so the epilogue only scales and stores.
//
//   launch 1  pack_split_w     rows of W: a power of two each, then fp16 hi + lo
//   launch 2  pack_operands    x rows in packed order as fp16 hi + lo; the factors, regenerated from the
//                              stream or read from a cache, as B (K-major fp16 hi + lo, fixed scale 2^11)
//                              and A (three bf16 parts, scaled by s and by the scale of W's row)
//   launch 3  linear_pack      persistent, ten warps: TMA producer, MMA issuer, eight epilogue warps
//
// linear_pack waits for its copies more than for the L2 (31 %), DRAM or the tensor pipe (below 30 %): what counts is the
// bytes in flight, so the store buffer holds 16 rows, which leaves room for a third stage at 128 columns, t takes no more
// columns than there are pairs, and the operands' rows start at a 128-byte line.  1022 members x 36 rows, 500 -> 250,
// rank 8: 108 us with two stages, 97 with three, 90 with aligned rows.
// Products of x, W and B are hi*hi + hi*lo + lo*hi in fp16 (2^-21 relative residue); t and A are split into
// three bf16 parts (24 bits, six products): bf16 has the exponent range of fp32, so that the rank-r term
// can be accumulated on top of the main product in its scale.  No multicast, no cluster launch; every wait
// is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "linear.cuh"
#include "pack.cuh"

namespace hses {

namespace {

using namespace tc;
using namespace pack;

constexpr int PK_TILE = 128;       // rows per tile
constexpr int PK_BK = 64;          // fp16 values per k-block (one 128-byte swizzle row)
constexpr int PK_THREADS = 320;    // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int PK_MAX_STAGES = 6;
constexpr int PK_SMEM_LIMIT = 232448;
constexpr int PK_TR_PITCH = 17;    // staged 16 x 16 output block of an epilogue warp
constexpr int PK_TR_BYTES = 8 * 16 * PK_TR_PITCH * 4;

template <int NJ, int RPW>
__global__ void __launch_bounds__(256) pack_split_kernel(SplitJob j, RowMap map, int* clear) {
    chain_begin();
    if (clear && blockIdx.x == 0 && threadIdx.x == 0) *clear = 0;
    split_rows<NJ, RPW>(j, map, blockIdx.x);
}

// x rows and factors in one launch: the first x_blocks blocks split rows, the others take (pair, segment).
template <int NJ, int RPW>
__global__ void __launch_bounds__(256) pack_operands_kernel(SplitJob x, RowMap map, int64_t x_blocks, int segs, FactorJob f) {
    __shared__ __align__(16) float buf[PK_SEG];
    __shared__ CalTab tab;
    __shared__ uint64_t state_s[32];
    const int64_t b = blockIdx.x;
    chain_next();
    if (b < x_blocks) {
        chain_wait();
        split_rows<NJ, RPW>(x, map, b);
    } else {
        const int64_t i = b - x_blocks;
        factor_segment(f, i / segs, (int)(i % segs), buf, tab, state_s);
    }
}

// ----------------------------------------------------------------------------- product
struct PackArgs {
    RowMap map;
    int64_t m_tiles;
    int groups;            // column-chunk groups a tile's work is cut into
    int n_chunks, bn, a, k_blocks;
    int nt;                // columns of t in a tile: pairs per tile * r16
    int r16, kb;
    int rb;                // 32-row blocks per pair
    int64_t pairs;
    const __nv_bfloat16* aimg;
    const float *row_scale, *col_scale;
    const int* x_lo_flag;
    int lif;
    float leak, v_th, out_scale;
    const float* out_scale_ptr;
    float* out;
    int64_t out_stride;
    float* pot;
    int stages, stage_bytes;
    int staged_stores;     // room for the transposed store buffer
    int* status;
};

template <bool PERT>
__global__ void __launch_bounds__(PK_THREADS, 1)
linear_pack_kernel(const __grid_constant__ CUtensorMap tm_xhi, const __grid_constant__ CUtensorMap tm_xlo,
                   const __grid_constant__ CUtensorMap tm_whi, const __grid_constant__ CUtensorMap tm_wlo,
                   const __grid_constant__ CUtensorMap tm_bhi, const __grid_constant__ CUtensorMap tm_blo,
                   const PackArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int X_BYTES = PK_TILE * PK_BK * 2;
    const int w_bytes = g.bn * PK_BK * 2, b_bytes = g.nt * PK_BK * 2;
    uint8_t* tpp = smem + (size_t)g.stages * g.stage_bytes;            // [part 3][nt / 8][128][8] bf16
    const int part_bytes = g.nt * PK_TILE * 2;
    float* tr = reinterpret_cast<float*>(tpp + (PERT ? 3 * part_bytes : 0));
    __shared__ uint64_t full[PK_MAX_STAGES], empty[PK_MAX_STAGES], tfull[2], tempty[2], tacc, tready;
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
    chain_wait();                          // before the allocation: a waiting block holds no tensor memory
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(PERT ? 512 : 256)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_next();
    const uint32_t tmem = tmem_slot;       // accumulators at columns 0 and 128, t at 256
    const int64_t units = g.m_tiles * g.groups;
    const int nkb = PERT ? g.r16 / g.kb : 1;
    // pairs of tile mt: first one and count
    auto pairs_of = [&](int64_t mt, int64_t& p0) {
        p0 = (mt * 4) / g.rb;
        const int64_t last = min((mt * 4 + 3) / (int64_t)g.rb, g.pairs - 1);
        return (int)(last - p0) + 1;
    };

    if (warp == 0) {
        if (lane == 0) {
            Ring ring{0, 0};
            bool ok = true;
            const bool skip_xlo = *g.x_lo_flag == 0;
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
                int64_t p0 = 0;
                int nd = 0;
                if (PERT) {
                    nd = pairs_of(mt, p0);
                    for (int kb = 0; kb < g.k_blocks; ++kb, ring.next(g.stages)) {
                        uint8_t* st = slot((skip_xlo ? 1 : 2) * X_BYTES + 2 * b_bytes);
                        if (!ok) break;
                        uint64_t* bar = &full[ring.s];
                        tma_load_2d(st, &tm_xhi, kb * PK_BK, (int)(mt * PK_TILE), bar);
                        if (!skip_xlo) tma_load_2d(st + X_BYTES, &tm_xlo, kb * PK_BK, (int)(mt * PK_TILE), bar);
                        tma_load_2d(st + 2 * X_BYTES, &tm_bhi, kb * PK_BK, (int)(p0 * g.r16), bar);
                        tma_load_2d(st + 2 * X_BYTES + b_bytes, &tm_blo, kb * PK_BK, (int)(p0 * g.r16), bar);
                    }
                }
                for (int c = c0; c < c1 && ok; ++c) {
                    for (int kb = 0; kb < g.k_blocks; ++kb, ring.next(g.stages)) {
                        uint8_t* st = slot((skip_xlo ? 1 : 2) * X_BYTES + 2 * w_bytes);
                        if (!ok) break;
                        uint64_t* bar = &full[ring.s];
                        tma_load_2d(st, &tm_xhi, kb * PK_BK, (int)(mt * PK_TILE), bar);
                        if (!skip_xlo) tma_load_2d(st + X_BYTES, &tm_xlo, kb * PK_BK, (int)(mt * PK_TILE), bar);
                        tma_load_2d(st + 2 * X_BYTES, &tm_whi, kb * PK_BK, c * g.bn, bar);
                        tma_load_2d(st + 2 * X_BYTES + w_bytes, &tm_wlo, kb * PK_BK, c * g.bn, bar);
                    }
                    if (PERT) {
                        const uint32_t bytes = 3u * g.kb * g.bn * 2;
                        for (int i = 0; i < nd * nkb && ok; ++i, ring.next(g.stages)) {
                            uint8_t* st = slot(bytes);
                            if (!ok) break;
                            const int d = i / nkb, kblk = i - d * nkb;
                            const size_t img = (((size_t)(p0 + d) * g.n_chunks + c) * nkb + kblk) * 3 * g.kb * g.bn;
                            bulk_load(st, g.aimg + img, bytes, &full[ring.s]);
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
        // the whole warp runs the loop, so that addresses and descriptors stay warp-uniform; an elected lane issues (one
        // lane in a branch of its own took about 128 cycles per product, twice what the tensor core does)
        const uint32_t idesc = make_idesc(g.bn), idesc_t = make_idesc(PERT ? g.nt : 16), idesc_u = make_idesc_bf16(g.bn);
        const uint64_t desc0 = make_smem_desc(smem), desc_step = (uint64_t)(g.stage_bytes >> 4);
        const uint64_t plain0 = make_plain_desc(smem, g.bn * 16), plain_t = make_plain_desc(tpp, PK_TILE * 16);
        const uint32_t a1 = (uint32_t)g.kb * g.bn * 2 >> 4, t1 = (uint32_t)part_bytes >> 4;   // one part of an image block, of t
        uint32_t acc_it = 0, unit_no = 0;
        Ring ring{0, 0};
        bool ok = true;
        const bool skip_xlo = *g.x_lo_flag == 0;
        auto arrive = [&]() -> bool {
            ok = __all_sync(0xffffffffu, mbar_wait(&full[ring.s], ring.ph, abort_flag, g.status, 3));
            if (ok) tc_fence_after();
            return ok;
        };
        // three fp16 passes over one k-block
        auto three = [&](uint32_t d, uint32_t bytes, uint32_t id, bool first) {
            const uint64_t xh = desc0 + __shfl_sync(0xffffffffu, ring.s, 0) * desc_step, xl = xh + (X_BYTES >> 4);
            const uint64_t wh = xl + (X_BYTES >> 4), wl = wh + (bytes >> 4);
#pragma unroll
            for (int ks = 0; ks < PK_BK / 16; ++ks) {             // 16 fp16 = 32 bytes along k
                const uint32_t acc = !(first && ks == 0);
                if (!skip_xlo) umma_f16_warp(d, xl + 2 * ks, wh + 2 * ks, id, acc);
                umma_f16_warp(d, xh + 2 * ks, wl + 2 * ks, id, skip_xlo ? acc : 1u);
                umma_f16_warp(d, xh + 2 * ks, wh + 2 * ks, id, 1);
            }
            umma_commit_warp(&empty[ring.s]);
        };
        for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x, ++unit_no) {
            const int64_t mt = u / g.groups;
            const int grp = (int)(u - mt * g.groups);
            const int c0 = g.n_chunks * grp / g.groups, c1 = g.n_chunks * (grp + 1) / g.groups;
            int64_t p0 = 0;
            int nd = 0;
            if (PERT) {
                nd = pairs_of(mt, p0);
                for (int kb = 0; kb < g.k_blocks; ++kb, ring.next(g.stages)) {
                    if (!arrive()) break;
                    three(tmem + 256, (uint32_t)b_bytes, idesc_t, kb == 0);
                }
                if (!ok) break;
                umma_commit_warp(&tacc);
            }
            for (int c = c0; c < c1 && ok; ++c, ++acc_it) {
                const int b = acc_it & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(&tempty[b], ((acc_it >> 1) & 1) ^ 1, abort_flag, g.status, 2));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(b * 128);
                for (int kb = 0; kb < g.k_blocks; ++kb, ring.next(g.stages)) {
                    if (!arrive()) break;
                    three(d, (uint32_t)w_bytes, idesc, kb == 0);
                }
                if (PERT && ok) {
                    if (c == c0) ok = __all_sync(0xffffffffu, mbar_wait(&tready, unit_no & 1, abort_flag, g.status, 4));
                    if (!ok) break;
                    tc_fence_after();
                    for (int dd = 0; dd < nd && ok; ++dd)
                        for (int kblk = 0; kblk < nkb; ++kblk, ring.next(g.stages)) {
                            if (!arrive()) break;
                            const uint64_t da0 = plain0 + __shfl_sync(0xffffffffu, ring.s, 0) * desc_step;
                            for (int ks = 0; ks < g.kb / 16; ++ks) {
                                const uint64_t dt = plain_t + (uint64_t)(((dd * g.r16 + kblk * g.kb + ks * 16) >> 3) * PK_TILE);
                                const uint64_t da = da0 + (uint64_t)(ks * 2 * g.bn);
                                umma_f16_warp(d, dt + 2 * t1, da, idesc_u, 1);
                                umma_f16_warp(d, dt, da + 2 * a1, idesc_u, 1);
                                umma_f16_warp(d, dt + t1, da + a1, idesc_u, 1);
                                umma_f16_warp(d, dt + t1, da, idesc_u, 1);
                                umma_f16_warp(d, dt, da + a1, idesc_u, 1);
                                umma_f16_warp(d, dt, da, idesc_u, 1);
                            }
                            umma_commit_warp(&empty[ring.s]);
                        }
                }
                if (ok) umma_commit_warp(&tfull[b]);
                __syncwarp();
            }
        }
    } else {
        // ------------------------------------------------------------------------- epilogue
        const int q4 = warp & 3, eh = (warp - 2) >> 2;      // TMEM quadrant, column half
        const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16);
        const float gain = g.out_scale_ptr ? *g.out_scale_ptr : g.out_scale;
        const bool wide = (reinterpret_cast<uintptr_t>(g.out) & 31) == 0 && (g.out_stride & 7) == 0 && (g.a & 7) == 0 &&
                          (!g.pot || (reinterpret_cast<uintptr_t>(g.pot) & 31) == 0);
        float* my_tr = tr + (warp - 2) * 16 * PK_TR_PITCH;
        uint32_t acc_it = 0, unit_no = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x, ++unit_no) {
            const int64_t mt = u / g.groups;
            const int grp = (int)(u - mt * g.groups);
            const int c0 = g.n_chunks * grp / g.groups, c1 = g.n_chunks * (grp + 1) / g.groups;
            const int64_t p = mt * PK_TILE + q4 * 32 + lane;
            int64_t R;
            bool odd;
            const bool valid = map_row(g.map, p, R, odd);
            const float rs = !valid ? 0.0f : g.row_scale ? g.row_scale[p] : 1.0f;
            if (PERT) {
                if (!mbar_wait(&tacc, unit_no & 1, abort_flag, g.status, 5)) { ok = false; break; }
                tc_fence_after();
                const int64_t p0 = (mt * 4) / g.rb;
                const int d = (int)((mt * 4 + q4) / (int64_t)g.rb - p0);
                for (int c8 = eh; c8 < g.nt / 8; c8 += 2) {
                    uint32_t w[3][4];
                    if (c8 * 8 >= d * g.r16 && c8 * 8 < (d + 1) * g.r16) {     // the columns of this slice's pair
                        uint32_t acc[8];
                        tmem_ld8(lane_base + 256 + c8 * 8, acc);
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            float v0 = __uint_as_float(acc[j]), v1 = __uint_as_float(acc[j + 1]);
                            if (odd) v0 = -v0, v1 = -v1;        // the odd member of a pair has A negated
#pragma unroll
                            for (int part = 0; part < 3; ++part) {
                                const __nv_bfloat162 b = __floats2bfloat162_rn(v0, v1);
                                w[part][j >> 1] = *reinterpret_cast<const uint32_t*>(&b);
                                v0 -= __bfloat162float(b.x);
                                v1 -= __bfloat162float(b.y);
                            }
                        }
                    } else {
#pragma unroll
                        for (int part = 0; part < 3; ++part) w[part][0] = w[part][1] = w[part][2] = w[part][3] = 0u;
                    }
#pragma unroll
                    for (int part = 0; part < 3; ++part)
                        *reinterpret_cast<uint4*>(tpp + part * part_bytes + c8 * (PK_TILE * 16) + (q4 * 32 + lane) * 16) =
                            make_uint4(w[part][0], w[part][1], w[part][2], w[part][3]);
                }
                fence_proxy_async();
                tc_fence_before();
                mbar_arrive(&tready);
            }
            for (int c = c0; c < c1 && ok; ++c, ++acc_it) {
                const int b = acc_it & 1;
                if (!mbar_wait(&tfull[b], (acc_it >> 1) & 1, abort_flag, g.status, 6)) { ok = false; break; }
                tc_fence_after();
                for (int cb = eh * 16; cb < g.bn; cb += 32) {
                    const int n0 = c * g.bn + cb;
                    if (n0 >= g.a) break;
                    uint32_t acc[16];
                    tmem_ld8_issue(lane_base + b * 128 + cb, *reinterpret_cast<uint32_t(*)[8]>(acc));
                    tmem_ld8_issue(lane_base + b * 128 + cb + 8, *reinterpret_cast<uint32_t(*)[8]>(acc + 8));
                    float cs[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) cs[j] = n0 + j < g.a ? __ldg(g.col_scale + n0 + j) : 0.0f;
                    tmem_ld_wait();
                    float v[16];     // the charge of a LIF step, or the scaled output
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        v[j] = __fmul_rn(__fmul_rn(__fmul_rn(__uint_as_float(acc[j]), rs), cs[j]), g.lif ? g.leak : gain);
                    if (wide) {
                        if (valid) {
                            float* o = g.out + (size_t)R * g.out_stride + n0;
                            float* q = g.pot ? g.pot + (size_t)R * g.out_stride + n0 : nullptr;
#pragma unroll
                            for (int h = 0; h < 16; h += 8) {
                                if (n0 + h >= g.a) break;
                                float s[8];
#pragma unroll
                                for (int j = 0; j < 8; ++j) s[j] = g.lif ? (v[h + j] >= g.v_th ? 1.0f : 0.0f) : v[h + j];
                                if (q) {
                                    *reinterpret_cast<float4*>(q + h) = make_float4(v[h], v[h + 1], v[h + 2], v[h + 3]);
                                    *reinterpret_cast<float4*>(q + h + 4) = make_float4(v[h + 4], v[h + 5], v[h + 6], v[h + 7]);
                                }
                                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + h), "f"(s[0]),
                                             "f"(s[1]), "f"(s[2]), "f"(s[3]), "f"(s[4]), "f"(s[5]), "f"(s[6]), "f"(s[7])
                                             : "memory");
                            }
                        }
                    } else if (g.staged_stores) {
                        // rows that start anywhere: through shared memory, 16 rows at a time, so that sixteen lanes
                        // write sixteen neighbouring values of a row
                        const int col = lane & 15;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if ((lane >> 4) == h) {
#pragma unroll
                                for (int j = 0; j < 16; ++j) my_tr[col * PK_TR_PITCH + j] = v[j];
                            }
                            __syncwarp();
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                const int row = 2 * i + (lane >> 4);
                                const int64_t Rr = __shfl_sync(0xffffffffu, R, h * 16 + row);
                                const bool vr = __shfl_sync(0xffffffffu, (int)valid, h * 16 + row) != 0;
                                const float x = my_tr[row * PK_TR_PITCH + col];
                                if (vr && n0 + col < g.a) {
                                    const size_t o = (size_t)Rr * g.out_stride + n0 + col;
                                    if (g.pot) g.pot[o] = x;
                                    g.out[o] = g.lif ? (x >= g.v_th ? 1.0f : 0.0f) : x;
                                }
                            }
                            __syncwarp();
                        }
                    } else if (valid) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (n0 + j < g.a) {
                                const size_t o = (size_t)R * g.out_stride + n0 + j;
                                if (g.pot) g.pot[o] = v[j];
                                g.out[o] = g.lif ? (v[j] >= g.v_th ? 1.0f : 0.0f) : v[j];
                            }
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PERT ? 512 : 256) : "memory");
    }
}

// ------------------------------------------------------------------------------ host side
struct PackPlan {
    bool ok;
    int rp, rb, r16, nt, kb, kp, pitch, bn, n_chunks, groups;
    int64_t pairs, rows, m_tiles;
    int stages, stage_bytes, staged, smem;
    size_t o_xhi, o_xlo, o_whi, o_wlo, o_rs, o_cs, o_bhi, o_blo, o_aimg, o_flag, bytes;
};

PackPlan plan_pack(const hses_linear_args& g) {
    PackPlan p{};
    const int64_t rows_nat = (int64_t)g.t_steps * g.n_pop * g.bm;
    p.kp = (g.k + 7) & ~7;
    p.pitch = (g.k + PK_BK - 1) / PK_BK * PK_BK;   // a box row of 128 bytes is one line of memory, not parts of two
    p.n_chunks = (g.a + 127) / 128;
    p.bn = ((g.a + p.n_chunks - 1) / p.n_chunks + 15) & ~15;
    p.n_chunks = (g.a + p.bn - 1) / p.bn;
    p.rows = rows_nat;
    p.rb = 1;
    if (g.perturb) {
        if (g.rank > 128) return p;
        const int64_t R = (int64_t)2 * g.bm * g.t_steps;
        p.r16 = g.rank <= 64 ? (g.rank + 15) & ~15 : 128;
        // a tile holds the t columns of all its pairs, at most 128 of them
        const int gran = p.r16 <= 32 ? 32 : p.r16 <= 64 ? 64 : 128;
        const int64_t rp = (R + gran - 1) / gran * gran;
        if (rp > (1 << 30)) return p;
        p.rp = (int)rp;
        p.rb = p.rp / 32;
        p.pairs = ((int64_t)g.first_thread + g.n_pop - 1) / 2 - g.first_thread / 2 + 1;
        const int nd = p.rp == 32 ? 4 : p.rp % 128 == 0 ? 1 : 2;
        p.nt = (int)std::min<int64_t>(nd, p.pairs) * p.r16;
        p.kb = std::min(p.r16, 64);
        p.rows = p.pairs * p.rp;
    }
    if (p.rows >= (1ll << 31) - 256) return p;
    p.m_tiles = (p.rows + PK_TILE - 1) / PK_TILE;
    // work units: an m-tile's chunks in 1 .. n_chunks groups, the number that makes the last wave cheapest (a
    // group repeats the tile's t product)
    const int sms = plan_sm_count();
    int64_t best = 0;
    for (int gr = 1; gr <= p.n_chunks; ++gr) {
        const int64_t waves = (p.m_tiles * gr + sms - 1) / sms;
        const int64_t cost = waves * ((int64_t)((p.n_chunks + gr - 1) / gr) * (p.bn + 32) + p.nt);
        if (gr == 1 || cost < best) {
            best = cost;
            p.groups = gr;
        }
    }
    p.stage_bytes = 2 * PK_TILE * PK_BK * 2 + 2 * std::max(p.bn, p.nt) * PK_BK * 2;
    const int fixed = 1024 + 3 * p.nt * PK_TILE * 2;
    p.staged = PK_SMEM_LIMIT - 1024 - fixed - PK_TR_BYTES >= 2 * p.stage_bytes;
    const int room = PK_SMEM_LIMIT - 1024 - fixed - (p.staged ? PK_TR_BYTES : 0);   // 1024: static shared memory
    p.stages = std::min(PK_MAX_STAGES, room / p.stage_bytes);
    if (p.stages < 2) return p;
    p.smem = fixed + (p.staged ? PK_TR_BYTES : 0) + p.stages * p.stage_bytes;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t nx = (size_t)p.rows * p.pitch * 2, nw = (size_t)g.a * p.pitch * 2;
    p.o_xhi = take(nx);
    p.o_xlo = take(nx);
    p.o_whi = take(nw);
    p.o_wlo = take(nw);
    p.o_rs = take((size_t)p.rows * 4);
    p.o_cs = take((size_t)g.a * 4);
    p.o_flag = take(4);
    if (g.perturb) {
        const size_t nb = (size_t)p.pairs * p.r16 * p.pitch * 2;
        p.o_bhi = take(nb);
        p.o_blo = take(nb);
        p.o_aimg = take((size_t)p.pairs * p.n_chunks * p.r16 * 3 * p.bn * 2);
    }
    p.bytes = o + 256;   // the base is rounded up to 256 bytes
    p.ok = p.bytes <= (24ull << 30);
    return p;
}

int encode_rows(CUtensorMap* map, const void* base, int64_t rows, int cols, int pitch, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return HSES_ERR_CUDA;
    }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)pitch * 2};
    cuuint32_t box[2] = {(cuuint32_t)PK_BK, (cuuint32_t)box_rows};
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

int vec_ok(const void* p, int64_t stride) { return ((uintptr_t)p & 15u) == 0 && stride % 4 == 0; }

}  // namespace

bool pack_path_supports(const hses_linear_args& g) {
    if (g.n_groups > 1 || g.x_op != HSES_X_NONE || g.lif == 2) return false;
    const PackPlan p = plan_pack(g);
    if (!p.ok || !g.perturb || p.m_tiles <= plan_sm_count()) return p.ok;
    // Beyond one wave, pairs of a few rows (2 .. 10 of a 32-row slice) may be so much padding that fp32 multiply-adds are
    // the faster ones.  Both in microseconds, fitted to 4246 members of 1 .. 5 rows, 288 -> 49 at rank 1 (110 here, 49 .. 73
    // there), 1000 -> 900 at rank 3 (735; 308 .. 1372), 300 -> 200 at rank 28 (215; 197 .. 397), and to 1246 members,
    // 302 -> 200 at rank 50 (147; 330): steps of a block of k in waves of tiles, bytes of padded rows and factors and
    // launches; multiply-adds at 13 T/s and the rank term, which grows with the rank and a pair's rows.
    const double R = 2.0 * g.bm * g.t_steps, k = g.k, a = g.a;
    const double waves = (double)((p.m_tiles + plan_sm_count() - 1) / plan_sm_count());
    const double pack = 39 + waves * (p.n_chunks + 1) * ((g.k + PK_BK - 1) / PK_BK) + 1.6e-6 * p.rows * k +
                        2.5e-6 * p.pairs * p.r16 * (k + a);
    const double fp32 = 25 + p.pairs * R * k * a / 13e6 + g.rank * R;
    return pack < fp32;
}

size_t pack_path_workspace_bytes(const hses_linear_args& g) { return plan_pack(g).bytes; }

int run_pack_path(hses_ctx* ctx, cudaStream_t st, const hses_linear_args& g) {
    const PackPlan p = plan_pack(g);
    HSES_REQUIRE(g.workspace != nullptr && g.workspace_bytes >= p.bytes,
                 "workspace too small; see hses_perturbed_linear_workspace_bytes");
    uint8_t* ws = reinterpret_cast<uint8_t*>(((uintptr_t)g.workspace + 255) & ~(uintptr_t)255);
    auto half_at = [&](size_t o) { return reinterpret_cast<__half*>(ws + o); };
    int* flag = reinterpret_cast<int*>(ws + p.o_flag);
    float* cs = reinterpret_cast<float*>(ws + p.o_cs);

    RowMap map{};
    map.packed = g.perturb ? 1 : 0;
    map.rp = p.rp;
    map.t_steps = g.t_steps;
    map.bm = g.bm;
    map.n_pop = g.n_pop;
    map.first_thread = g.first_thread;
    map.first_pair = g.first_thread / 2;
    map.rows = p.rows;
    RowMap plain{};
    plain.rows = g.a;

    const SplitJob jw{g.param, g.param_row_stride, g.a, g.k, p.kp, vec_ok(g.param, g.param_row_stride),
                      half_at(p.o_whi), half_at(p.o_wlo), cs, nullptr, 0, p.pitch};
    SplitJob jx{g.x, g.x_row_stride, p.rows, g.k, p.kp, vec_ok(g.x, g.x_row_stride),
                half_at(p.o_xhi), half_at(p.o_xlo), reinterpret_cast<float*>(ws + p.o_rs), flag, 0, p.pitch};
    // a caller-provided fp16 copy of an x that is exact in fp16 is the operand as it stands
    const bool x_ready = !g.perturb && g.x_half != nullptr && ((uintptr_t)g.x_half & 15u) == 0 && p.kp == g.k;

    FactorJob f{};
    int segs = 0;
    if (g.perturb) {
        if (g.cache) {
            int rc = resolve_factor_cache(g, &f.cache_a, &f.cache_b);
            if (rc != HSES_OK) return rc;
        }
        f.jump = ctx->t.jump_tabs;
        f.lane4 = ctx->t.jump_lane4;
        f.lane16 = ctx->t.jump_lane16;
        f.cal = ctx->cal();
        f.key = g.key;
        f.true_epoch = true_epoch_of(g.epoch, g.noise_reuse);
        f.first_pair = map.first_pair;
        f.pairs = p.pairs;
        f.r = g.rank;
        f.r16 = p.r16;
        f.k = g.k;
        f.kp = p.kp;
        f.pitch = p.pitch;
        f.a = g.a;
        f.row_a0 = g.factor_order == 1 ? 0 : g.k;
        f.row_b0 = g.factor_order == 1 ? g.a : 0;
        f.bn = p.bn;
        f.n_chunks = p.n_chunks;
        f.kb = p.kb;
        f.base_sigma = g.sigma / sqrtf((float)g.rank);
        f.col_scale = cs;
        f.bhi = half_at(p.o_bhi);
        f.blo = half_at(p.o_blo);
        f.aimg = reinterpret_cast<__nv_bfloat16*>(ws + p.o_aimg);
        segs = plan_segments(f, ctx->sm_count);
    }
    auto prepare = [&](auto nj_c, auto rpw_c) -> int {
        constexpr int NJ = decltype(nj_c)::value, RPW = decltype(rpw_c)::value;
        {
            HSES_KERNEL(ctx, st, "pack_split_w");
            chain_launch(pack_split_kernel<NJ, RPW>, (unsigned)((g.a + 8 * RPW - 1) / (8 * RPW)), 256, 0, st, jw, plain, flag);
            HSES_LAUNCH_CHECK();
        }
        const int64_t xb = x_ready ? 0 : (p.rows + 8 * RPW - 1) / (8 * RPW), fb = p.pairs * segs;
        HSES_REQUIRE(xb + fb < (1ll << 31), "too many rows");
        if (g.perturb) {
            HSES_KERNEL(ctx, st, "pack_operands");
            chain_launch(pack_operands_kernel<NJ, RPW>, (unsigned)(xb + fb), 256, 0, st, jx, map, xb, segs, f);
            HSES_LAUNCH_CHECK();
        } else if (xb) {
            HSES_KERNEL(ctx, st, "pack_split_x");
            chain_launch(pack_split_kernel<NJ, RPW>, (unsigned)xb, 256, 0, st, jx, map, nullptr);
            HSES_LAUNCH_CHECK();
        }
        return HSES_OK;
    };
    using std::integral_constant;
    // pieces of 128 values per row and rows in flight per warp: as many as the registers hold
    int rc = p.kp <= 128    ? prepare(integral_constant<int, 1>{}, integral_constant<int, 8>{})
             : p.kp <= 256  ? prepare(integral_constant<int, 2>{}, integral_constant<int, 4>{})
             : p.kp <= 1024 ? prepare(integral_constant<int, 8>{}, integral_constant<int, 2>{})
                            : prepare(integral_constant<int, 0>{}, integral_constant<int, 1>{});
    if (rc != HSES_OK) return rc;

    PackArgs a{};
    a.map = map;
    a.m_tiles = p.m_tiles;
    a.groups = p.groups;
    a.n_chunks = p.n_chunks;
    a.bn = p.bn;
    a.a = g.a;
    a.k_blocks = (g.k + PK_BK - 1) / PK_BK;
    a.nt = p.nt;
    a.r16 = p.r16;
    a.kb = p.kb;
    a.rb = p.rb;
    a.pairs = p.pairs;
    a.aimg = f.aimg;
    a.row_scale = x_ready ? nullptr : jx.inv_scale;
    a.col_scale = cs;
    a.x_lo_flag = flag;
    a.lif = g.lif;
    a.leak = g.lif ? 1.0f / g.tau_m : 0.0f;
    a.v_th = g.v_th;
    a.out_scale = g.out_scale;
    a.out_scale_ptr = g.out_scale_ptr;
    a.out = g.out;
    a.out_stride = g.out_row_stride;
    a.pot = g.lif ? g.potentials : nullptr;
    a.stages = p.stages;
    a.stage_bytes = p.stage_bytes;
    a.staged_stores = p.staged;
    a.status = ctx->t.status_word;
    CUtensorMap mx, mxl, mw, mwl, mb, mbl;
    const int xpitch = x_ready ? p.kp : p.pitch;
    const void* xhi = x_ready ? g.x_half : static_cast<const void*>(jx.hi);
    rc = encode_rows(&mx, xhi, p.rows, p.kp, xpitch, PK_TILE);
    if (rc == HSES_OK) rc = encode_rows(&mxl, x_ready ? g.x_half : static_cast<const void*>(jx.lo), p.rows, p.kp, xpitch, PK_TILE);
    if (rc == HSES_OK) rc = encode_rows(&mw, jw.hi, g.a, p.kp, p.pitch, p.bn);
    if (rc == HSES_OK) rc = encode_rows(&mwl, jw.lo, g.a, p.kp, p.pitch, p.bn);
    mb = mw;
    mbl = mwl;
    if (rc == HSES_OK && g.perturb) rc = encode_rows(&mb, f.bhi, p.pairs * p.r16, p.kp, p.pitch, p.nt);
    if (rc == HSES_OK && g.perturb) rc = encode_rows(&mbl, f.blo, p.pairs * p.r16, p.kp, p.pitch, p.nt);
    if (rc != HSES_OK) return rc;
    const int64_t units = p.m_tiles * p.groups;
    const unsigned grid = (unsigned)std::min<int64_t>(units, ctx->sm_count);
    HSES_KERNEL(ctx, st, "linear_pack");
    if (g.perturb) {
        HSES_CUDA(cudaFuncSetAttribute(linear_pack_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem));
        chain_launch(linear_pack_kernel<true>, grid, PK_THREADS, p.smem, st, mx, mxl, mw, mwl, mb, mbl, a);
    } else {
        HSES_CUDA(cudaFuncSetAttribute(linear_pack_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem));
        chain_launch(linear_pack_kernel<false>, grid, PK_THREADS, p.smem, st, mx, mxl, mw, mwl, mb, mbl, a);
    }
    HSES_LAUNCH_CHECK();
    return HSES_OK;
}

}  // namespace hses
