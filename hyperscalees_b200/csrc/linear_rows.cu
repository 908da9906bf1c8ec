// Tensor-core path of the perturbed linear layer (EggRoll::do_mm, hyperscalees-noiser/src/eggroll.rs:419-446) for layers
// whose members own many rows and whose weights fit shared memory: the token-level models' projections (k <= 256,
// a <= 256, rank <= 16, several parameters stacked along the outputs).
//
//   launch 1  rows_weights    W as three bf16 parts (24 bits) in the layout the tensor core reads
//   launch 2  rows_factors    the same of every pair's B and s·A, from a cache or the stream
//   launch 3  linear_rows     a persistent CTA walks over 128-row tiles, W resident:
//       warps 2-9    x from memory, once, into bf16 parts in shared memory (registers hold the next block meanwhile)
//       warp 0       MMAs: y = x·Wᵀ and t = x·B; the rank term u = t·(sA)ᵀ
//       warps 10-13  t to operand layout
//       warps 14-21  y + u to memory, with what follows the layer if asked (see RowsPost)
//       warp 1       W once, a pair's factors when the tiles reach it
// x is read once and the result written once: 64 -> 64 of 2.1 M rows moves 1.07 GB (165 us at the copy rate); the path
// over lowrank_t and linear_tc split x into fp16 operands in a pass of its own and took 755.  Parts need no row scales,
// so the split needs no look at the whole row.  No multicast, no cluster launch, bounded waits only.
#include <algorithm>

#include "linear.cuh"
#include "pack.cuh"

namespace hses {

namespace {

using namespace tc;
using namespace pack;

constexpr int LR_THREADS = 704;
constexpr int LR_TILE = 128;
constexpr int LR_PART = LR_TILE * 128;       // bytes of one part of 128 rows x 64 values
constexpr int LR_MAXK = 256, LR_MAXA = 256, LR_MAXR = 16, LR_MAXG = 4;
constexpr int LR_SMEM = 232448;

struct RowsFactors {
    const float *cache_a, *cache_b;          // raw (pairs, a, r) and (pairs, G, k, r), or NULL: from the stream (G = 1)
    const uint64_t *jump, *lane4, *lane16;
    NoiseCal cal;
    uint64_t key;
    int32_t true_epoch, first_pair;
    int r, rg, k, kb, a, groups, order;      // rg: a group's share of t's columns; kb: 64-wide blocks of k; order 1: A's rows
                                             // come first in the stream
    float base_sigma;
    uint8_t *bimg, *aimg;                    // per pair: (kb, part, groups * rg rows, 128 B); (slab, part, 2, outputs of a slab, 8)
    size_t b_bytes, a_bytes;
};

// W (a, k) -> (kb, part, a rows, 128 bytes), 16-byte pieces swizzled
__global__ void __launch_bounds__(256) rows_weights_kernel(const float* __restrict__ w, int64_t stride, int a, int k, int kb,
                                                           uint8_t* __restrict__ img) {
    chain_begin();
    const int e = blockIdx.x * 256 + threadIdx.x, c = e & 7, blk = (e >> 3) % kb, n = (e >> 3) / kb;
    if (n >= a) return;
    uint32_t v[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int kk = blk * 64 + c * 8 + 2 * j;
        const Parts s = split2(kk < k ? __ldg(w + (size_t)n * stride + kk) : 0.0f,
                               kk + 1 < k ? __ldg(w + (size_t)n * stride + kk + 1) : 0.0f);
#pragma unroll
        for (int part = 0; part < 3; ++part) v[part][j] = s.p[part];
    }
#pragma unroll
    for (int part = 0; part < 3; ++part)
        *reinterpret_cast<uint4*>(img + ((size_t)(blk * 3 + part) * a + n) * 128 + ((c ^ (n & 7)) << 4)) =
            make_uint4(v[part][0], v[part][1], v[part][2], v[part][3]);
}

// one block per (pair, group): its normals into shared memory, then both images
__global__ void __launch_bounds__(256) rows_factors_kernel(const __grid_constant__ RowsFactors f) {
    extern __shared__ __align__(16) float buf[];
    __shared__ CalTab tab;
    __shared__ uint64_t state_s[64];
    chain_next();
    const int tid = threadIdx.x, G = f.groups, ag = f.a / G, r = f.r;
    const int64_t p = blockIdx.x / G;
    const int gi = blockIdx.x % G, nb = f.k * r, na = ag * r;
    const float *B = buf, *A = buf + nb;
    if (f.cache_b) {
        chain_wait();
        for (int i = tid; i < nb; i += 256) buf[i] = __ldg(f.cache_b + ((size_t)p * G + gi) * nb + i);
        for (int i = tid; i < na; i += 256) buf[nb + i] = __ldg(f.cache_a + ((size_t)p * G + gi) * na + i);
    } else {
        NoiseCal cal = f.cal;
        stage_cal(cal, tab);
        stream_fill(cal, f.jump, f.lane4, f.lane16, noise_seed(f.key, f.true_epoch, f.first_pair + (int32_t)p) | 1ull, 0,
                    nb + na, state_s, [&](int off, float (&z)[4]) {
                        *reinterpret_cast<float4*>(buf + off) = make_float4(z[0], z[1], z[2], z[3]);
                    });
        if (f.order) A = buf, B = buf + na;
        chain_wait();
    }
    __syncthreads();
    for (int e = tid; e < f.kb * f.rg * 8; e += 256) {        // eight k of one rank value
        const int q = (e >> 3) % f.rg, blk = (e >> 3) / f.rg, c = e & 7, row = gi * f.rg + q;
        uint32_t v[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int kk = blk * 64 + c * 8 + 2 * j;
            const Parts s = split2(q < r && kk < f.k ? B[kk * r + q] : 0.0f, q < r && kk + 1 < f.k ? B[(kk + 1) * r + q] : 0.0f);
#pragma unroll
            for (int part = 0; part < 3; ++part) v[part][j] = s.p[part];
        }
#pragma unroll
        for (int part = 0; part < 3; ++part)
            *reinterpret_cast<uint4*>(f.bimg + p * f.b_bytes + ((size_t)(blk * 3 + part) * G * f.rg + row) * 128 +
                                      ((c ^ (row & 7)) << 4)) = make_uint4(v[part][0], v[part][1], v[part][2], v[part][3]);
    }
    // s·A: slabs of 16 of t's columns; with rank <= 8 two groups share a slab, each with zeros in the other's half
    const int gs = 16 / f.rg, slab = gi / gs, own = gi % gs, sn = gs * ag;
    for (int e = tid; e < ag * 2; e += 256) {                 // eight rank values of one output
        const int n = e % ag, g8 = e / ag, q0 = gs == 2 ? (g8 == own ? 0 : r) : g8 * 8;
        uint32_t v[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = q0 + 2 * j;
            const Parts s = split2(q < r ? __fmul_rn(A[n * r + q], f.base_sigma) : 0.0f,
                                   q + 1 < r ? __fmul_rn(A[n * r + q + 1], f.base_sigma) : 0.0f);
#pragma unroll
            for (int part = 0; part < 3; ++part) v[part][j] = s.p[part];
        }
#pragma unroll
        for (int part = 0; part < 3; ++part)
            *reinterpret_cast<uint4*>(f.aimg + p * f.a_bytes + (((size_t)(slab * 3 + part) * 2 + g8) * sn + own * ag + n) * 16) =
                make_uint4(v[part][0], v[part][1], v[part][2], v[part][3]);
    }
}

struct RowsArgs {
    const float* x;
    int64_t x_stride;
    int k, kb, a, slabs, nt;                 // nt: columns of t, 16 per slab
    int merged;                              // B lies behind W's rows: one product gives y and t
    int64_t n_pop, pairs;
    int t_steps, bm;
    int tps;                                 // tiles per pair and step
    int64_t tiles;
    const uint8_t *wimg, *bimg, *aimg;
    uint32_t w_bytes, b_bytes, a_bytes;
    int xbufs, fbufs, tbufs;                 // buffers of x's parts, of the factors, accumulators
    int chunk, chunks;                       // outputs at a time: all, or 128 (one block of k) in two accumulators
    float* out;
    int64_t out_stride;
    int wide_out;                            // 32-byte aligned rows
    float out_scale;
    const float* out_scale_ptr;
    RowsPost post;
    int* status;
};

// The tiles in order: those of a pair one after the other, step by step.  Counted, since a division per tile and role
// costs more than a tile's products.
struct Walk {
    int pair, step, sub;
    __device__ __forceinline__ Walk(const RowsArgs& g, int i) {
        const int tpp = g.tps * g.t_steps;
        pair = i / tpp;
        step = (i - pair * tpp) / g.tps;
        sub = i - pair * tpp - step * g.tps;
    }
    __device__ __forceinline__ bool next(const RowsArgs& g) {   // true: the next pair begins
        if (++sub < g.tps) return false;
        sub = 0;
        if (++step < g.t_steps) return false;
        step = 0;
        ++pair;
        return true;
    }
    __device__ __forceinline__ int first() const { return sub * LR_TILE; }   // row inside the pair's rows of the step
    __device__ __forceinline__ int rows(const RowsArgs& g) const { return min(LR_TILE, 2 * g.bm - first()); }
    __device__ __forceinline__ int64_t row0(const RowsArgs& g) const {
        return ((int64_t)step * g.n_pop + 2 * pair) * g.bm + first();
    }
};
// one of n buffers in turn, and the parity of its use
struct Turn {
    int b;
    uint32_t ph;
    __device__ __forceinline__ void next(int n) {
        if (++b == n) {
            b = 0;
            ph ^= 1;
        }
    }
};
// hses_lif_rate of 16 currents: the steps outside, so that 16 chains run side by side; the division by a power of two is a
// product with the same result
template <bool HARD>
__device__ __forceinline__ void lif_rates(float (&v)[2][8], const RowsPost& post) {
    float m[16], s[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) m[j] = s[j] = 0.0f;
    for (int t = 0; t < post.steps; ++t)
#pragma unroll
        for (int j = 0; j < 16; ++j)
            s[j] = __fadd_rn(s[j], lif_update(m[j], v[j >> 3][j & 7], post.leak, post.v_th, HARD ? HSES_RESET_HARD : HSES_RESET_SUBTRACT));
    const float n = (float)post.steps, inv = 1.0f / n;
    const bool pow2 = (post.steps & (post.steps - 1)) == 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j >> 3][j & 7] = pow2 ? __fmul_rn(s[j], inv) : __fdiv_rn(s[j], n);
}
__device__ __forceinline__ void store8f(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
                 "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

template <int POST>
__global__ void __launch_bounds__(LR_THREADS, 1) linear_rows_kernel(const __grid_constant__ RowsArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* wsm = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t w_tile = (uint32_t)(g.a + (g.merged ? g.nt : 0)) * 128;   // of one block of k and part
    uint8_t* xsm = wsm + g.kb * 3 * w_tile;                   // [buf][part 3][128 rows][128 B]
    uint8_t* bsm = xsm + (size_t)g.xbufs * 3 * LR_PART;       // [buf] B's image, unless merged
    uint8_t* asm_ = bsm + (g.merged ? 0 : (size_t)g.fbufs * g.b_bytes);      // [buf] A's image
    uint8_t* tsm = asm_ + (size_t)g.fbufs * g.a_bytes;        // t: [part 3][nt / 8][128][8] bf16
    const int t_part = g.nt * LR_TILE * 2;
    __shared__ uint64_t wfull, xfull[2], xempty[2], ffull[2], fempty[2], tfull[2], tempty[2], tacc, tready;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag_s;
    volatile int* abort_flag = &abort_flag_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_flag_s = 0;
        mbar_init(&wfull, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&xfull[b], 256);
            mbar_init(&xempty[b], 1);
            mbar_init(&ffull[b], 1);
            mbar_init(&fempty[b], 1);
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 256);
        }
        mbar_init(&tacc, 1);
        mbar_init(&tready, 128);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    chain_wait();                                             // before the allocation: a waiting block holds no tensor memory
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_next();
    const uint32_t tmem = tmem_slot;                          // y at buf * 128 (256 with one buffer), u (and t) 256 further
    const int64_t lo = g.tiles * blockIdx.x / gridDim.x, hi = g.tiles * (blockIdx.x + 1) / gridDim.x;
    const int count = (int)(hi - lo);                         // this CTA's tiles
    const Walk start(g, (int)lo);

    if (warp == 1) {
        if (lane == 0) {
            mbar_expect_tx(&wfull, g.w_bytes);
            for (int i = 0; i < g.kb * 3; ++i)
                bulk_load(wsm + (size_t)i * w_tile, g.wimg + (size_t)i * g.a * 128, (uint32_t)g.a * 128, &wfull);
            Walk w = start;
            Turn f{0, 0};
            bool ok = true, fresh = true;
            for (int i = 0; i < count && ok; ++i) {
                if (fresh) {
                    ok = mbar_wait(&fempty[f.b], f.ph ^ 1, abort_flag, g.status, 1);
                    if (!ok) break;
                    mbar_expect_tx(&ffull[f.b], g.b_bytes + g.a_bytes);
                    const uint8_t* src = g.bimg + (size_t)w.pair * g.b_bytes;
                    if (g.merged)
                        for (int j = 0; j < g.kb * 3; ++j)
                            bulk_load(wsm + (size_t)j * w_tile + g.a * 128, src + (size_t)j * g.nt * 128, (uint32_t)g.nt * 128, &ffull[f.b]);
                    else
                        bulk_load(bsm + (size_t)f.b * g.b_bytes, src, g.b_bytes, &ffull[f.b]);
                    bulk_load(asm_ + (size_t)f.b * g.a_bytes, g.aimg + (size_t)w.pair * g.a_bytes, g.a_bytes, &ffull[f.b]);
                    f.next(g.fbufs);
                }
                fresh = w.next(g);
            }
            if (!ok)   // copies already issued still land in this CTA's shared memory: give them a bounded moment
                for (uint32_t i = 0; i < 4096; ++i) {
                    if (mbar_try(&wfull, 0) && (mbar_try(&ffull[0], 0) || mbar_try(&ffull[0], 1)) &&
                        (g.fbufs == 1 || mbar_try(&ffull[1], 0) || mbar_try(&ffull[1], 1)))
                        break;
                    __nanosleep(256);
                }
        }
    } else if (warp == 0) {
        const int sn = g.a / g.slabs;                         // outputs of a slab
        const uint32_t idesc_t = make_idesc_bf16(g.nt), idesc_u = make_idesc_bf16(sn);
        const uint64_t dx0 = make_smem_desc(xsm), dw0 = make_smem_desc(wsm), db0 = make_smem_desc(bsm);
        const uint64_t dt0 = make_plain_desc(tsm, LR_TILE * 16), da0 = make_plain_desc(asm_, sn * 16);
        const uint32_t w_part = w_tile >> 4, b_part = (uint32_t)g.nt * 128 >> 4, x_part = LR_PART >> 4;
        const uint32_t a_part = (uint32_t)(16 * sn * 2) >> 4, a_slab = 3 * a_part;
        bool ok = __all_sync(0xffffffffu, mbar_wait(&wfull, 0, abort_flag, g.status, 2));
        Walk w = start;
        Turn x{0, 0}, f{0, 0}, acc{0, 0};
        bool fresh = true;
        const int row_units = 128 * 128 >> 4;                 // a chunk's rows of W, in units of a descriptor's address
        const uint32_t t1 = (uint32_t)t_part >> 4;
        // the rank term of outputs n0 .. n1-1 and the accumulator's hand-over
        auto rank_term = [&](int b, int fb, int n0, int n1) {
            const uint32_t u0 = tmem + 256 + (uint32_t)(b * 128);
            const uint64_t da = da0 + (uint64_t)(fb * (g.a_bytes >> 4));
            for (int sl = n0 / sn; sl * sn < n1; ++sl) {      // a slab's outputs in this chunk: all of them, or 128
                const uint64_t t = dt0 + (uint64_t)(sl * 2 * 128);
                const uint64_t a = da + (uint64_t)(sl * a_slab + max(0, n0 - sl * sn));
                const uint32_t u = u0 + (uint32_t)max(0, sl * sn - n0), id = sn > g.chunk ? make_idesc_bf16(n1 - n0) : idesc_u;
                umma_f16_warp(u, t + 2 * t1, a, id, 0);
                umma_f16_warp(u, t, a + 2 * a_part, id, 1);
                umma_f16_warp(u, t + t1, a + a_part, id, 1);
                umma_f16_warp(u, t + t1, a, id, 1);
                umma_f16_warp(u, t, a + a_part, id, 1);
                umma_f16_warp(u, t, a, id, 1);
            }
            umma_commit_warp(&tfull[b]);
        };
        for (int i = 0; i < count && ok; ++i) {
            if (fresh) {
                ok = __all_sync(0xffffffffu, mbar_wait(&ffull[f.b], f.ph, abort_flag, g.status, 3));
                if (!ok) break;
            }
            const int fb = __shfl_sync(0xffffffffu, f.b, 0);
            const uint64_t db = db0 + (uint64_t)(fb * (g.b_bytes >> 4));
            int b0 = 0;
            for (int ch = 0; ch < g.chunks && ok; ++ch, acc.next(g.tbufs)) {
                const int b = __shfl_sync(0xffffffffu, acc.b, 0), n = min(g.chunk, g.a - ch * g.chunk);
                ok = __all_sync(0xffffffffu, mbar_wait(&tempty[b], acc.ph ^ 1, abort_flag, g.status, 4));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(b * 128), du = d + 256;
                const uint32_t idesc = make_idesc_bf16(n + (g.merged ? g.nt : 0));
                const bool with_t = ch == 0 && !g.merged;
                for (int kb = 0; kb < g.kb; ++kb) {
                    const int xb = __shfl_sync(0xffffffffu, x.b, 0);
                    if (ch == 0) {
                        ok = __all_sync(0xffffffffu, mbar_wait(&xfull[xb], x.ph, abort_flag, g.status, 5));
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const uint64_t dx = dx0 + (uint64_t)(xb * 3 * x_part), dbk = db + (uint64_t)(kb * 3 * b_part),
                                   dw = dw0 + (uint64_t)(kb * 3 * w_part + ch * row_units);
                    const int ksteps = min(4, (g.k - kb * 64 + 15) / 16);
                    for (int ks = 0; ks < ksteps; ++ks) {     // 16 values = 32 bytes along k; smallest terms first
                        const uint64_t xd = dx + 2 * ks, wd = dw + 2 * ks, bb = dbk + 2 * ks;
                        const uint32_t more = (kb | ks) != 0;
                        if (with_t) {
                            umma_f16_warp(du, xd + 2 * x_part, bb, idesc_t, more);
                            umma_f16_warp(du, xd, bb + 2 * b_part, idesc_t, 1);
                            umma_f16_warp(du, xd + x_part, bb + b_part, idesc_t, 1);
                            umma_f16_warp(du, xd + x_part, bb, idesc_t, 1);
                            umma_f16_warp(du, xd, bb + b_part, idesc_t, 1);
                            umma_f16_warp(du, xd, bb, idesc_t, 1);
                        }
                        umma_f16_warp(d, xd + 2 * x_part, wd, idesc, more);
                        umma_f16_warp(d, xd, wd + 2 * w_part, idesc, 1);
                        umma_f16_warp(d, xd + x_part, wd + w_part, idesc, 1);
                        umma_f16_warp(d, xd + x_part, wd, idesc, 1);
                        umma_f16_warp(d, xd, wd + w_part, idesc, 1);
                        umma_f16_warp(d, xd, wd, idesc, 1);
                    }
                    if (ch + 1 == g.chunks) {
                        umma_commit_warp(&xempty[xb]);
                        x.next(g.xbufs);
                    }
                }
                if (!ok) break;
                if (ch == 0) {
                    umma_commit_warp(&tacc);
                    b0 = b;
                }
            }
            if (!ok) break;
            // t's way to shared memory and back, while the second chunk's products run
            ok = __all_sync(0xffffffffu, mbar_wait(&tready, i & 1, abort_flag, g.status, 6));
            if (!ok) break;
            tc_fence_after();
            rank_term(b0, fb, 0, g.chunk);
            if (g.chunks == 2) rank_term(b0 ^ 1, fb, g.chunk, g.a);
            fresh = w.next(g);
            if (fresh) {
                umma_commit_warp(&fempty[fb]);
                f.next(g.fbufs);
            }
            __syncwarp();
        }
    } else if (warp < 10) {
        // ---------------------------------------------------------------- x to parts
        const int tid = threadIdx.x - 64, c = tid & 7, r0 = tid >> 3;
        float4 v[4][2];                                       // four rows, eight values each, of the next block
        Walk w = start;                                       // tile and block of k that are loaded next
        int kb = 0;
        Turn x{0, 0};
        auto load = [&](float4 (&dst)[4][2]) {
            const int kk = kb * 64 + c * 8, cnt = w.rows(g);
            const int64_t row0 = w.row0(g);
            if (++kb == g.kb) {
                kb = 0;
                w.next(g);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = r0 + 32 * u;
                const bool in = r < cnt && kk < g.k;
                const float4* src = reinterpret_cast<const float4*>(g.x + (size_t)(row0 + (in ? r : 0)) * g.x_stride + (in ? kk : 0));
                dst[u][0] = in ? __ldcs(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                dst[u][1] = in ? __ldcs(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        auto put = [&](const float4 (&src)[4][2]) -> bool {
            const int xb = x.b;
            if (!mbar_wait(&xempty[xb], x.ph ^ 1, abort_flag, g.status, 7)) return false;
            x.next(g.xbufs);
            uint8_t* dst = xsm + (size_t)xb * 3 * LR_PART;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = r0 + 32 * u;
                const Parts a = split2(src[u][0].x, src[u][0].y), b = split2(src[u][0].z, src[u][0].w);
                const Parts e = split2(src[u][1].x, src[u][1].y), f = split2(src[u][1].z, src[u][1].w);
#pragma unroll
                for (int part = 0; part < 3; ++part)
                    *reinterpret_cast<uint4*>(dst + part * LR_PART + r * 128 + ((c ^ (r & 7)) << 4)) =
                        make_uint4(a.p[part], b.p[part], e.p[part], f.p[part]);
            }
            fence_proxy_async();
            mbar_arrive(&xfull[xb]);
            return true;
        };
        const int blocks = count * g.kb;
        if (blocks > 0) load(v);
        for (int blk = 0; blk < blocks; ++blk) {
            if (!put(v)) break;
            if (blk + 1 < blocks) load(v);
        }
    } else if (warp < 14) {
        // ---------------------------------------------------------------- t to operand layout
        const int q4 = warp & 3, gt = q4 * 32 + lane;         // TMEM quadrant, row of the tile
        const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16) + (g.merged ? g.a : 256);
        Walk w = start;
        Turn acc{0, 0};
        for (int i = 0; i < count; ++i, w.next(g)) {
            const int b = acc.b;                              // the accumulator of the tile's first chunk
            for (int ch = 0; ch < g.chunks; ++ch) acc.next(g.tbufs);
            const bool odd = w.first() + gt >= g.bm;          // the odd member of a pair has A negated
            if (!__all_sync(0xffffffffu, mbar_wait(&tacc, i & 1, abort_flag, g.status, 8))) break;
            tc_fence_after();
            for (int c8 = 0; c8 < g.nt / 8; ++c8) {
                uint32_t tv[8];
                tmem_ld8(lane_base + b * 128 + c8 * 8, tv);
                Parts s[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float v0 = __uint_as_float(tv[2 * j]), v1 = __uint_as_float(tv[2 * j + 1]);
                    s[j] = split2(odd ? -v0 : v0, odd ? -v1 : v1);
                }
#pragma unroll
                for (int part = 0; part < 3; ++part)
                    *reinterpret_cast<uint4*>(tsm + part * t_part + (c8 * LR_TILE + gt) * 16) =
                        make_uint4(s[0].p[part], s[1].p[part], s[2].p[part], s[3].p[part]);
            }
            fence_proxy_async();
            tc_fence_before();
            mbar_arrive(&tready);
        }
    } else {
        // ---------------------------------------------------------------- rows out
        const int q4 = warp & 3, eh = (warp - 14) >> 2;       // column blocks eh, eh + 2, ..
        const int gt = q4 * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(q4 * 32) << 16);
        const float gain = g.out_scale_ptr ? *g.out_scale_ptr : g.out_scale;
        Walk w = start;
        Turn acc{0, 0};
        for (int i = 0; i < count * g.chunks; ++i, acc.next(g.tbufs)) {
            const int b = acc.b, cnt = w.rows(g), ch = g.chunks == 2 ? i & 1 : 0, c_lo = ch * g.chunk, c_hi = min(c_lo + g.chunk, g.a);
            float* orow = g.out + (size_t)(w.row0(g) + gt) * g.out_stride;
            // the residual's values of a block of columns are asked for one block ahead
            float4 old[4];
            const bool add = POST == HSES_POST_ADD && gt < cnt;
            auto fetch = [&](int cb) {
                if (!add || cb >= c_hi) return;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float* o = orow + cb + 4 * j;
                    old[j] = g.wide_out ? *reinterpret_cast<const float4*>(o) : make_float4(o[0], o[1], o[2], o[3]);
                }
            };
            fetch(c_lo + eh * 16);
            if (ch + 1 == g.chunks) w.next(g);
            if (!__all_sync(0xffffffffu, mbar_wait(&tfull[b], acc.ph, abort_flag, g.status, 9))) break;
            tc_fence_after();
            for (int cb = c_lo + eh * 16; cb < c_hi; cb += 32) {
                uint32_t y[2][8], u[2][8];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    tmem_ld8_issue(lane_base + b * 128 + cb - c_lo + 8 * h, y[h]);
                    tmem_ld8_issue(lane_base + b * 128 + 256 + cb - c_lo + 8 * h, u[h]);
                }
                tmem_ld_wait();
                float v[2][8];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        v[h][j] = __fmul_rn(__fadd_rn(__uint_as_float(y[h][j]), __uint_as_float(u[h][j])), gain);
                if (POST == HSES_POST_SWISH) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j >> 3][j & 7] = swish_of(v[j >> 3][j & 7]);
                } else if (POST == HSES_POST_LIF_RATE) {
                    if (g.post.reset == HSES_RESET_HARD) lif_rates<true>(v, g.post);
                    else lif_rates<false>(v, g.post);
                }
                if (add) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float* p = &v[j >> 1][(j & 1) * 4];
                        p[0] = __fadd_rn(old[j].x, p[0]), p[1] = __fadd_rn(old[j].y, p[1]);
                        p[2] = __fadd_rn(old[j].z, p[2]), p[3] = __fadd_rn(old[j].w, p[3]);
                    }
                    fetch(cb + 32);
                }
                if (gt < cnt) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float* o = orow + cb + 8 * h;
                        if (g.wide_out) {
                            store8f(o, v[h]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; ++j) o[j] = v[h][j];
                        }
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(&tempty[b]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

struct RowsPlan {
    bool ok;
    int kb, rg, nt, merged, xbufs, fbufs, tbufs, chunk, smem;
    int64_t pairs;
    uint32_t w_bytes, b_bytes, a_bytes;
    size_t o_b, o_a, bytes;
};

RowsPlan plan_rows(const hses_linear_args& g) {
    RowsPlan p{};
    const int G = g.n_groups > 1 ? g.n_groups : 1;
    if (!g.perturb || g.lif != 0 || g.precision != HSES_PRECISION_FP32 || g.x_op != HSES_X_NONE || g.x_half != nullptr) return p;
    if (g.k % 8 != 0 || g.k > LR_MAXK || g.a > LR_MAXA || g.rank > LR_MAXR || G > LR_MAXG || g.a % G != 0 || g.a / G % 16 != 0) return p;
    if (g.first_thread % 2 != 0 || g.n_pop % 2 != 0 || (G > 1 && (g.cache == nullptr || g.factor_order != 0))) return p;
    if (((uintptr_t)g.x & 15u) != 0 || g.x_row_stride % 4 != 0) return p;
    // A tile never leaves a pair: from one full tile per pair and step on, and with tiles for every SM.  Below that the
    // packed or narrow paths fill a tile with several pairs.
    if (g.bm < LR_TILE / 2 || (int64_t)g.bm > (1 << 29)) return p;
    const int64_t tiles = g.n_pop / 2 * g.t_steps * ((2 * (int64_t)g.bm + LR_TILE - 1) / LR_TILE);
    if (tiles < plan_sm_count()) return p;
    p.pairs = g.n_pop / 2;
    p.kb = (g.k + 63) / 64;
    p.rg = G % 2 == 0 && g.rank <= 8 ? 8 : 16;
    const int nt = p.nt = G * p.rg;
    // With a few tiles per pair B may wait for the pair before: it lies behind W and one product makes y and t (a product of
    // 16 columns costs the tensor core about what one of 64 does)
    p.merged = g.a + nt <= (p.kb == 1 ? 128 : 256) && tiles / p.pairs >= 4;
    // more than 128 outputs: two accumulators of 128 in turn while x's only block of k is there, else one of 256
    const int sn = g.a / (nt / 16);
    p.chunk = g.a > 128 && p.kb == 1 && (sn == g.a || 128 % sn == 0) ? 128 : g.a;
    p.tbufs = p.chunk + (p.merged ? nt : 0) <= 128 ? 2 : 1;
    p.w_bytes = (uint32_t)p.kb * 3 * g.a * 128;
    p.b_bytes = (uint32_t)p.kb * 3 * nt * 128;
    p.a_bytes = (uint32_t)3 * 16 * g.a * 2;
    for (int bufs = 3;; --bufs) {                 // x's parts, then the factors in two buffers, where they fit
        if (bufs < 0) return p;
        p.xbufs = bufs & 2 ? 2 : 1;
        p.fbufs = bufs & 1 && !p.merged ? 2 : 1;
        p.smem = 1024 + (int)p.w_bytes + 3 * nt * 256 + p.xbufs * 3 * LR_PART + p.fbufs * (int)(p.b_bytes + p.a_bytes);
        if (p.smem <= LR_SMEM - 1024) break;
    }
    size_t o = (p.w_bytes + 255) / 256 * 256;
    p.o_b = o;
    o += ((size_t)p.pairs * p.b_bytes + 255) / 256 * 256;
    p.o_a = o;
    o += (size_t)p.pairs * p.a_bytes;
    p.bytes = o + 256;
    p.ok = p.bytes <= (4ull << 30) && tiles < (1ll << 31);
    return p;
}

}  // namespace

bool rows_path_supports(const hses_linear_args& g) { return plan_rows(g).ok; }

size_t rows_path_workspace_bytes(const hses_linear_args& g) { return plan_rows(g).bytes; }

int run_rows_path(hses_ctx* ctx, cudaStream_t st, const hses_linear_args& g, const RowsPost& post) {
    const RowsPlan p = plan_rows(g);
    HSES_REQUIRE(p.ok, "shape not covered");
    HSES_REQUIRE(g.workspace != nullptr && g.workspace_bytes >= p.bytes, "workspace too small; see hses_perturbed_linear_workspace_bytes");
    uint8_t* ws = reinterpret_cast<uint8_t*>(((uintptr_t)g.workspace + 255) & ~(uintptr_t)255);
    const int G = g.n_groups > 1 ? g.n_groups : 1;
    RowsFactors f{};
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
    f.first_pair = g.first_thread / 2;
    f.r = g.rank;
    f.rg = p.rg;
    f.k = g.k;
    f.kb = p.kb;
    f.a = g.a;
    f.groups = G;
    f.order = g.factor_order;
    f.base_sigma = g.sigma / sqrtf((float)g.rank);
    f.bimg = ws + p.o_b;
    f.aimg = ws + p.o_a;
    f.b_bytes = p.b_bytes;
    f.a_bytes = p.a_bytes;
    {
        HSES_KERNEL(ctx, st, "rows_weights");
        chain_launch(rows_weights_kernel, (unsigned)((g.a * p.kb * 8 + 255) / 256), 256, 0, st, g.param, g.param_row_stride, g.a,
                     g.k, p.kb, ws);
        HSES_LAUNCH_CHECK();
    }
    {
        const int smem = ((g.k + g.a / G) * g.rank + 4) * 4;
        HSES_REQUIRE(p.pairs * G < (1ll << 31), "too many pairs");
        HSES_CUDA(cudaFuncSetAttribute(rows_factors_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        HSES_KERNEL(ctx, st, "rows_factors");
        chain_launch(rows_factors_kernel, (unsigned)(p.pairs * G), 256, smem, st, f);
        HSES_LAUNCH_CHECK();
    }
    RowsArgs a{};
    a.x = g.x;
    a.x_stride = g.x_row_stride;
    a.k = g.k;
    a.kb = p.kb;
    a.a = g.a;
    a.nt = p.nt;
    a.slabs = p.nt / 16;
    a.merged = p.merged;
    a.n_pop = g.n_pop;
    a.pairs = p.pairs;
    a.t_steps = g.t_steps;
    a.bm = g.bm;
    a.tps = (2 * g.bm + LR_TILE - 1) / LR_TILE;
    a.tiles = p.pairs * g.t_steps * a.tps;
    a.wimg = ws;
    a.bimg = f.bimg;
    a.aimg = f.aimg;
    a.w_bytes = p.w_bytes;
    a.b_bytes = p.b_bytes;
    a.a_bytes = p.a_bytes;
    a.xbufs = p.xbufs;
    a.fbufs = p.fbufs;
    a.tbufs = p.tbufs;
    a.chunk = p.chunk;
    a.chunks = (g.a + p.chunk - 1) / p.chunk;
    a.out = g.out;
    a.out_stride = g.out_row_stride;
    a.wide_out = ((uintptr_t)g.out & 31u) == 0 && g.out_row_stride % 8 == 0;
    a.out_scale = g.out_scale;
    a.out_scale_ptr = g.out_scale_ptr;
    a.post = post;
    a.status = ctx->t.status_word;
    auto kernel = post.kind == HSES_POST_SWISH ? linear_rows_kernel<HSES_POST_SWISH>
                  : post.kind == HSES_POST_ADD ? linear_rows_kernel<HSES_POST_ADD>
                  : post.kind == HSES_POST_LIF_RATE ? linear_rows_kernel<HSES_POST_LIF_RATE> : linear_rows_kernel<0>;
    HSES_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, p.smem));
    HSES_KERNEL(ctx, st, "linear_rows");
    chain_launch(kernel, (unsigned)std::min<int64_t>(a.tiles, ctx->sm_count), LR_THREADS, p.smem, st, a);
    HSES_LAUNCH_CHECK();
    return HSES_OK;
}

}  // namespace hses
