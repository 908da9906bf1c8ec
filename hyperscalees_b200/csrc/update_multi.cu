// The fitness-weighted update of several matrices at once
//   sum_p (f_2p - f_2p+1) * A_p B_pᵀ          (simple_lora_update, eggroll.rs:353-373, pair-folded)
// on the tensor cores for any rank: the contraction (a, K)·(K, b) over K = pairs * rank of every matrix of
// a model, all sharing one fitness vector, in four launches.
//
//   launch 1  pair_weight_range    one power-of-two scale for all pair weights
//   launch 2  update_operands      a CTA makes one operand tile (up to 128 rows of A or B, 64 values of K:
//                                  64 / rank pairs side by side) of one matrix: the normals, regenerated from
//                                  the stream or read from a factor cache, in shared memory, then weighted,
//                                  split into fp16 hi + lo and written as the 128B-swizzled image the tensor
//                                  core reads
//   launch 3  update_gemm_tc       one CTA per (matrix, output tile, K split): images by plain bulk copies,
//                                  tcgen05 hi*hi + hi*lo + lo*hi, partial sums
//   launch 4  update_reduce        adds the splits in a fixed order, undoes the scales
// One set of launches instead of four per matrix matters as much as the tensor cores: a transformer's
// matrices are 16 x 64 to 64 x 256.  Wide ranks with cached factors stay on update_tc.cu, which reads the
// fp32 factors once and writes nothing back.  No multicast, no cluster launch, bounded waits.
#include <cuda_fp16.h>

#include <algorithm>

#include "tc_common.cuh"
#include "update_tc.cuh"

namespace hses {

namespace {

using namespace tc;

constexpr int UM_ROWS = 128;                 // rows of an operand tile, at most
constexpr int UM_EXP_A = 12, UM_EXP_B = 11;  // A' = (w * 2^-e_w) * A * 2^12 <= 23.7e3, B' = B * 2^11 <= 11.9e3
constexpr int UM_STAGES = 3;
constexpr int UM_STAGE_BYTES = 4 * UM_ROWS * 128;   // hi and lo tiles of both operands
constexpr size_t kImageChunkBytes = 512ull << 20;   // operand images of one chunk of pairs
constexpr int UM_BUF = 8704;                        // floats of a tile's normals in shared memory, padded

struct UmMat {
    uint64_t key;
    const float *cache_a, *cache_b;   // of the call's first pair, or NULL
    float* grad;
    size_t img_a, img_b;              // byte offsets of the operand images
    size_t part;                      // float offset of the partial sums
    int a, b, bn;                     // bn: columns per output tile
    int mt, nt;                       // row and column tiles
    int kb_a, kb_b;                   // k-blocks a CTA of update_operands makes of an A and of a B tile
    int gen0, gen0_b, gemm0, red0;    // first block of this matrix in each launch (gen0_b: of its B tiles)
};
struct UmArgs {
    int n;
    const uint64_t *jump, *lane4, *lane16;
    NoiseCal cal;
    int32_t true_epoch, first_pair;   // first_pair: of this chunk
    int64_t pair_off;                 // pairs of the call before this chunk
    int64_t pairs;                    // pairs of this chunk
    int r, pb;                        // rank, pairs per k-block (rank <= 64)
    int rkb;                          // k-blocks per pair (rank > 64), else 1
    int64_t kblks;
    const float* fitness;             // of the chunk's first member on
    const int* e_w;
    int sign_factors, splits, accumulate, add_to_grad;
    float scale;
    uint8_t* images;
    float* partial;
    int* status;
    UmMat m[kUpdateMulti];
};
__device__ __forceinline__ int rows8(int n) { return (n + 7) & ~7; }
__device__ __forceinline__ int sign_of(float v) { return v > 0.0f ? 1 : v < 0.0f ? -1 : 0; }

__global__ void um_weight_range_kernel(const float* __restrict__ fitness, int64_t pairs, int* __restrict__ e_out) {
    chain_begin();
    __shared__ float red[32];
    float m = 0.0f;
    for (int64_t p = threadIdx.x; p < pairs; p += blockDim.x) {
        m = fmaxf(m, fabsf(__fsub_rn(fitness[2 * p], fitness[2 * p + 1])));
    }
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = fmaxf(m, red[i]);
        int e = 0;
        if (m > 0.0f && m < INFINITY) {
            frexpf(m, &e);  // m = f * 2^e, f in [0.5, 1)
            e = max(-100, min(100, e));
        }
        *e_out = e;
    }
}

// The tiles of one row block in a few consecutive k-blocks.  Their normals are runs of consecutive stream values
// ("segments": the rows of the tile for one pair, or, with rank > 64, 64 values of one row).  The start states of all
// segments come from the power-of-two tables, one per thread side by side; from there a lane table gives the start of
// every piece of a segment.  Narrow matrices take several k-blocks at a time, up to 8704 values: one k-block of 16 rows at
// a time left most threads with a piece of four values and the lane table's 16 reads for it (430 us for 62 M normals of
// 33 matrices, two thirds of it the generator).  Bound by the generator's instruction issue.
constexpr int UM_STATES = 256;
constexpr int UM_GROUP = 16;                         // k-blocks at a time, at most
__host__ __device__ inline int um_pitch(int L) { return ((L + 3) & ~3) + 4; }
// values per start state: pieces of 16 or, where that leaves threads without one, of 4; start states per segment
__host__ __device__ inline int um_run(int L, int values) { return L >= 512 || (L >= 64 && values >= 4096) ? 512 : 128; }
__host__ __device__ inline int um_starts(int L, int run) { return (L + run - 1) / run; }

__global__ void __launch_bounds__(256, 4) update_operands_kernel(const __grid_constant__ UmArgs g) {
    __shared__ __align__(16) float buf[UM_BUF];
    __shared__ CalTab tab_s;
    __shared__ uint64_t seg_state[UM_STATES];
    __shared__ float mul_s[64 * UM_GROUP];
    const int tid = threadIdx.x;
    int i = 0;
    while (i + 1 < g.n && (int)blockIdx.x >= g.m[i + 1].gen0) ++i;
    const UmMat& m = g.m[i];
    const bool is_a = (int)blockIdx.x < m.gen0_b;
    const int rel = (int)blockIdx.x - (is_a ? m.gen0 : m.gen0_b), tiles = is_a ? m.mt : m.nt, kbn = is_a ? m.kb_a : m.kb_b;
    const int s = rel % tiles;
    const int64_t kb_lo = (int64_t)(rel / tiles) * kbn, kb_hi = min(kb_lo + kbn, g.kblks);
    const int dim = is_a ? m.a : m.b, step = is_a ? UM_ROWS : m.bn;
    const int row0 = s * step, nrows = min(step, dim - row0);
    const int r = g.r;
    const bool wide = r > 64;
    const int seg_len = wide ? 64 : nrows * r, segs = wide ? nrows : g.pb, LP = um_pitch(seg_len);
    const int group = wide ? 1 : max(1, min(min(UM_GROUP, kbn), UM_BUF / (segs * LP)));   // k-blocks made at a time
    const int run = um_run(seg_len, group * segs * seg_len), chn = run / 32, cps = um_starts(seg_len, run);
    const int ns = segs * cps;                  // start states of a k-block
    const float* cache = is_a ? m.cache_a : m.cache_b;
    chain_next();
    if (cache) chain_wait();
    NoiseCal cal = g.cal;
    if (!cache) {
        stage_cal(cal, tab_s);
        for (int e = tid; e < ns * (int)(kb_hi - kb_lo); e += 256) {
            const int kr = e / ns, f = e - kr * ns, sg = f / cps, c = f - sg * cps;
            const int64_t kb = kb_lo + kr;
            const int64_t pair = wide ? kb / g.rkb : kb * g.pb + sg;
            if (pair >= g.pairs) continue;
            const uint64_t pos = (uint64_t)r * (uint64_t)((is_a ? m.b : 0) + row0 + (wide ? sg : 0)) +
                                 (wide ? (uint64_t)(kb % g.rkb) * 64u : 0u) + (uint64_t)c * run;
            const uint64_t s0 = noise_seed(m.key, g.true_epoch, g.first_pair + (int32_t)pair) | 1ull;
            seg_state[e] = jump_by(g.jump, s0, 2ull * pos);
        }
    }
    // eight consecutive K values of a row per thread; eight lanes fill a 128-byte row of the image
    const int nr8 = is_a ? rows8(nrows) : min(m.bn, (nrows + 15) & ~15);
    const int dim_pad = is_a ? rows8(m.a) : m.nt * m.bn;         // rows of the operand in a k-block's images
    const int lo_ofs = (is_a ? nr8 : m.bn) * 128;
    const int c8 = tid & 7, pp0 = wide ? 0 : c8 * 8 / r, q_first = c8 * 8 - pp0 * r;
    for (int64_t kb = kb_lo; kb < kb_hi; kb += group) {
        const int gk = (int)min((int64_t)group, kb_hi - kb);
        const int64_t pair0 = wide ? kb / g.rkb : kb * g.pb;     // first pair of the tiles (inside the chunk)
        const int q0 = wide ? (int)(kb - pair0 * g.rkb) * 64 : 0;
        const int npairs = wide ? 1 : (int)min((int64_t)gk * g.pb, g.pairs - pair0);
        const int nq = wide ? min(64, r - q0) : r;               // rank values of the tile
        const int nseg = wide ? nrows : npairs;
        const int L = wide ? nq : nrows * r;                     // values per segment
        __syncthreads();   // the states are there; the previous tiles' values are no longer read
        if (cache) {
            for (int sg = 0; sg < nseg; ++sg) {
                const float* src = wide ? cache + ((size_t)(g.pair_off + pair0) * dim + row0 + sg) * r + q0
                                        : cache + ((size_t)(g.pair_off + pair0 + sg) * dim + row0) * r;
                if ((r & 3) == 0) {
                    for (int e = tid; e < L / 4; e += 256)
                        *reinterpret_cast<float4*>(buf + sg * LP + 4 * e) = __ldg(reinterpret_cast<const float4*>(src) + e);
                } else {
                    for (int e = tid; e < L; e += 256) buf[sg * LP + e] = __ldg(src + e);
                }
            }
        } else {
            const uint64_t* states = seg_state + (int)(kb - kb_lo) * ns;
            const int ppp = min(32, (min(L, run) + chn - 1) / chn);   // pieces per start state
            const uint64_t* tab = chn == 16 ? g.lane16 : g.lane4;
            for (int u = tid; u < nseg * cps * ppp; u += 256) {
                const int e = ppp == 32 ? u >> 5 : u / ppp, piece = u - e * ppp;
                const int sg = cps == 1 ? e : e / cps, c = e - sg * cps;
                const int off = c * run + piece * chn;
                if (off >= L) continue;
                uint64_t st = lane_jump(tab, states[e], piece);
                float* dst = buf + sg * LP + off;
#pragma unroll 1
                for (int j = 0; j < chn && off + j < L; j += 4) {
                    float z[4];
                    normals4(st, cal, z);
                    *reinterpret_cast<float4*>(dst + j) = make_float4(z[0], z[1], z[2], z[3]);
                }
            }
        }
        chain_wait();      // the normals need nothing of the kernels before
        for (int i = tid; i < npairs; i += 256) {
            const float* f = g.fitness + 2 * (pair0 + i);
            const float sc_a = ldexpf(1.0f, UM_EXP_A - *g.e_w);   // a power of two
            mul_s[i] = is_a ? __fmul_rn(__fsub_rn(f[0], f[1]), sc_a) : (float)(1 << UM_EXP_B);
        }
        __syncthreads();
        uint8_t* img0 = g.images + (is_a ? m.img_a : m.img_b) + (size_t)kb * dim_pad * 256 + (size_t)row0 * 256;
        int row = tid >> 3, j = 0;                               // row and k-block of the group
        while (row >= nr8) row -= nr8, ++j;
        while (j < gk) {
            float v[8];
            if (!wide && (r & 7) == 0) {                         // eight values of one pair
                const int pp = j * g.pb + pp0;
                const bool live = row < nrows && pp < npairs && pp0 < g.pb;
                const float* src = buf + pp * LP + row * r + q_first;
                const float4 x = live ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 y = live ? *reinterpret_cast<const float4*>(src + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float w = live ? mul_s[pp] : 0.0f;
                v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w, v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(g.sign_factors ? (float)sign_of(v[k]) : v[k], w);
            } else {
                int pl = pp0, q = q_first;                       // pair of the k-block, rank value
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int pp = j * g.pb + pl;
                    float x = 0.0f;
                    if (row < nrows && pl < g.pb && pp < npairs && q < nq) {
                        x = wide ? buf[row * LP + q] : buf[pp * LP + row * r + q];
                        if (g.sign_factors) x = (float)sign_of(x);   // AltEggRoll contracts the sign patterns
                        x = __fmul_rn(x, mul_s[pp]);
                    }
                    v[k] = x;
                    if (++q == r && !wide) q = 0, ++pl;
                }
            }
            uint32_t h[4], l[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const __half2 hh = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
                const float2 b = __half22float2(hh);
                const __half2 ll = __floats2half2_rn(v[2 * k] - b.x, v[2 * k + 1] - b.y);
                h[k] = *reinterpret_cast<const uint32_t*>(&hh);
                l[k] = *reinterpret_cast<const uint32_t*>(&ll);
            }
            uint8_t* img = img0 + (size_t)j * dim_pad * 256 + (row >> 3) * 1024 + (row & 7) * 128 + ((c8 ^ (row & 7)) << 4);
            *reinterpret_cast<uint4*>(img) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(img + lo_ofs) = make_uint4(l[0], l[1], l[2], l[3]);
            row += 32;
            while (row >= nr8) row -= nr8, ++j;
        }
    }
}

// warp 0: copies, warp 1: MMAs, warps 2-5: sums.  The tensor core adds into its accumulator with truncation, an error
// that grows with the chain: after UM_CHAIN k-blocks (24 MMAs) the MMAs go on in the other of two accumulators and the
// warps add the finished one to fp32 sums in registers, one output row per thread.  One chain over 64 k-blocks left
// gradients 2e-4 of their spread away from the fp32 kernel's.
constexpr int UM_CHAIN = 2;
__global__ void __launch_bounds__(192, 1) update_gemm_tc_kernel(const __grid_constant__ UmArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[UM_STAGES], empty[UM_STAGES], tfull[2], tempty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag_s;
    volatile int* abort_flag = &abort_flag_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int i = 0;
    while (i + 1 < g.n && (int)blockIdx.x >= g.m[i + 1].gemm0) ++i;
    const UmMat& m = g.m[i];
    const int rel = (int)blockIdx.x - m.gemm0;
    const int split = rel % g.splits, tile = rel / g.splits;
    const int nt = tile % m.nt, mt = tile / m.nt;
    const int64_t k_lo = g.kblks * split / g.splits, k_hi = g.kblks * (split + 1) / g.splits;
    const uint32_t kn = (uint32_t)(k_hi - k_lo);
    const int arows = rows8(min(UM_ROWS, m.a - mt * UM_ROWS));
    const uint32_t a_bytes = (uint32_t)arows * 128, b_bytes = (uint32_t)m.bn * 128;
    if (threadIdx.x == 0) {
        abort_flag_s = 0;
        for (int s = 0; s < UM_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    chain_wait();          // before the allocation: a waiting block holds no tensor memory
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(256)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    chain_next();
    const uint32_t tmem = tmem_slot;
    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            const uint8_t* ia = g.images + m.img_a + (size_t)mt * UM_ROWS * 256;
            const uint8_t* ib = g.images + m.img_b + (size_t)nt * m.bn * 256;
            const size_t sa = (size_t)rows8(m.a) * 256, sb = (size_t)m.nt * m.bn * 256;
            for (uint32_t it = 0; it < kn; ++it) {
                const int s = it % UM_STAGES;
                if (!mbar_wait(&empty[s], ((it / UM_STAGES) & 1) ^ 1, abort_flag, g.status, 11)) { ok = false; break; }
                uint8_t* st = smem + (size_t)s * UM_STAGE_BYTES;
                mbar_expect_tx(&full[s], 2 * a_bytes + 2 * b_bytes);
                bulk_load(st, ia + (k_lo + it) * sa, 2 * a_bytes, &full[s]);              // hi, then lo
                bulk_load(st + 2 * UM_ROWS * 128, ib + (k_lo + it) * sb, 2 * b_bytes, &full[s]);
            }
            if (!ok)
                for (int s = 0; s < UM_STAGES; ++s)
                    for (uint32_t j = 0; j < 4096; ++j) {
                        if (mbar_try(&full[s], 0) || mbar_try(&full[s], 1)) break;
                        __nanosleep(256);
                    }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = make_idesc(m.bn);
            for (uint32_t it = 0; it < kn; ++it) {
                const uint32_t chain = it / UM_CHAIN, b = chain & 1;
                if (it % UM_CHAIN == 0) {
                    if (!mbar_wait(&tempty[b], ((chain >> 1) & 1) ^ 1, abort_flag, g.status, 14)) break;
                    tc_fence_after();
                }
                const int s = it % UM_STAGES;
                if (!mbar_wait(&full[s], (it / UM_STAGES) & 1, abort_flag, g.status, 12)) break;
                tc_fence_after();
                uint8_t* st = smem + (size_t)s * UM_STAGE_BYTES;
                const uint64_t dah = make_smem_desc(st), dal = make_smem_desc(st + a_bytes);
                const uint64_t dbh = make_smem_desc(st + 2 * UM_ROWS * 128), dbl = make_smem_desc(st + 2 * UM_ROWS * 128 + b_bytes);
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    const uint64_t off = (uint64_t)(ks * 32 >> 4);
                    umma_f16(tmem + b * 128, dal + off, dbh + off, idesc, (it % UM_CHAIN | ks) != 0);
                    umma_f16(tmem + b * 128, dah + off, dbl + off, idesc, 1);
                    umma_f16(tmem + b * 128, dah + off, dbh + off, idesc, 1);
                }
                umma_commit(&empty[s]);
                if (it % UM_CHAIN == UM_CHAIN - 1 || it + 1 == kn) umma_commit(&tfull[b]);
            }
        }
    } else {
        const int q4 = warp & 3;
        float sum[UM_ROWS];
#pragma unroll
        for (int j = 0; j < UM_ROWS; ++j) sum[j] = 0.0f;
        for (uint32_t chain = 0; chain * UM_CHAIN < kn; ++chain) {
            const uint32_t b = chain & 1;
            bool have = mbar_wait(&tfull[b], (chain >> 1) & 1, abort_flag, g.status, 13);
            have = __all_sync(0xffffffffu, have);                  // the TMEM loads are warp-wide
            if (!have) break;
            tc_fence_after();
#pragma unroll
            for (int j0 = 0; j0 < UM_ROWS; j0 += 16) {
                if (j0 < m.bn) {
                    uint32_t acc[2][8];
                    tmem_ld8_issue(tmem + ((uint32_t)(q4 * 32) << 16) + b * 128 + j0, acc[0]);
                    tmem_ld8_issue(tmem + ((uint32_t)(q4 * 32) << 16) + b * 128 + j0 + 8, acc[1]);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[j0 + j] = __fadd_rn(sum[j0 + j], __uint_as_float(acc[j >> 3][j & 7]));
                }
            }
            tc_fence_before();
            mbar_arrive(&tempty[b]);
        }
        const int row = mt * UM_ROWS + q4 * 32 + lane, n0 = nt * m.bn;
        if (row < m.a) {
            float* dst = g.partial + m.part + ((size_t)split * m.a + row) * m.b;
#pragma unroll
            for (int j = 0; j < UM_ROWS; ++j)
                if (j < m.bn && n0 + j < m.b) dst[n0 + j] = g.accumulate ? __fadd_rn(dst[n0 + j], sum[j]) : sum[j];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
    }
}

// Eight warps per 32 elements: warp w adds the splits w, w + 8, .. in index order, then the eight sums are added in
// warp order: a fixed order, the same bits on every rank.
__global__ void __launch_bounds__(256) update_multi_reduce_kernel(const __grid_constant__ UmArgs g) {
    chain_begin();
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int i = 0;
    while (i + 1 < g.n && (int)blockIdx.x >= g.m[i + 1].red0) ++i;
    const UmMat& m = g.m[i];
    const size_t len = (size_t)m.a * m.b, e = (size_t)(blockIdx.x - m.red0) * 32 + lane;
    const float* p = g.partial + m.part;
    float s = 0.0f;
    if (e < len)
        for (int k = warp; k < g.splits; k += 8) s = __fadd_rn(s, p[(size_t)k * len + e]);
    part[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || e >= len) return;
    const int nw = min(8, g.splits);
    for (int w = 1; w < nw; ++w) s = __fadd_rn(s, part[w][lane]);
    s = __fmul_rn(ldexpf(s, *g.e_w - UM_EXP_A - UM_EXP_B), g.scale);
    m.grad[e] = g.add_to_grad ? __fadd_rn(m.grad[e], s) : s;
}

struct UmPlan {
    int pb, rkb, splits;
    int64_t pairs, chunk_pairs;
    size_t image_bytes, partial_floats, bytes;
};
int64_t kblks_of(const UmPlan& p, int64_t pairs) { return p.rkb > 1 ? pairs * p.rkb : (pairs + p.pb - 1) / p.pb; }

// tiles and operand rows of one matrix
void shape_of(int a, int b, int& mt, int& nt, int& bn) {
    mt = (a + UM_ROWS - 1) / UM_ROWS;
    nt = (b + UM_ROWS - 1) / UM_ROWS;
    bn = ((b + nt - 1) / nt + 15) & ~15;
    nt = (b + bn - 1) / bn;
}

UmPlan plan_multi(const int* a, const int* b, int n, int rank, int64_t members) {
    UmPlan p{};
    p.pairs = members / 2;
    p.pb = rank <= 64 ? 64 / rank : 1;
    p.rkb = rank <= 64 ? 1 : (rank + 63) / 64;
    size_t rows = 0, len = 0;
    int64_t tiles = 0;
    for (int i = 0; i < n; ++i) {
        int mt, nt, bn;
        shape_of(a[i], b[i], mt, nt, bn);
        rows += (size_t)((a[i] + 7) & ~7) + (size_t)nt * bn;
        len += (size_t)a[i] * b[i];
        tiles += (int64_t)mt * nt;
    }
    // chunks of whole k-blocks
    int64_t fit = (int64_t)(kImageChunkBytes / (rows * 256));
    if (fit < 1) fit = 1;
    const int64_t all = kblks_of(p, p.pairs);
    if (p.rkb > 1) fit = std::max<int64_t>(fit / p.rkb, 1) * p.rkb;
    const int64_t kb = std::min(fit, all);
    p.chunk_pairs = p.rkb > 1 ? kb / p.rkb : std::min(p.pairs, kb * p.pb);
    // one wave of CTAs; a split that owns less than two k-blocks is all set-up
    int64_t s = plan_sm_count() / std::max<int64_t>(tiles, 1);
    s = std::min(s, (kb + 1) / 2);
    p.splits = (int)std::max<int64_t>(s, 1);
    p.image_bytes = (rows * 256 * (size_t)kb + 255) / 256 * 256;
    p.partial_floats = len * p.splits;
    p.bytes = 512 + p.image_bytes + (p.partial_floats * 4 + 255) / 256 * 256;
    return p;
}

}  // namespace

size_t update_multi_workspace_bytes(const int* a, const int* b, int n, int rank, int64_t members) {
    if (n < 1 || n > kUpdateMulti || members < 2) return 0;
    return plan_multi(a, b, n, rank, members).bytes;
}

int run_update_multi(hses_ctx* ctx, cudaStream_t st, const UpdateMultiItem* items, int n, const UpdateMultiCall& c) {
    HSES_REQUIRE(n >= 1 && n <= kUpdateMulti, "too many matrices for one set of launches");
    int a[kUpdateMulti], b[kUpdateMulti];
    for (int i = 0; i < n; ++i) a[i] = items[i].a, b[i] = items[i].b;
    const UmPlan p = plan_multi(a, b, n, c.rank, c.n);
    HSES_REQUIRE(c.workspace != nullptr && c.workspace_bytes >= p.bytes, "workspace too small; see the *_workspace_bytes call");
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)c.workspace + 255) & ~(uintptr_t)255);
    UmArgs g{};
    g.n = n;
    g.jump = ctx->t.jump_tabs;
    g.lane4 = ctx->t.jump_lane4;
    g.lane16 = ctx->t.jump_lane16;
    g.cal = ctx->cal();
    g.true_epoch = true_epoch_of(c.epoch, c.noise_reuse);
    g.r = c.rank;
    g.pb = p.pb;
    g.rkb = p.rkb;
    g.e_w = reinterpret_cast<int*>(base);
    g.sign_factors = c.sign_factors;
    g.splits = p.splits;
    g.scale = c.scale;
    g.images = base + 256;
    g.partial = reinterpret_cast<float*>(base + 256 + p.image_bytes);
    g.status = ctx->t.status_word;
    const int32_t first_pair = c.first_thread / 2;
    HSES_CUDA(cudaFuncSetAttribute(update_gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   UM_STAGES * UM_STAGE_BYTES + 1024));
    {
        HSES_KERNEL(ctx, st, "pair_weight_range");
        chain_launch(um_weight_range_kernel, 1, 1024, 0, st, c.fitness, p.pairs, const_cast<int*>(g.e_w));
        HSES_LAUNCH_CHECK();
    }
    for (int64_t done = 0; done < p.pairs; done += p.chunk_pairs) {
        g.pairs = std::min(p.chunk_pairs, p.pairs - done);
        g.pair_off = done;
        g.first_pair = first_pair + (int32_t)done;
        g.fitness = c.fitness + 2 * done;
        g.kblks = kblks_of(p, g.pairs);
        g.accumulate = done > 0;
        size_t img = 0, part = 0;
        int64_t gen = 0, gemm = 0, red = 0;
        for (int i = 0; i < n; ++i) {
            UmMat& m = g.m[i];
            m.key = items[i].key;
            m.cache_a = items[i].cache_a;
            m.cache_b = items[i].cache_b;
            m.grad = items[i].grad;
            m.a = a[i];
            m.b = b[i];
            shape_of(m.a, m.b, m.mt, m.nt, m.bn);
            m.img_a = img;
            img += (size_t)((m.a + 7) & ~7) * 256 * g.kblks;
            m.img_b = img;
            img += (size_t)m.nt * m.bn * 256 * g.kblks;
            m.part = part;
            part += (size_t)p.splits * m.a * m.b;
            // enough k-blocks per CTA that its set-up (tables, start states) is a small part of it, as long as the
            // launch still has blocks for every SM; the states of all of them have room in shared memory
            auto k_blocks_of = [&](int rows, int tiles) {
                const int L = c.rank > 64 ? 64 : rows * c.rank;
                const int ns = (c.rank > 64 ? rows : p.pb) * um_starts(L, L >= 512 ? 512 : 128);
                const int64_t want = std::max<int64_t>(1, 16384 / (64 * rows));
                const int64_t fill = std::max<int64_t>(1, g.kblks * tiles * n / (4 * (int64_t)ctx->sm_count));
                return (int)std::max<int64_t>(1, std::min({want, fill, (int64_t)(UM_STATES / ns)}));
            };
            m.kb_a = k_blocks_of(std::min(m.a, UM_ROWS), m.mt);
            m.kb_b = k_blocks_of(std::min(m.b, m.bn), m.nt);
            m.gen0 = (int)gen;
            m.gemm0 = (int)gemm;
            m.red0 = (int)red;
            gen += (g.kblks + m.kb_a - 1) / m.kb_a * m.mt;
            m.gen0_b = (int)gen;
            gen += (g.kblks + m.kb_b - 1) / m.kb_b * m.nt;
            gemm += (int64_t)m.mt * m.nt * p.splits;
            red += ((int64_t)m.a * m.b + 31) / 32;
        }
        HSES_REQUIRE(gen < (1ll << 31) && gemm < (1ll << 31) && red < (1ll << 31), "too many tiles");
        {
            HSES_KERNEL(ctx, st, "update_operands");
            chain_launch(update_operands_kernel, (unsigned)gen, 256, 0, st, g);
            HSES_LAUNCH_CHECK();
        }
        {
            HSES_KERNEL(ctx, st, "update_gemm_tc");
            chain_launch(update_gemm_tc_kernel, (unsigned)gemm, 192, UM_STAGES * UM_STAGE_BYTES + 1024, st, g);
            HSES_LAUNCH_CHECK();
        }
        if (done + p.chunk_pairs >= p.pairs) {
            g.add_to_grad = c.add_to_grad;
            HSES_KERNEL(ctx, st, "update_reduce");
            chain_launch(update_multi_reduce_kernel, (unsigned)red, 256, 0, st, g);
            HSES_LAUNCH_CHECK();
        }
    }
    return HSES_OK;
}

}  // namespace hses
