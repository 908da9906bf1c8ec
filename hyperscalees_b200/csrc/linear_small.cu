// Perturbed linear layers for narrow layers (k <= 64 inputs, a <= 64 outputs, rank <= 16): the
// per-head and per-token projections of the SNN-rate transformer
// (hyperscalees-models/src/snn_transformer.rs:273-297) at population scale, one launch for up to 16 of them that read
// the same x.
//
// Such a layer is a few kilobytes of weights and factors per antithetic pair, and 32 rows of x: too little for a tile of
// the wide kernels.  Here a warp owns a slice of 16 outputs of one layer: W's fragments stay in its registers while its
// CTA (four slices) walks over pairs; x (32 rows) and the factors of the next pair arrive by asynchronous copies (or the
// factors are made here from the stream) while this pair's products run.  t = x·B and y = x·Wᵀ + t·(sA)ᵀ are warp-level
// tensor-core products of values split into three bf16 parts (24 bits: the six largest of the nine part products, fp32
// sums), and t's accumulator is the operand of the rank term as it lies.
// fp32 multiply-adds from shared memory took 48 us for 64 -> 16 of 65536 rows and 166 us for twelve such heads at once,
// bound by the reads of shared memory and by waiting for the factors.
#include <algorithm>
#include <type_traits>

#include <cuda_bf16.h>

#include "common.cuh"
#include "linear.cuh"
#include "pack.cuh"

namespace hses {

namespace {

using pack::Parts;
using pack::split2;

constexpr int SP_ROWS = 32;          // rows staged at a time
constexpr int SP_MAXK = 64, SP_MAXA = 64, SP_MAXR = 16;
constexpr int SP_JOBS = 16;          // layers per launch
constexpr int SP_SLICES = 4;         // warps per CTA
constexpr int SP_THREADS = 32 * SP_SLICES;
constexpr int SP_XF = SP_MAXK + 4;   // pitch of x as it arrives, floats
constexpr int SP_XB = SP_MAXK + 8;   // pitch of x's bf16 parts: eight rows of 16 bytes lie in different banks
constexpr int SP_RUNS = SP_SLICES * (SP_MAXK * SP_MAXR / 128 + 2);

struct SmallJob {
    const float* w;
    int64_t w_stride;
    const float *A, *B;              // raw (pairs, a, rank), (pairs, k, rank) from the call's first pair on, or NULL
    uint64_t key;
    float* out;
    int64_t out_stride;
    float* pot;
    int a, slice0;                   // outputs, first slice
    int vec;                         // two neighbouring outputs are one aligned store
};
struct SmallArgs {
    const float* x;
    int64_t x_stride;
    int t_steps, bm, k, rank;
    int64_t n_pop;
    int32_t first_thread;
    int64_t pairs;
    float base_sigma;
    int lif;
    float leak, v_th, out_scale;
    const float* out_scale_ptr;
    NoiseCal cal;
    const uint64_t *jump, *lane4;
    int32_t true_epoch, first_pair;
    int vec_x, vec_f;                // x rows, factors: 16-byte copies
    int jobs, slices, groups;        // groups: CTAs that share a pair
    SmallJob job[SP_JOBS];
};

template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += the product of two values in parts, smallest terms first
__device__ __forceinline__ void mma_parts(float (&c)[4], const uint32_t (&a)[3][4], const Parts& b0, const Parts& b1) {
    mma_bf16(c, a[2], b0.p[0], b1.p[0]);
    mma_bf16(c, a[1], b0.p[1], b1.p[1]);
    mma_bf16(c, a[0], b0.p[2], b1.p[2]);
    mma_bf16(c, a[1], b0.p[0], b1.p[0]);
    mma_bf16(c, a[0], b0.p[1], b1.p[1]);
    mma_bf16(c, a[0], b0.p[0], b1.p[0]);
}
__device__ __forceinline__ void load_a(uint32_t (&a)[4], const __nv_bfloat16* tile) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(tile)));
}

// bytes of dynamic shared memory: two buffers of x and of the factors
__host__ __device__ inline int sp_factor_floats(int k, int rank) { return SP_SLICES * (k + 16) * rank; }
__host__ __device__ inline int sp_bytes(int k, int rank) { return 2 * (SP_ROWS * SP_XF + sp_factor_floats(k, rank)) * 4; }

// NQ: pieces of eight rank values; MEAN: out is the mean over the steps, one row per sample
template <int NQ, bool MEAN>
__global__ void __launch_bounds__(SP_THREADS, 3) small_pair_kernel(const __grid_constant__ SmallArgs g) {
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) __nv_bfloat16 xs[3][SP_ROWS][SP_XB];
    __shared__ CalTab tab;
    __shared__ uint64_t state_s[SP_RUNS];
    chain_begin();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gr = lane >> 2, tq = lane & 3;
    const int k = g.k, rank = g.rank, ksteps = (k + 15) >> 4;
    const int group = blockIdx.x % g.groups, cta = blockIdx.x / g.groups, ctas = gridDim.x / g.groups;
    const int ff = sp_factor_floats(k, rank);
    float* xbuf[2] = {sm, sm + SP_ROWS * SP_XF};
    float* fbuf[2] = {sm + 2 * SP_ROWS * SP_XF, sm + 2 * SP_ROWS * SP_XF + ff};
    auto job_at = [&](int s) {
        int j = 0;
        while (j + 1 < g.jobs && g.job[j + 1].slice0 <= s) ++j;
        return j;
    };
    // this warp's slice; a CTA's layers are consecutive: layer i of it has its B at i * k * rank, slice s its A behind them
    const int s_lo = group * SP_SLICES, s_hi = min(s_lo + SP_SLICES, g.slices), slice = s_lo + warp;
    const bool busy = slice < s_hi;
    const int j_lo = job_at(s_lo), j_hi = job_at(s_hi - 1) + 1, jn = busy ? job_at(slice) : j_lo;
    const SmallJob& jb = g.job[jn];
    const int c0 = busy ? (slice - jb.slice0) * 16 : 0;      // first output of the slice
    const int a_base = SP_SLICES * k * rank, kr = k * rank, ar = 16 * rank;
    // W's fragments: 16 outputs x k
    Parts wf[4][2][2];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int n = c0 + nt * 8 + gr, kk = ks * 16 + h * 8 + tq * 2;
                const float* row = jb.w + (size_t)min(n, jb.a - 1) * jb.w_stride;
                const bool in = busy && n < jb.a;
                wf[ks][nt][h] = split2(in && kk < k ? __ldg(row + kk) : 0.0f, in && kk + 1 < k ? __ldg(row + kk + 1) : 0.0f);
            }
    // the columns of x past k stay zero
    for (int i = tid; i < 2 * SP_ROWS * SP_XF; i += SP_THREADS) sm[i] = 0.0f;
    const float gain = g.out_scale_ptr ? *g.out_scale_ptr : g.out_scale;
    const bool regen = g.job[0].A == nullptr;
    NoiseCal cal = g.cal;
    if (regen) stage_cal(cal, tab);
    __syncthreads();
    const int rows_per_step = 2 * g.bm;                       // both members of a pair
    // rows of the pair, 32 at a time; for the mean, the steps of 32 samples one after the other
    const int span = MEAN ? rows_per_step : rows_per_step * g.t_steps, inner = MEAN ? g.t_steps : 1;
    const int iters = (span + SP_ROWS - 1) / SP_ROWS * inner;
    auto row_of = [&](int64_t p, int it, int r) -> int64_t {   // global row of row r of the tile, or -1
        const int t = MEAN ? it % inner : 0, lr = (MEAN ? it / inner : it) * SP_ROWS + r;
        if (lr >= span) return -1;
        const int step = MEAN ? t : lr / rows_per_step, rr = MEAN ? lr : lr - step * rows_per_step;
        return ((int64_t)step * g.n_pop + p * 2) * g.bm + rr;
    };
    auto fetch_x = [&](int64_t p, int it, float* dst) {
        // four threads per row
        const int r = tid >> 2;
        const int64_t row = row_of(p, it, r);
        if (row < 0) return;
        const float* src = g.x + (size_t)row * g.x_stride;
        if (g.vec_x)
            for (int kk = (tid & 3) * 4; kk < k; kk += 16) copy_async<16>(dst + r * SP_XF + kk, src + kk);
        else
            for (int kk = tid & 3; kk < k; kk += 4) copy_async<4>(dst + r * SP_XF + kk, src + kk);
    };
    auto fetch_factors = [&](int64_t p, float* dst) {
        for (int j = j_lo; j < j_hi; ++j) {
            const float* src = g.job[j].B + (size_t)p * kr;
            if (g.vec_f)
                for (int e = tid * 4; e < kr; e += SP_THREADS * 4) copy_async<16>(dst + (j - j_lo) * kr + e, src + e);
            else
                for (int e = tid; e < kr; e += SP_THREADS) copy_async<4>(dst + (j - j_lo) * kr + e, src + e);
        }
        if (busy) {
            const int cnt = min(16, jb.a - c0) * rank;
            const float* src = jb.A + ((size_t)p * jb.a + c0) * rank;
            float* d = dst + a_base + warp * ar;
            if (g.vec_f)
                for (int e = lane * 4; e < cnt; e += 128) copy_async<16>(d + e, src + e);
            else
                for (int e = lane; e < cnt; e += 32) copy_async<4>(d + e, src + e);
        }
    };
    // B of the CTA's layers and A of its slices from their streams, in runs of 128 values
    const int runs_b = (kr + 127) / 128, runs_a = (ar + 127) / 128;
    auto make_factors = [&](int64_t p, float* dst) {
        const int nb = (j_hi - j_lo) * runs_b, total = nb + (s_hi - s_lo) * runs_a;
        for (int e = tid; e < total; e += SP_THREADS) {
            const int s = e < nb ? 0 : (e - nb) / runs_a, j = e < nb ? j_lo + e / runs_b : job_at(s_lo + s);
            const int pos = e < nb ? e % runs_b * 128
                                   : kr + (s_lo + s - g.job[j].slice0) * ar + (e - nb) % runs_a * 128;
            state_s[e] = jump_by(g.jump, noise_seed(g.job[j].key, g.true_epoch, g.first_pair + (int32_t)p) | 1ull, 2ull * pos);
        }
        __syncthreads();
        for (int e = warp; e < total; e += SP_SLICES) {
            const int off = (e < nb ? e % runs_b : (e - nb) % runs_a) * 128 + lane * 4, cnt = e < nb ? kr : ar;
            if (off >= cnt) continue;
            float* d = e < nb ? dst + e / runs_b * kr : dst + a_base + (e - nb) / runs_a * ar;
            uint64_t st = lane_jump(g.lane4, state_s[e], lane);
            float z[4];
            normals4(st, cal, z);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (off + i < cnt) d[off + i] = z[i];
        }
    };
    uint32_t n_x = 0, n_f = 0;                                // buffers filled so far
    if (cta < g.pairs) {
        fetch_x(cta, 0, xbuf[0]);
        if (!regen) fetch_factors(cta, fbuf[0]);
        copies_commit();
    }
    for (int64_t p = cta; p < g.pairs; p += ctas, ++n_f) {
        float* fb = fbuf[regen ? 0 : n_f & 1];
        Parts bf[4][NQ][2], af[2][NQ];
        float sum[MEAN ? 2 : 1][2][4];
        for (int it = 0; it < iters; ++it, ++n_x) {
            const float* xb = xbuf[n_x & 1];
            copies_wait();
            __syncthreads();                                  // the copies of all threads are there; xs has been read
            const bool last = it + 1 == iters;
            if (!last) fetch_x(p, it + 1, xbuf[(n_x + 1) & 1]);
            else if (p + ctas < g.pairs) {
                fetch_x(p + ctas, 0, xbuf[(n_x + 1) & 1]);
                if (!regen) fetch_factors(p + ctas, fbuf[(n_f + 1) & 1]);
            }
            copies_commit();
            if (regen && it == 0) make_factors(p, fb);
            // x to parts: four threads per row, 16 inputs each
            {
                const int r = tid >> 2, q0 = (tid & 3) * 16;
                if (q0 < ksteps * 16) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 v = *reinterpret_cast<const float4*>(xb + r * SP_XF + q0 + i);
                        const Parts lo = split2(v.x, v.y), hi = split2(v.z, v.w);
#pragma unroll
                        for (int part = 0; part < 3; ++part)
                            *reinterpret_cast<uint2*>(&xs[part][r][q0 + i]) = make_uint2(lo.p[part], hi.p[part]);
                    }
                }
            }
            __syncthreads();
            if (!busy) continue;
            if (it == 0) {
                // fragments of B (k x rank) and of sA (16 outputs x rank)
                const float* B = fb + (jn - j_lo) * kr;
                const float* A = fb + a_base + warp * ar;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                    for (int nq = 0; nq < NQ; ++nq)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int q = nq * 8 + gr, kk = ks * 16 + h * 8 + tq * 2;
                            bf[ks][nq][h] = split2(q < rank && kk < k ? B[kk * rank + q] : 0.0f,
                                                   q < rank && kk + 1 < k ? B[(kk + 1) * rank + q] : 0.0f);
                        }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int h = 0; h < NQ; ++h) {
                        const int n = nt * 8 + gr, q = h * 8 + tq * 2;
                        const bool in = c0 + n < jb.a;
                        af[nt][h] = split2(in && q < rank ? __fmul_rn(A[n * rank + q], g.base_sigma) : 0.0f,
                                           in && q + 1 < rank ? __fmul_rn(A[n * rank + q + 1], g.base_sigma) : 0.0f);
                    }
            }
            const int nrows = min(SP_ROWS, span - (MEAN ? it / inner : it) * SP_ROWS), t = MEAN ? it % inner : 0;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                if (mt * 16 >= nrows) break;
                float y[2][4] = {}, tt[NQ][4] = {};
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    if (ks >= ksteps) break;
                    uint32_t a[3][4];
#pragma unroll
                    for (int part = 0; part < 3; ++part)
                        load_a(a[part], &xs[part][mt * 16 + (lane & 15)][ks * 16 + (lane >> 4) * 8]);
#pragma unroll
                    for (int nq = 0; nq < NQ; ++nq) mma_parts(tt[nq], a, bf[ks][nq][0], bf[ks][nq][1]);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) mma_parts(y[nt], a, wf[ks][nt][0], wf[ks][nt][1]);
                }
                // t's accumulator is the left operand of the rank term: its column pairs are the k pairs of a fragment
                uint32_t a[3][4] = {};
#pragma unroll
                for (int nq = 0; nq < NQ; ++nq) {
                    const Parts r0 = split2(tt[nq][0], tt[nq][1]), r1 = split2(tt[nq][2], tt[nq][3]);
#pragma unroll
                    for (int part = 0; part < 3; ++part) a[part][2 * nq] = r0.p[part], a[part][2 * nq + 1] = r1.p[part];
                }
                float u[2][4] = {};
                const Parts none{};
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) mma_parts(u[nt], a, af[nt][0], NQ == 2 ? af[nt][NQ - 1] : none);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int r = mt * 16 + half * 8 + gr;
                    if (r >= nrows) continue;
                    const int lr = (MEAN ? it / inner : it) * SP_ROWS + r;
                    const int rr = MEAN ? lr : lr % rows_per_step;
                    const bool odd = rr >= g.bm;              // first_thread is even: a pair's second member
                    const int64_t row = MEAN ? p * 2 * g.bm + rr : row_of(p, it, r);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) {
                        float v[2];
                        const int n = c0 + nt * 8 + tq * 2;
                        float* o = jb.out + (size_t)row * jb.out_stride + n;
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const float uu = u[nt][half * 2 + c];
                            v[c] = __fadd_rn(y[nt][half * 2 + c], odd ? -uu : uu);
                            if (MEAN) {                       // time_mean's arithmetic
                                float& acc = sum[MEAN ? mt : 0][nt][half * 2 + c];
                                v[c] = __fmul_rn(v[c], gain);
                                acc = t == 0 ? __fadd_rn(0.0f, v[c]) : __fadd_rn(acc, v[c]);
                                if (t + 1 == inner) v[c] = __fdiv_rn(acc, (float)inner);
                            } else if (g.lif) {
                                v[c] = __fmul_rn(v[c], g.leak);
                                if (jb.pot && n + c < jb.a) jb.pot[(size_t)row * jb.out_stride + n + c] = v[c];
                                v[c] = v[c] >= g.v_th ? 1.0f : 0.0f;
                            } else {
                                v[c] = __fmul_rn(v[c], gain);
                            }
                        }
                        if (MEAN && t + 1 < inner) continue;
                        if (jb.vec) {
                            if (n < jb.a) *reinterpret_cast<float2*>(o) = make_float2(v[0], v[1]);
                        } else {
                            if (n < jb.a) o[0] = v[0];
                            if (n + 1 < jb.a) o[1] = v[1];
                        }
                    }
                }
            }
        }
    }
}

}  // namespace

bool small_path_supports(const hses_linear_args& g) {
    if (!g.perturb || g.lif == 2 || g.factor_order != 0) return false;
    if (g.k > SP_MAXK || g.a > SP_MAXA || g.rank > SP_MAXR) return false;
    return g.first_thread % 2 == 0 && g.n_pop % 2 == 0;
}

// layers that read the same rows of x with the same noise arguments
bool small_path_joins(const hses_linear_args* g, int n) {
    if (n < 1 || n > SP_JOBS) return false;
    for (int i = 0; i < n; ++i) {
        const hses_linear_args &a = g[i], &b = g[0];
        if (!small_path_supports(a) || a.algo != HSES_ALGO_AUTO || a.x_op || a.n_groups > 1 || a.precision != b.precision) return false;
        if (a.x != b.x || a.x_row_stride != b.x_row_stride || a.t_steps != b.t_steps || a.n_pop != b.n_pop || a.bm != b.bm ||
            a.k != b.k || a.sigma != b.sigma || a.rank != b.rank || a.epoch != b.epoch || a.first_thread != b.first_thread ||
            a.noise_reuse != b.noise_reuse || a.lif != b.lif || (a.cache == nullptr) != (b.cache == nullptr) ||
            a.out_scale != b.out_scale || a.out_scale_ptr != b.out_scale_ptr || a.tau_m != b.tau_m || a.v_th != b.v_th)
            return false;
    }
    return true;
}

int run_small_path(hses_ctx* ctx, cudaStream_t st, const hses_linear_args* args, int n, bool mean) {
    const hses_linear_args& g = args[0];
    SmallArgs s{};
    s.x = g.x;
    s.x_stride = g.x_row_stride;
    s.t_steps = g.t_steps;
    s.bm = g.bm;
    s.k = g.k;
    s.rank = g.rank;
    s.n_pop = g.n_pop;
    s.first_thread = g.first_thread;
    s.pairs = g.n_pop / 2;
    s.base_sigma = g.sigma / sqrtf((float)g.rank);
    s.lif = g.lif;
    s.leak = g.lif ? 1.0f / g.tau_m : 0.0f;
    s.v_th = g.v_th;
    s.out_scale = g.out_scale;
    s.out_scale_ptr = g.out_scale_ptr;
    s.cal = ctx->cal();
    s.jump = ctx->t.jump_tabs;
    s.lane4 = ctx->t.jump_lane4;
    s.true_epoch = true_epoch_of(g.epoch, g.noise_reuse);
    s.first_pair = g.first_thread / 2;
    s.jobs = n;
    s.vec_x = ((uintptr_t)g.x & 15u) == 0 && g.x_row_stride % 4 == 0 && g.k % 4 == 0;
    s.vec_f = g.rank % 4 == 0;
    for (int i = 0; i < n; ++i) {
        SmallJob& j = s.job[i];
        const hses_linear_args& a = args[i];
        if (a.cache) {
            int rc = resolve_factor_cache(a, &j.A, &j.B);
            if (rc != HSES_OK) return rc;
        }
        if (((uintptr_t)j.A & 15u) || ((uintptr_t)j.B & 15u)) s.vec_f = 0;
        j.w = a.param;
        j.w_stride = a.param_row_stride;
        j.key = a.key;
        j.out = a.out;
        j.out_stride = a.out_row_stride;
        j.pot = a.lif ? a.potentials : nullptr;
        j.a = a.a;
        j.slice0 = s.slices;
        j.vec = ((uintptr_t)a.out & 7u) == 0 && a.out_row_stride % 2 == 0 && a.a % 2 == 0;
        s.slices += (a.a + 15) / 16;
    }
    s.groups = (s.slices + SP_SLICES - 1) / SP_SLICES;
    const int smem = sp_bytes(s.k, s.rank);
    // one wave of resident CTAs, so that W is split once per CTA
    const int per_sm = std::max(1, std::min(3, 225 * 1024 / (smem + 24 * 1024)));
    const int64_t walkers = std::max<int64_t>(1, std::min<int64_t>(s.pairs, (int64_t)ctx->sm_count * per_sm / s.groups));
    auto kernel = s.rank > 8 ? (mean ? small_pair_kernel<2, true> : small_pair_kernel<2, false>)
                             : (mean ? small_pair_kernel<1, true> : small_pair_kernel<1, false>);
    HSES_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    HSES_KERNEL(ctx, st, "small_pair");
    chain_launch(kernel, (unsigned)(walkers * s.groups), SP_THREADS, smem, st, s);
    HSES_LAUNCH_CHECK();
    return HSES_OK;
}

}  // namespace hses
