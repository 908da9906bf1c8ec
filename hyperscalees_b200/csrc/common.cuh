// Shared declarations of the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <string>
#include <vector>

#include "../../include/hses.h"
#include "rng.cuh"

namespace hses {

void set_error(const std::string& msg);

struct DeviceTables {
    // the generator's tables (see NoiseCal)
    float4* log_tab = nullptr;
    float4* cos_tab = nullptr;
    float* cos_width = nullptr;
    uint32_t* log_flip = nullptr;
    uint32_t* cos_flip = nullptr;
    // inputs the host libm does not round correctly (reported by hses_ctx_calibration_info)
    uint64_t n_log_flips = 0, n_cos_flips = 0;
    // generator jump tables: entry k advances the state by 2^k steps
    uint64_t* jump_tabs = nullptr;  // see jump_by: 16 matrices for each of kJumpLevels / 4 digits
    // lane tables (see lane_jump): lane l goes 4 l or 16 l normals (two steps each) ahead
    uint64_t *jump_lane4 = nullptr, *jump_lane16 = nullptr;
    // one int per device: kernels with bounded waits record here why they gave up
    int* status_word = nullptr;
};

// Nibble table (kJumpWords uint64) that advances the generator by `distance`
// steps, built on first use and cached per device.
int get_hop_table(hses_ctx* ctx, uint64_t distance, const uint64_t** dev_tab);

constexpr int kJumpLevels = 48;

// Multiprocessor count the split-K planners size their grids for: that of the current CUDA
// device, read once (the *_workspace_bytes entry points have no context to ask).  Every device
// this library accepts is an sm_100 part, so a process sees one value.
int plan_sm_count();

// Per-context launch counters and optional CUDA-event timing of every kernel
// the library launches (hses_profile_* in the C ABI).
struct KernelStat {
    const char* name = nullptr;
    int64_t launches = 0;
    double ms = 0.0;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pending;
};
struct Profiler {
    bool timing = false;
    std::vector<KernelStat> stats;
    std::vector<cudaEvent_t> pool;
    KernelStat& get(const char* name);
    cudaEvent_t event();
};
struct KernelScope {
    Profiler* prof;
    KernelStat* stat;
    cudaStream_t stream;
    cudaEvent_t start = nullptr;
    KernelScope(Profiler& p, cudaStream_t s, const char* name) : prof(&p), stat(&p.get(name)), stream(s) {
        stat->launches++;
        if (p.timing) {
            start = p.event();
            cudaEventRecord(start, s);
        }
    }
    ~KernelScope() {
        if (start) {
            cudaEvent_t stop = prof->event();
            cudaEventRecord(stop, stream);
            stat->pending.emplace_back(start, stop);
        }
    }
};

}  // namespace hses

struct hses_ctx {
    int device = 0;
    int sm_count = 0;
    hses::DeviceTables t;
    hses::Profiler prof;
    hses::NoiseCal cal() const { return {t.log_tab, t.cos_tab, t.cos_width, t.log_flip, t.cos_flip}; }
};

#define HSES_CUDA(call)                                                                   \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            hses::set_error(std::string(#call) + " failed: " + cudaGetErrorString(e_));   \
            return HSES_ERR_CUDA;                                                         \
        }                                                                                 \
    } while (0)

#define HSES_REQUIRE(cond, msg)                                   \
    do {                                                          \
        if (!(cond)) {                                            \
            hses::set_error(std::string(__func__) + ": " + (msg)); \
            return HSES_ERR_INVALID;                              \
        }                                                         \
    } while (0)

// Counts (and, when profiling is on, times) the kernel launched right after it.
#define HSES_KERNEL(ctx, stream, name) hses::KernelScope hses_kernel_scope_((ctx)->prof, (stream), (name))

// Launches of a chain of kernels on one stream (programmatic dependent launch): the next kernel's blocks may be set up while
// this one still runs, which saves 2 to 4 us per link of a chain of short kernels.  A kernel launched by chain_launch calls
// chain_next (its successor may be set up once every block has) and, before it touches memory that any kernel before it
// writes or reads, chain_wait: that returns when its predecessor has ended, and so, since each of them waits, all before.
#if defined(__CUDACC__)
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_begin() {
    chain_next();
    chain_wait();
}
template <class... P, class... A>
inline void chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);   // an error is the launch check's to report
}
#endif

#define HSES_LAUNCH_CHECK()                                                                 \
    do {                                                                                    \
        cudaError_t e_ = cudaGetLastError();                                                \
        if (e_ != cudaSuccess) {                                                            \
            hses::set_error(std::string(__func__) + ": launch failed: " + cudaGetErrorString(e_)); \
            return HSES_ERR_CUDA;                                                           \
        }                                                                                   \
    } while (0)

namespace hses {
// Raw factors of `pairs` antithetic pairs starting at first_pair:
// A (pairs, a, r) and B (pairs, b, r), row-major.  When pair_weight is given
// (device, 2 floats per pair: the fitnesses of the even and the odd member),
// A is multiplied by (f_even - f_odd).
int launch_pair_factors(hses_ctx* ctx, cudaStream_t stream, uint64_t key, int32_t true_epoch,
                        int32_t first_pair, int64_t pairs, int rank, int a, int b,
                        const float* pair_weight, float* A, float* B);
// One solver step (hses_solver_step's arithmetic) over several tensors in one launch, from `src` (NULL: in place) into
// `params`; tensors with a NULL parameter skipped.
int solver_step_multi(hses_ctx* ctx, cudaStream_t st, const hses_solver* solver, int32_t step, float grad_scale, int n_tensors,
                      const float* const* src, float* const* params, float* const* m_bufs, float* const* v_bufs,
                      const int64_t* lens, const float* const* grads);
#if defined(__CUDACC__)
// The normals pos0 .. pos0+cnt of the stream seeded by s0, made by the whole block: emit(offset, z) gets four at a time
// (offset a multiple of four; the last four may run past cnt).  The states of runs of 512 (128 when there is little to
// do) come from the power-of-two tables, one per thread side by side, those of a warp's lanes inside a run from a lane
// table.  state_s: room for max(32, ceil(cnt / 512)) states; cal: staged (stage_cal), the call synchronises.
constexpr int kStreamCoarse = 2048;   // from here on sixteen normals per thread and table round keep half a block busy
template <class Emit>
__device__ __forceinline__ void stream_fill(const NoiseCal& cal, const uint64_t* __restrict__ jump,
                                            const uint64_t* __restrict__ lane4, const uint64_t* __restrict__ lane16,
                                            uint64_t s0, uint64_t pos0, int cnt, uint64_t* state_s, Emit emit) {
    const bool coarse = cnt >= kStreamCoarse;
    const int chn = coarse ? 16 : 4, run = 32 * chn, runs = (cnt + run - 1) / run, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < runs; e += blockDim.x) state_s[e] = jump_by(jump, s0, 2ull * (pos0 + (uint64_t)e * run));
    __syncthreads();
    for (int e = threadIdx.x >> 5; e < runs; e += blockDim.x >> 5) {
        const int off = e * run + lane * chn;
        if (off >= cnt) continue;
        uint64_t st = lane_jump(coarse ? lane16 : lane4, state_s[e], lane);
#pragma unroll 1
        for (int j = 0; j < chn && off + j < cnt; j += 4) {
            float z[4];
            normals4(st, cal, z);
            emit(off + j, z);
        }
    }
}
#endif
#if defined(__CUDACC__)
__device__ __forceinline__ uint32_t poisson_seed(uint32_t idx, uint32_t mix) {
    return 1000000007u * idx + mix + 0x9E3779B9u;
}

__device__ __forceinline__ uint32_t xs32(uint32_t x) {
    x ^= x << 13;
    x ^= x >> 17;
    x ^= x << 5;
    return x;
}

// The reference compares u = fl((k+1)/8388609) with p at every step, k being the top 23 bits of the xorshift32 output.
// fl(n/D) is monotone in n, so a step spikes when k < q, q = the number of n >= 1 whose quotient stays below p; one
// division per element finds it, and a step is a comparison of the raw state: k < q is state <= (q << 9) - 1.
struct PoissonCell {
    uint32_t x, last;
};
__device__ __forceinline__ PoissonCell poisson_cell(float p, uint32_t seed) {
    const float D = 8388609.0f;
    uint32_t q = 0;                                // 0 .. 2^23
    if (p >= 1.0f) {
        q = 8388608u;
    } else if (p > 0.0f) {
        // below: the largest integer under pD = hi + lo.  Its quotient may reach p by rounding up; that of the integer
        // before cannot, it is more than half a unit in the last place away
        const float hi = __fmul_rn(p, D), lo = __fmaf_rn(p, D, -hi), f = floorf(hi);
        const float below = hi > f || lo > 0.0f ? f : __fsub_rn(f, 1.0f);
        if (below >= 1.0f) q = (uint32_t)below - (__fdiv_rn(below, D) >= p ? 1u : 0u);
    }
    PoissonCell c;
    c.x = q ? seed : 1u;                           // a cell that never spikes: any state but 0, which stays as it is
    c.last = q ? (q << 9) - 1u : 0u;
    return c;
}
// fitness of one sample (hyperscalees-envs/src/snn_mnist.rs:180-201)
__device__ __forceinline__ float sample_fitness(const float* row, int classes, int label, int reward) {
    float mx = row[0];
    int arg = 0;
    for (int c = 1; c < classes; ++c)
        if (row[c] > mx) { mx = row[c]; arg = c; }
    if (reward == HSES_REWARD_BINARY) return arg == label ? 1.0f : 0.0f;
    float sum = 0.0f;
    for (int c = 0; c < classes; ++c) sum = __fadd_rn(sum, expf(__fsub_rn(row[c], mx)));
    const float picked = (label >= 0 && label < classes) ? row[label] : __int_as_float(0x7fc00000);
    return __fsub_rn(__fsub_rn(picked, mx), logf(sum));
}
#endif
#if defined(__CUDACC__)
// x * sigmoid(x)
__device__ __forceinline__ float swish_of(float v) { return __fmul_rn(v, __frcp_rn(__fadd_rn(1.0f, expf(-v)))); }
#endif
// lif_step (hyperscalees-models/src/snn.rs:53-65): charge, threshold, reset; returns the spike
__device__ __forceinline__ float lif_update(float& v, float cur, float leak, float v_th, int reset) {
    float d = __fadd_rn(-v, cur);
    float m = __fmul_rn(d, leak);
    float c = __fadd_rn(v, m);
    float s = c >= v_th ? 1.0f : 0.0f;
    v = reset == HSES_RESET_HARD ? __fmul_rn(c, __fadd_rn(-s, 1.0f)) : __fsub_rn(c, __fmul_rn(s, v_th));
    return s;
}


}  // namespace hses

static inline cudaStream_t as_stream(hses_stream s) { return reinterpret_cast<cudaStream_t>(s); }
