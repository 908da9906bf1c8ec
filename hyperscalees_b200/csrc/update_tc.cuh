// Interface between the update dispatcher (update.cu) and its tensor-core path (update_tc.cu).
#pragma once

#include "common.cuh"

namespace hses {

struct UpdateTcPlan {
    int64_t pairs, chunk_pairs;
    int bn, n_tiles, m_tiles, splits;
    size_t partial_bytes, raw_bytes, bytes;
};

// rank a multiple of 64: the shapes the tcgen05 contraction covers (ragged a and b are zero-filled)
bool update_tc_supports(int a, int b, int rank);
// need_raw: room for one chunk of regenerated fp32 factors (no factor cache)
UpdateTcPlan plan_update_tc(int a, int b, int rank, int64_t n, bool need_raw);
// grad (+)= scale * sum_p (f_2p - f_2p+1) A_p B_pᵀ; arguments already validated by the caller
// reuse_range: the power-of-two range of the pair weights that an earlier call with the same
// fitness vector and workspace left at the start of the workspace is still there (the layers of one
// model share both), so it is not computed again
int run_update_tc(hses_ctx* ctx, cudaStream_t stream, const hses_update_args& u, float scale,
                  bool reuse_range = false);
// hses_es_update_ex with that option
int es_update_ex_impl(hses_ctx* ctx, hses_stream stream, const hses_update_args* args, bool reuse_range);

// The update of several matrices that share rank, fitness vector and members, for any rank, in one set of launches
// (update_multi.cu).
constexpr int kUpdateMulti = 48;
struct UpdateMultiItem {
    uint64_t key;
    int a, b;
    const float *cache_a, *cache_b;   // raw factors of the call's first pair, or NULL: regenerate
    float* grad;                      // (a, b) dense
};
struct UpdateMultiCall {
    int32_t epoch, noise_reuse, first_thread;
    int64_t n;                        // members (whole pairs)
    int rank;
    const float* fitness;
    float scale;                      // of the sum
    int sign_factors;
    int add_to_grad;                  // add to `grad` instead of writing it
    void* workspace;
    size_t workspace_bytes;
};
size_t update_multi_workspace_bytes(const int* a, const int* b, int n, int rank, int64_t members);
int run_update_multi(hses_ctx* ctx, cudaStream_t stream, const UpdateMultiItem* items, int n, const UpdateMultiCall& call);
// checks a cache descriptor against an update and returns the factors of its first pair
int resolve_update_cache(const hses_factor_cache& c, uint64_t key, int32_t true_epoch, int rank, int a, int b, int32_t first_pair,
                         int64_t pairs, const float** cache_a, const float** cache_b);

}  // namespace hses
