// Interface between the SNN population step (snn.cu) and its fused forward pass (snn_layer.cu).
#pragma once

#include "common.cuh"

namespace hses {

struct SnnInput {
    // exactly one of the two: spikes (T, rows, dims[0]) f32 with a row stride, or images (rows, dims[0]) to encode
    const float* spikes;
    const float* images;
    int64_t stride;
    const uint32_t* seeds;
};
struct SnnScore {              // per-member fitness behind the readout; labels NULL: logits only
    const int32_t* labels;
    int32_t reward;
    float* raw_fitness;        // (n_pop)
};
// Models whose hidden layers and readout all run in the fused kernels; decided by shapes alone.
bool snn_fused_supports(const hses_snn_model* m, const hses_pop_args* p);
size_t snn_fused_workspace_bytes(const hses_snn_model* m, const hses_pop_args* p);
// logits (rows, classes) may be NULL when a score is asked for
int run_snn_fused(hses_ctx* ctx, cudaStream_t st, const hses_snn_model* m, const hses_pop_args* p, const SnnInput& in,
                  float* logits, const SnnScore& score, void* workspace, size_t workspace_bytes);

}  // namespace hses
