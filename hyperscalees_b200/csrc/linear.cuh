// Interface between the perturbed-linear dispatcher and its tensor-core path.
#pragma once

#include "common.cuh"

namespace hses {

// True when the tcgen05 kernel covers the shapes/pitches of this call.
bool tensor_path_supports(const hses_linear_args& g);
size_t tensor_path_workspace_bytes(const hses_linear_args& g);
int run_tensor_path(hses_ctx* ctx, cudaStream_t stream, const hses_linear_args& g);

// The path for few rows per antithetic pair and wide factors (linear_pair.cu): clean product
// through the other paths, then one CTA per pair that streams the pair's factors once.
bool pair_path_supports(const hses_linear_args& g);
bool pair_path_fuses_scan(const hses_linear_args& g);   // lif == 2 is finished inside the per-pair kernel
size_t pair_path_workspace_bytes(const hses_linear_args& g);
// scanned: the rows are currents that a LIF scan turns into spikes
int run_pair_path(hses_ctx* ctx, cudaStream_t stream, const hses_linear_args& g, bool scanned);

// Narrow layers (k, a <= 64, rank <= 16; linear_small.cu): persistent CTAs keep W in registers and
// walk over pairs.  Taken by HSES_ALGO_AUTO only.
// Several layers over the same x run in one launch when small_path_joins says so.
bool small_path_supports(const hses_linear_args& g);
bool small_path_joins(const hses_linear_args* args, int n);
int run_small_path(hses_ctx* ctx, cudaStream_t stream, const hses_linear_args* args, int n, bool mean);

// Layers with many rows per member and weights that fit shared memory (linear_rows.cu).  Taken by HSES_ALGO_AUTO only.
struct RowsPost {          // what follows the layer: nothing, swish, out += y, the firing rate of constant currents
    int kind, steps;
    float leak, v_th;
    int reset;
};
bool rows_path_supports(const hses_linear_args& g);
size_t rows_path_workspace_bytes(const hses_linear_args& g);
int run_rows_path(hses_ctx* ctx, cudaStream_t stream, const hses_linear_args& g, const RowsPost& post);

// Any other shape on the tensor cores (linear_pack.cu): rows packed per antithetic pair, ragged widths and
// pitches, ranks up to 128.  Taken by HSES_ALGO_AUTO only.
bool pack_path_supports(const hses_linear_args& g);
size_t pack_path_workspace_bytes(const hses_linear_args& g);
int run_pack_path(hses_ctx* ctx, cudaStream_t stream, const hses_linear_args& g);

// Checks args.cache against the call and returns the cached raw factors of the call's
// first pair: A rows (pair, a, rank) and B rows (pair, k, rank).
int resolve_factor_cache(const hses_linear_args& g, const float** A, const float** B);

}  // namespace hses
