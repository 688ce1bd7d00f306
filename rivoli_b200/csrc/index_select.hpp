// Interface between the indexer's host entry points (index_mma.cu) and the cluster selection kernel
// (index_select.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/rivoli_kernels.h"

constexpr int SEL_MAX_CLUSTER = 8;   // portable cluster size

struct SelArgs {
    DsaGeom g;
    const float* scores; int score_stride; const int32_t* seq_len;
    const uint8_t* qcodes; const float* qscales; const float* w; const float* cb;
    const uint8_t* index_pool; const float* index_scale; const int32_t* block_table;
    uint32_t* rows; int32_t* n_sel; int k;
    unsigned int* stats;   // [B][2]: band size, sure-in count (may be NULL)
    int vec_ok;            // key scales allow 16-byte loads (paged scores)
    int vec_scores;        // score rows do
    int* err;              // error word of the scorer
    int nt_single; long long value_stride;   // selection over given scores: tokens when seq_len is NULL, pitch of the score rows
};

namespace rivoli {
// Launches the selection as a programmatic dependent of the kernel before it in the stream. 0, a guard code or
// -(cudaError_t).
int launch_index_select_cluster(const SelArgs& a, int B, cudaStream_t st);
// Exact top-k of given scores (ties -> lower index, ascending output), B rows of up to max_nt <= 131,072 scores; seq_len
// NULL = nt_single each, n_sel may be NULL. 1002 beyond that length.
int launch_topk_values(const float* scores, long long stride, const int32_t* seq_len, int nt_single, int B, int k,
                       uint32_t* rows, int32_t* n_sel, int max_nt, cudaStream_t st);
}  // namespace rivoli
