// Internal interfaces between the kernels that make up a layer's forward.
#pragma once
#include "common.cuh"

namespace natsl {

constexpr int TBL_LOGITS = 100;            // dtype code of launch_tables: selection logits instead of types

// The selection tables (natsl_build_tables without the compact list), from types or from bf16 logits (then types_raw
// [B,TN,HN,2] bf16 receives the sampled types and the last block is forced to both).  starting_h_idx may be NULL.
int launch_tables(const void* types, int dtype, void* types_raw, int B, int TN, int HN, int T, int nbs, int* types_i, int* indices,
                  int* n_blocks, int* n_chunks_lin, int* starting_h_idx, int* attn_n_iters, cudaStream_t st);

}  // namespace natsl
