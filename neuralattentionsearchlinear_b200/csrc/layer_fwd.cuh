// Internal interfaces between the kernels that make up a layer's forward.
#pragma once
#include "common.cuh"

namespace natsl {

constexpr int TBL_LOGITS = 100;            // dtype code of launch_tables: selection logits instead of types

// The selection tables (natsl_build_tables without the compact list), from types or from bf16 logits (then types_raw
// [B,TN,HN,2] bf16 receives the sampled types and the last block is forced to both).  starting_h_idx may be NULL.
int launch_tables(const void* types, int dtype, void* types_raw, int B, int TN, int HN, int T, int nbs, int* types_i, int* indices,
                  int* n_blocks, int* n_chunks_lin, int* starting_h_idx, int* attn_n_iters, cudaStream_t st);

// Narrow projections with their pointwise steps (narrow_tc.cu).
struct NarrowArgs {
    const __nv_bfloat16 *x, *w0, *w1;         // x [B,T,Kdim]; w0 [n0,Kdim], w1 [n1,Kdim] or NULL
    int n0, n1, T, Kdim, mode;                // mode 0: decays (w0) and betas (w1); mode 1: softmax over pairs of rows
    const void *A_log, *dt_bias;
    int alog_f32, dt_f32, neg_eigval, wide;   // wide (set by the launch): mode 1 stores 16 bytes
    float *g, *gcs, *dt;                      // [B,T,n0]; gcs, dt or NULL
    __nv_bfloat16* out;                       // mode 0: beta [B,T,n1]; mode 1: weights [B,T,n0]
};
int launch_narrow(const NarrowArgs& a, int B, cudaStream_t st);

}  // namespace natsl
