// Split-K tensor-core GEMM whose k slices are the blocks of a cluster: the products of one transformer layer between two
// attentions, for decode batches of at most 64 sequences (q3_gemm_cl.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "q3_layered.h"

namespace q3 {

constexpr int CL_PLANES = 3;       // bf16 planes of the activations: exact to fp32
constexpr int CL_MAX_TOK = 64;     // most tokens of a call (65 / 96 / 128 sequences at 256 positions, this chain 1694 / 1957 / 2291 us a step, one launch
                                   // per phase 1610 / 1829 / 2057)
constexpr int CL_SSQ_PARTS = 32;   // partial sums of squares of a residual row: one per 32 elements

enum { CL_QKV = 0, CL_RESID = 1, CL_SILU = 2 };

// The residual stream's side of a layer: the fp32 rows, their planes (already times the next norm's gain, not yet times
// its scale) and the partial sums of squares the scale is taken from.
struct ClusterGemmCall {
    int kind;
    const void* w[3];          // CL_QKV: Wq, Wk, Wv; CL_RESID: Wo or Wd; CL_SILU: Wg, Wu
    int K;                     // 1024, 2048 or 3072
    const bf16_raw* in;        // bf16 [CL_PLANES][prow][K]
    int prow, n_tok;
    float* out;                // CL_QKV: [n_tok][4096]; CL_RESID: x [n_tok][1024], updated in place
    bf16_raw* planes;          // CL_RESID: [CL_PLANES][prow][1024]; CL_SILU: [CL_PLANES][prow][3072]
    const bf16_raw* gain;      // CL_RESID: gain of the norm that reads x next
    float* ssq;                // [CL_SSQ_PARTS][ssq_ld]: written by CL_RESID, read by the other two
    int ssq_ld;
    uint32_t* status;
};
cudaError_t launch_gemm_cluster(const ClusterGemmCall& c, cudaStream_t st);
int gemm_cluster_rows(int n_tok);   // rows a plane needs for n_tok tokens

// x[t] = embed[token[t]], its planes times `gain`, its partial sums of squares; otherwise as launch_embed
cudaError_t launch_embed_planes(const long long* token, const bf16_raw* embed, int vocab, float* x, const bf16_raw* gain, bf16_raw* planes, int prow,
                                float* ssq, int ssq_ld, uint32_t* status, int batch, cudaStream_t st, unsigned long long* argmax_keys,
                                unsigned* argmax_tickets, const int* seq_len, int len_bound);

}  // namespace q3
