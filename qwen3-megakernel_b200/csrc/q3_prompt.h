// The dense products of a prompt's layers (q3_prompt.cu) and the tiled causal attention between them (q3_prefill_attn_tc.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "q3_layered.h"

struct CUtensorMap_st;   // <cuda.h>'s tensor map

namespace q3 {

constexpr int PR_SSQ_PARTS = 16;   // partial sums of squares of a residual row that the embedding gather leaves: one per 64 elements
constexpr int PR_SSQ_MOST = 32;    // ... that a launch may leave: one per tile of weight rows

enum { PR_QKV = 0, PR_RESID = 1, PR_SILU = 2 };

// out = epilogue(in . w^T) for T tokens.  `in` is ONE bf16 plane [T][K]; for PR_QKV and PR_SILU it holds x * gain and lacks the RMS
// norm's scale, which the epilogue takes from the partial sums of squares.
struct PromptGemmCall {
    int kind, T, K;
    const void* w[3];              // PR_QKV: Wq, Wk, Wv; PR_RESID: Wo or Wd; PR_SILU: Wg, Wu
    const ::CUtensorMap_st* in;    // boxes of prompt_box_rows(T) rows x 64 columns over [T][K]
    float* ssq;                    // [PR_SSQ_MOST][ssq_ld]: written by PR_RESID, read by the other two
    int ssq_ld;
    int* parts;                    // how many of them a row has: set by PR_RESID, read by the other two
    // PR_QKV: head norm, RoPE, then
    bf16_raw *q_hi, *q_lo;         // [T][2048] q times the softmax scale as two planes (read by the tiled attention), or
    float* qkv;                    // [T][4096] fp32 q, k, v rows (read by the split attention of few tokens)
    bf16_raw *kc, *vc;             // this layer's cache rows [T..][1024]
    const bf16_raw *qn, *kn;       // [128] head gains of this layer
    const float* rope;             // [positions][128], 16-byte aligned
    // PR_RESID
    float* x;                      // [T][1024], updated in place
    bf16_raw* xn;                  // [T][1024] plane of x * gain
    const bf16_raw* gain;          // gain of the norm that reads x next
    // PR_SILU
    bf16_raw* hid;                 // [T][3072]
    uint32_t* status;
};
// rows of the boxes over the activations: no more than the prompt has (rows past it would be filled with zeros at a row's price: 16 tokens 1045 -> 837 us)
inline int prompt_box_rows(int T) { return T < 128 ? (T + 15) / 16 * 16 : 128; }
cudaError_t launch_prompt_gemm(const PromptGemmCall& c, cudaStream_t st);

// x[t] = embed[ids[t]], its plane times `gain`, its partial sums of squares; a bad id is reported and read as 0
cudaError_t launch_prompt_embed(const long long* ids, const bf16_raw* embed, int vocab, float* x, const bf16_raw* gain, bf16_raw* xn, float* ssq, int ssq_ld,
                                uint32_t* status, int T, cudaStream_t st);

// causal attention of a prompt of T >= 1 tokens: q planes and caches as above -> bf16 plane [T][2048]
cudaError_t launch_prefill_attn_tc(const ::CUtensorMap_st& q_hi, const ::CUtensorMap_st& q_lo, const ::CUtensorMap_st& k, const ::CUtensorMap_st& v, int layer,
                                   void* plane, int T, uint32_t* status, cudaStream_t st);

}  // namespace q3
