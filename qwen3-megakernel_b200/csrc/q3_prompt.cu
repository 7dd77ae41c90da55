// The dense products of a prompt's layers on tcgen05, finished in the epilogue: q/k/v with head norms, RoPE, q planes and cache rows;
// Wo and down with the residual, the next norm's plane and its sums of squares; gate/up with SiLU.  Five launches a layer (q/k/v,
// attention, Wo, gate/up, down) and nothing between them.
//
// The tokens are the M operand (TMEM lanes) and the weight rows the columns, so that everything an epilogue does to a token's row
// (its norm's scale, a head's norm, RoPE's pairs) stays inside one TMEM lane.
//
// The RMS norm commutes with the product: the producer of x writes bf16(x * gain) and sixteen partial sums of squares per row, the
// consumer's epilogue multiplies by rsqrt(mean + eps) in fp32.  One bf16 plane, rounded once, like the planes of x * r * gain before it.
#include <cuda.h>

#include "q3_engine.h"
#include "q3_gemm_tc.h"
#include "q3_prompt.h"
#include "q3_tc_ptx.cuh"

namespace q3 {

constexpr int PR_BM = 128;         // tokens of a block
constexpr float PR_QS = ATTN_SCALE * 1.4426950408889634f;   // scores in units of log2, as the tiled attention wants them

struct PromptParams {
    int T, kb_total, ssq_ld, ssq_parts;   // ssq_parts: partial sums of squares a row of ssq_in has
    const float* ssq_in;
    float* ssq_out;
    bf16_raw *q_hi, *q_lo;
    float* qkv;
    bf16_raw *kc, *vc;
    const bf16_raw *qn, *kn;
    const float* rope;
    float* x;
    bf16_raw* xn;
    const bf16_raw* gain;
    bf16_raw* hid;
    uint32_t* status;
    int n_tiles, n_items, stages;   // pair kernel
    int a_rows;                     // rows of the activations' box
};

__device__ __forceinline__ uint32_t pr_pack(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ uint2 pr_pack4(float4 v) { return make_uint2(pr_pack(v.x, v.y), pr_pack(v.z, v.w)); }
__device__ __forceinline__ float4 pr_unpack4(uint2 u) { return make_float4(bf_lo(u.x), bf_hi(u.x), bf_lo(u.y), bf_hi(u.y)); }
__device__ __forceinline__ float4 pr_mul(float4 a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
__device__ __forceinline__ float4 pr_mul(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 pr_add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float pr_dot(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }
// a prompt's products are bf16: __expf and the approximate division are far inside that
__device__ __forceinline__ float pr_silu(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }

// scale of token t's RMS norm from the partial sums of squares
__device__ __forceinline__ float pr_scale(const PromptParams& p, int t) {
    float ss = 0.f;
    for (int i0 = 0; i0 < p.ssq_parts; i0 += 16)
#pragma unroll
        for (int i = 0; i < 16; ++i) ss += p.ssq_in[(size_t)(i0 + i) * p.ssq_ld + t];
    return rsqrtf(ss / (float)HIDDEN + EPS);
}

// RoPE's cosines and sines of dims d .. d + 3 of position t.  The table is nobody's output: read past the stores around it.
struct PrRope { float4 c, s; };
__device__ __forceinline__ PrRope pr_rope(const PromptParams& p, int t, int d) {
    const float* row = p.rope + (size_t)t * HEAD_DIM + d;
    return PrRope{__ldg(reinterpret_cast<const float4*>(row)), __ldg(reinterpret_cast<const float4*>(row + 64))};
}
// One half-row step of a finished q, k or v head: dims d .. d + 3 (lo) and 64 + d .. 64 + d + 3 (hi) of `col0`'s head (a multiple of 128
// in q | k | v) of token t.  lo and hi are normalised except for the head's gain (v: final).
__device__ __forceinline__ void pr_finish_head(const PromptParams& p, int col0, int t, int d, float4 lo, float4 hi, float4 glo, float4 ghi, const PrRope& r) {
    if (col0 < Q_DIM + KV_DIM) {
        lo = pr_mul(lo, glo); hi = pr_mul(hi, ghi);
        const float4 c = r.c, s = r.s;
        const float4 a = make_float4(lo.x * c.x - hi.x * s.x, lo.y * c.y - hi.y * s.y, lo.z * c.z - hi.z * s.z, lo.w * c.w - hi.w * s.w);
        hi = make_float4(hi.x * c.x + lo.x * s.x, hi.y * c.y + lo.y * s.y, hi.z * c.z + lo.z * s.z, hi.w * c.w + lo.w * s.w);
        lo = a;
    }
    if (p.qkv != nullptr) {
        float* o = p.qkv + (size_t)t * QKV_DIM + col0 + d;
        *reinterpret_cast<float4*>(o) = lo;
        *reinterpret_cast<float4*>(o + 64) = hi;
        if (col0 < Q_DIM) return;
    }
    if (col0 < Q_DIM) {
        lo = pr_mul(lo, PR_QS); hi = pr_mul(hi, PR_QS);
        const size_t o = (size_t)t * Q_DIM + col0 + d;
        const uint2 l = pr_pack4(lo), h = pr_pack4(hi);
        *reinterpret_cast<uint2*>(p.q_hi + o) = l;
        *reinterpret_cast<uint2*>(p.q_hi + o + 64) = h;
        const float4 lr = pr_unpack4(l), hr = pr_unpack4(h);
        *reinterpret_cast<uint2*>(p.q_lo + o) = pr_pack4(make_float4(lo.x - lr.x, lo.y - lr.y, lo.z - lr.z, lo.w - lr.w));
        *reinterpret_cast<uint2*>(p.q_lo + o + 64) = pr_pack4(make_float4(hi.x - hr.x, hi.y - hr.y, hi.z - hr.z, hi.w - hr.w));
    } else {
        bf16_raw* o = (col0 < Q_DIM + KV_DIM ? p.kc + (col0 - Q_DIM) : p.vc + (col0 - Q_DIM - KV_DIM)) + (size_t)t * KV_DIM + d;
        *reinterpret_cast<uint2*>(o) = pr_pack4(lo);
        *reinterpret_cast<uint2*>(o + 64) = pr_pack4(hi);
    }
}
__device__ __forceinline__ const bf16_raw* pr_head_gain(const PromptParams& p, int col0) { return col0 < Q_DIM ? p.qn : p.kn; }

__device__ __forceinline__ uint32_t pr_map(uint32_t smem_addr, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void pr_cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void pr_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void pr_mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void pr_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(bar)), "r"(bytes) : "memory");
}

// ------------------------------------------------------------------------------------------------------------------------------
// Short prompts: a block takes 128 tokens x BN weight rows (PR_RESID: x one of C slices of K).  What such a launch takes is a chain of latencies, so BN
// is chosen for about one block an SM, and the epilogue for the fewest exchanges:
//   PR_QKV    BN columns of a head, half of them from either half of the head, so that RoPE's pairs stay in a thread; the blocks of a head are a
//             cluster and exchange the sums of squares of their columns (512 bytes), nothing else
//   PR_SILU   BN / 2 rows of Wg and the same of Wu, nothing to exchange
//   PR_RESID  K is long (2048, 3072) and N short (1024): the C slices of K are the blocks of a cluster, each owns a run of the tile's token rows,
//             sends its partial sums of the others' rows to their owners with bulk copies through distributed shared memory and finishes its
//             own: no atomics, no cleared buffers, the same result on every run
// Exchanging partial tiles is what costs (48 KB a block 2 to 4 us, 16 KB about 1): q/k/v of 128 tokens in four slices of K took 9.2 us from its wait
// to its last exit, without slices 7.4; gate/up in two slices 7.9, without 6.0.
//
// OCC: blocks that fit an SM.  One with a ring of up to 222 KB has nearly all of its loads under way at once; two overlap one another's
// phases where a launch has more blocks than SMs.  Either way a block of the next launch finds room as this launch's blocks end, sets up and requests its
// weights before the wait.  A partial tile is [row][BN] fp32 with the 16-byte chunks of a row XORed by row & 7, so
// that a thread per row writes it and a group of lanes per row reads it without bank conflicts; it overlays the stages.
//
// Tensor memory of an SM: a block waits for its cluster while it holds its columns, so the blocks that fit on an SM may not ask for more than 512
// together (q3_gemm_cl.cu).  Two of these are 256 at most and leave no room for a decode product's 58 KB; one of a single-block shape leaves none
// either, and has no cluster to wait for or 64 columns at most.
// A block of the pair kernel (512 columns) has more shared memory than any of them leaves.
//
// A wait that gives up: as in q3_gemm_cl.cu (a block without its sums sends and stores nothing, everyone meets at every cluster
// barrier, and what was under way is drained before the block leaves).
// ------------------------------------------------------------------------------------------------------------------------------
constexpr int PS_THREADS = 192;    // warp 0: TMA, warp 1: MMA and TMEM, warps 2..5: epilogue
constexpr int PS_MAX_STAGES = 12;
constexpr unsigned long long PS_RED_WAIT_NS = 2 * TC_WAIT_NS;

template <int KIND, int BN, int C, int OCC> struct PsShape {
    static constexpr int CL = KIND == PR_QKV ? HEAD_DIM / BN : C;                     // blocks of a cluster: a head's columns, or the slices of K
    static constexpr int ROWS = PR_BM / C;                                            // most rows a block finishes
    static constexpr uint32_t A_BYTES = PR_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr uint32_t RED = (C - 1) * ROWS * BN * 4;                          // partial rows from the other blocks
    static constexpr int FIT = ((OCC == 1 ? 222 : KIND == PR_QKV && CL > 1 ? 110 : 112) * 1024 - RED) / STAGE;   // (two blocks an SM: 113 KB each, with the static ones)
    static constexpr int STAGES = FIT < PS_MAX_STAGES ? FIT : PS_MAX_STAGES;
    static constexpr size_t SMEM = STAGES * STAGE + RED;
    static constexpr uint32_t COLS = BN <= 32 ? 32 : BN <= 64 ? 64 : BN <= 128 ? 128 : 256;   // TMEM columns
    static_assert(C == 1 || STAGES * STAGE >= PR_BM * BN * 4, "the stages hold the block's partial tile");
    static_assert(ROWS % 8 == 0, "the chunk swizzle of a row is the same at its owner");
    static_assert(KIND == PR_RESID || C == 1, "only Wo and down are cut along K");
};

template <int KIND, int BN, int C, int OCC>
__global__ void __launch_bounds__(PS_THREADS, OCC) prompt_split_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
                                                                     const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_x,
                                                                     const PromptParams p) {
    using S = PsShape<KIND, BN, C, OCC>;
    constexpr int STAGES = S::STAGES, CL = S::CL;
    extern __shared__ __align__(1024) unsigned char ps_raw[];
    __shared__ __align__(8) uint64_t full_bar[PS_MAX_STAGES], empty_bar[PS_MAX_STAGES], acc_bar, red_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;
    __shared__ float s_ss[KIND == PR_QKV ? CL : 1][PR_BM];      // q/k/v: the sums of squares of a row's columns in every block of the cluster
    unsigned char* const base = ps_raw;
    float* const red = reinterpret_cast<float*>(base + (size_t)STAGES * S::STAGE);      // [C - 1][R][BN]

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int rank = CL > 1 ? (int)blockIdx.x : 0;     // the cluster spans x
    const int tile = blockIdx.y, m0 = blockIdx.z * PR_BM;
    const int slice = C > 1 ? rank : 0;
    const int base_kb = p.kb_total / C, rem_kb = p.kb_total % C;
    const int kb0 = slice * base_kb + min(slice, rem_kb), nkb = base_kb + (slice < rem_kb ? 1 : 0);
    const int rows = min(PR_BM, p.T - m0);             // tokens of this tile
    const int R = C > 1 ? (((rows + C - 1) / C + 7) & ~7) : PR_BM;      // rows a block owns: [slice R, slice R + R)
    auto rows_of = [&](int owner) { return max(0, min(R, rows - owner * R)); };
    const int my_rows = rows_of(slice);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { pr_mbar_init(&full_bar[s], 1); pr_mbar_init(&empty_bar[s], 1); }
        pr_mbar_init(&acc_bar, 1);
        pr_mbar_init(&red_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (C > 1 && my_rows > 0) pr_expect(&red_bar, (uint32_t)((C - 1) * my_rows * BN * 4));
        abort_flag = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(S::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    pdl_launch();
    if (CL > 1) pr_cluster_arrive();      // (matched before the first remote write: every block of the cluster has set its barriers up by then)

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        int armed = 0;                   // k blocks whose loads have been requested
        const bool one = elect_one();
        if (one) {
            const CUtensorMap* tm_w = &tm_w0;
            int r0 = tile * BN;
            if (KIND == PR_QKV) {        // dims [rank BN / 2, ..) of head `tile` and those 64 further: RoPE's pairs stay in a block
                r0 = tile * HEAD_DIM + rank * (BN / 2);
                if (tile >= Q_HEADS) { tm_w = &tm_w1; r0 -= Q_DIM; }
                if (tile >= Q_HEADS + KV_HEADS) { tm_w = &tm_w2; r0 -= KV_DIM; }
            }
            if (KIND == PR_SILU) r0 = tile * (BN / 2);
            const uint32_t bytes = (uint32_t)p.a_rows * TC_BK * 2 + S::B_BYTES;
            auto weights = [&](int kb, int s) {
                const uint32_t st = tc_smem(base + (size_t)s * S::STAGE) + S::A_BYTES;
                pr_expect(&full_bar[s], bytes);
                tc_load_box(st, tm_w, (kb0 + kb) * TC_BK, r0, &full_bar[s]);
                if (KIND == PR_QKV) tc_load_box(st + S::B_BYTES / 2, tm_w, (kb0 + kb) * TC_BK, r0 + 64, &full_bar[s]);
                if (KIND == PR_SILU) tc_load_box(st + S::B_BYTES / 2, &tm_w1, (kb0 + kb) * TC_BK, r0, &full_bar[s]);
                armed = kb + 1;
            };
            const int ahead = min(nkb, STAGES);
            for (int kb = 0; kb < ahead; ++kb) weights(kb, kb);
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_x) : "memory");
            pdl_wait();
            for (int kb = 0, s = 0, turn = 0; kb < nkb; ++kb, ++s) {
                if (s == STAGES) { s = 0; ++turn; }
                if (turn > 0) {
                    if (!tc_wait(&empty_bar[s], (turn - 1) & 1, &abort_flag, p.status, 60)) break;
                    weights(kb, s);
                }
                tc_load_box(tc_smem(base + (size_t)s * S::STAGE), &tm_x, (kb0 + kb) * TC_BK, m0, &full_bar[s]);
            }
        }
        __syncwarp();
        if (CL > 1) { pr_cluster_wait(); pr_cluster_arrive(); pr_cluster_wait(); }
        else asm volatile("bar.sync 3, 192;" ::: "memory");
        if (one && abort_flag)           // (the last STAGES of them may still be on their way)
            for (int kb = max(0, armed - STAGES); kb < armed; ++kb) tc_drain(&full_bar[kb % STAGES], (kb / STAGES) & 1);
        return;
    }
    if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(PR_BM >> 4) << 24);
            // (descriptors count 16-byte units: a k step of 16 elements is 2 of them)
            const uint64_t da0 = tc_desc(tc_smem(base)), db0 = tc_desc(tc_smem(base) + S::A_BYTES);
            uint64_t ds = 0;
            for (int kb = 0, s = 0, phase = 0; kb < nkb; ++kb, ++s, ds += S::STAGE >> 4) {
                if (s == STAGES) { s = 0; phase ^= 1; ds = 0; }
                if (!tc_wait(&full_bar[s], phase, &abort_flag, p.status, 61)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k) {
                    const uint64_t da = da0 + ds + 2 * k, db = db0 + ds + 2 * k;
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                 ::"r"(tmem_base), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)(kb | k)), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&empty_bar[s])) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&acc_bar)) : "memory");
        }
        __syncwarp();
        if (CL > 1) pr_cluster_wait();
        asm volatile("bar.sync 2, 160;" ::: "memory");              // the epilogue warps have read the accumulator
        if (abort_flag) tc_drain(&acc_bar, 0);                      // ... or gave it up: the products that were issued end first
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::COLS) : "memory");
        if (CL > 1) { pr_cluster_arrive(); pr_cluster_wait(); }
        else asm volatile("bar.sync 3, 192;" ::: "memory");
        return;
    }

    // ---------------------------------------------------------------------- epilogue
    const int te = (int)threadIdx.x - 64, quad = warp & 3;
    const uint32_t tacc = tmem_base + ((uint32_t)(quad * 32) << 16);
    const int row = quad * 32 + lane, trow = m0 + row;  // this thread's accumulator row and its token
    const bool live = row < rows;

    if constexpr (KIND == PR_QKV) {
        // A thread holds BN / 2 dims of a head's row and the BN / 2 that RoPE pairs them with, for the row's scale and norm; then the warp's 32 rows go
        // through shared memory (a stage: every MMA has completed), so that SUBS lanes finish a row and global accesses are runs of 8 SUBS to 16 SUBS bytes
        // (a thread per row all the way: prompts of 128 / 256 / 512 tokens 1002 / 1154 / 1550 us, so 975 / 1079 / 1437).
        constexpr int HALF = BN / 2, SUBS = BN / 8, STEP = 32 / SUBS, RB = SUBS < 8 ? SUBS : 8, LD = BN + 4;   // RB: rows whose RoPE entries are requested together
        const int col0 = tile * HEAD_DIM, d0 = rank * HALF, sub = lane % SUBS, lr0 = lane / SUBS, w0 = m0 + quad * 32, wrows = min(32, rows - quad * 32);
        const bool normed = col0 < Q_DIM + KV_DIM;
        float* const piece = reinterpret_cast<float*>(base) + (size_t)quad * 32 * LD;
        static_assert(STAGES * S::STAGE >= 128 * LD * 4, "the stages hold the rows");
        PrRope rope[RB];
        auto rope_rows = [&](int i0) {
#pragma unroll
            for (int i = 0; i < RB; ++i) rope[i] = pr_rope(p, w0 + max(0, min((i0 + i) * STEP + lr0, wrows - 1)), d0 + sub * 4);
        };
        if (normed && wrows > 0) rope_rows(0);
        const bf16_raw* gp = pr_head_gain(p, col0) + d0 + sub * 4;
        const float4 glo = pr_unpack4(__ldg(reinterpret_cast<const uint2*>(gp))), ghi = pr_unpack4(__ldg(reinterpret_cast<const uint2*>(gp + 64)));
        pdl_wait();
        const float r = live ? pr_scale(p, trow) : 0.f;
        const bool summed = __all_sync(0xffffffffu, tc_wait_warp(&acc_bar, 0, &abort_flag, p.status, 62) && !abort_flag);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // (a whole head's 128 columns are read twice: once for their squares, once to be scaled)
        constexpr bool TWICE = BN > 64;
        uint32_t v[TWICE ? 1 : BN / 32][32];
        float ss4[4] = {0.f, 0.f, 0.f, 0.f};
        auto squares = [&](const uint32_t (&u)[32]) {
#pragma unroll
            for (int j = 0; j < 32; ++j) { const float y = __uint_as_float(u[j]) * r; ss4[j & 3] = fmaf(y, y, ss4[j & 3]); }
        };
        auto read_out = [&]() {                          // the accumulator may go
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("bar.arrive 2, 160;" ::: "memory");
        };
        if constexpr (TWICE) {
            if (normed)
#pragma unroll
                for (int c = 0; c < BN / 32; ++c) {
                    tc_ld32(v[0], tacc + (uint32_t)(c * 32));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    squares(v[0]);
                }
        } else {
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) tc_ld32(v[c], tacc + (uint32_t)(c * 32));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            read_out();
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) squares(v[c]);
        }
        float ss = (ss4[0] + ss4[1]) + (ss4[2] + ss4[3]);
        if (CL > 1) {
            // (a block whose sums are not complete sends NaN: no other passes its rows off as whole)
            if (!summed) ss = __int_as_float(0x7fffffff);
            pr_cluster_wait();
            s_ss[rank][row] = ss;
#pragma unroll
            for (int o = 1; o < CL; ++o)
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(pr_map(tc_smem(&s_ss[rank][row]), (rank + o) % CL)), "f"(ss) : "memory");
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            ss = 0.f;
#pragma unroll
            for (int o = 0; o < CL; ++o) ss += s_ss[o][row];
        }
        const float f = normed ? r * rsqrtf(ss / (float)HEAD_DIM + EPS) : r;
        auto put = [&](const uint32_t (&u)[32], int c) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(piece + lane * LD + c * 32 + j) = make_float4(__uint_as_float(u[j]) * f, __uint_as_float(u[j + 1]) * f, __uint_as_float(u[j + 2]) * f, __uint_as_float(u[j + 3]) * f);
        };
        if constexpr (TWICE) {
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                tc_ld32(v[0], tacc + (uint32_t)(c * 32));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (summed) put(v[0], c);
            }
            read_out();
        }
        if (summed && wrows > 0) {
            if constexpr (!TWICE) {
#pragma unroll
                for (int c = 0; c < BN / 32; ++c) put(v[c], c);
            }
            __syncwarp();
#pragma unroll 1
            for (int i0 = 0; i0 * STEP < wrows; i0 += RB) {
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    const int lr = (i0 + i) * STEP + lr0;
                    if (lr < wrows)
                        pr_finish_head(p, col0, w0 + lr, d0 + sub * 4, *reinterpret_cast<const float4*>(piece + lr * LD + sub * 4),
                                       *reinterpret_cast<const float4*>(piece + lr * LD + HALF + sub * 4), glo, ghi, rope[i]);
                }
                if (normed && (i0 + RB) * STEP < wrows) rope_rows(i0 + RB);
            }
        }
        if (CL == 1) asm volatile("bar.sync 3, 192;" ::: "memory");
        return;
    }
    if constexpr (KIND == PR_SILU) {
        // (through shared memory, for runs of BN bytes in a row: the warp's 32 rows, an odd number of 16-byte units apart)
        constexpr int HALF = BN / 2, STEP = HALF % 16 ? 8 : 16, UNITS = HALF / 8, LD = UNITS | 1;
        uint4* const piece = reinterpret_cast<uint4*>(base) + (size_t)quad * 32 * LD;
        static_assert(STAGES * S::STAGE >= 128 * LD * 16, "the stages hold the rows");
        pdl_wait();
        const float r = live ? pr_scale(p, trow) : 0.f;
        const bool summed = __all_sync(0xffffffffu, tc_wait_warp(&acc_bar, 0, &abort_flag, p.status, 62) && !abort_flag);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int wrows = min(32, rows - quad * 32);
        if (summed && wrows > 0) {
#pragma unroll
            for (int c0 = 0; c0 < HALF; c0 += 3 * STEP) {
                uint32_t g[3][STEP], u[3][STEP];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (c0 + c * STEP < HALF) {
                        if constexpr (STEP == 16) { tc_ld16(g[c], tacc + (uint32_t)(c0 + c * STEP)); tc_ld16(u[c], tacc + (uint32_t)(HALF + c0 + c * STEP)); }
                        else { tc_ld8(g[c], tacc + (uint32_t)(c0 + c * STEP)); tc_ld8(u[c], tacc + (uint32_t)(HALF + c0 + c * STEP)); }
                    }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (c0 + c * STEP < HALF) {
                        uint32_t w[STEP / 2];
#pragma unroll
                        for (int j = 0; j < STEP / 2; ++j)
                            w[j] = pr_pack(pr_silu(__uint_as_float(g[c][2 * j]) * r, __uint_as_float(u[c][2 * j]) * r),
                                           pr_silu(__uint_as_float(g[c][2 * j + 1]) * r, __uint_as_float(u[c][2 * j + 1]) * r));
#pragma unroll
                        for (int j = 0; j < STEP / 8; ++j) piece[lane * LD + (c0 + c * STEP) / 8 + j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                    }
            }
            __syncwarp();
            bf16_raw* const dst = p.hid + (size_t)(m0 + quad * 32) * INTER + tile * HALF;
#pragma unroll 4
            for (int i = lane; i < wrows * UNITS; i += 32) {
                const int lr = i / UNITS, j = i - lr * UNITS;
                *reinterpret_cast<uint4*>(dst + (size_t)lr * INTER + j * 8) = piece[lr * LD + j];
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("bar.arrive 2, 160;" ::: "memory");
        asm volatile("bar.sync 3, 192;" ::: "memory");
        return;
    }
    if constexpr (KIND == PR_RESID) {
    constexpr int SUBS = BN / 4, STEP = 128 / SUBS;     // lanes a row (a chunk of 16 bytes each), rows the four warps take at a time
    constexpr int PER = (S::ROWS + STEP - 1) / STEP;    // rows a thread has a chunk of
    const int sub = te % SUBS, lr0 = te / SUBS;
    const int t0 = m0 + slice * R;                      // first owned token
    float4 xr[PER];
    pdl_wait();
    // while the products run: the residual they are added to
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int lr = i * STEP + lr0;
        xr[i] = lr < my_rows ? *reinterpret_cast<const float4*>(p.x + (size_t)(t0 + lr) * HIDDEN + tile * BN + sub * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // (the MMA thread commits to acc_bar after a wait of its own gave up, too, so that its products can be drained: the flag tells)
    const bool summed = __all_sync(0xffffffffu, tc_wait_warp(&acc_bar, 0, &abort_flag, p.status, 62) && !abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // the partial tile, a thread per token row (the stages are free: every MMA has completed)
    if (summed && quad * 32 < rows) {
        unsigned char* dst = base + (size_t)row * BN * 4;
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {
            uint32_t r[32];
            tc_ld32(r, tacc + (uint32_t)c0);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 8; ++j)
                *reinterpret_cast<uint4*>(dst + (((c0 / 4 + j) ^ (row & 7)) << 4)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (C > 1) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.arrive 2, 160;" ::: "memory");
    if (C > 1) pr_cluster_wait();                       // every block of the cluster has set its mbarriers up
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const bool whole = !abort_flag;                     // no warp of this block gave up on the accumulator
    bool received = whole;
    if (C > 1) {
        if (whole && te < C && te != slice && rows_of(te) > 0) {
            const int slot = slice < te ? slice : slice - 1;
            const uint32_t src = tc_smem(base) + (uint32_t)(te * R * BN * 4);
            asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(pr_map(tc_smem(red) + (uint32_t)(slot * R * BN * 4), te)), "r"(src), "r"((uint32_t)(rows_of(te) * BN * 4)), "r"(pr_map(tc_smem(&red_bar), te)) : "memory");
        }
        __syncwarp();
        received = my_rows > 0 && whole && tc_wait_warp(&red_bar, 0, &abort_flag, p.status, 63, PS_RED_WAIT_NS);
    }

    // 16-byte chunk `j` of owned row `lr`, the slices added in order
    auto sum = [&](int lr, int j) {
        const uint32_t off = (uint32_t)(lr * BN * 4) + (uint32_t)((j ^ (lr & 7)) << 4);
        float4 v;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const unsigned char* src = c == slice ? base + (size_t)slice * R * BN * 4 : reinterpret_cast<unsigned char*>(red) + (size_t)(c < slice ? c : c - 1) * R * BN * 4;
            const float4 u = *reinterpret_cast<const float4*>(src + off);
            v = c ? pr_add(v, u) : u;
        }
        return v;
    };
    if (received) {
        const float4 g = pr_unpack4(*reinterpret_cast<const uint2*>(p.gain + tile * BN + sub * 4));
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            if (i * STEP + (te & ~31) / SUBS >= my_rows) break;     // (the same for the whole warp)
            const int lr = i * STEP + lr0, lc = min(lr, my_rows - 1), t = t0 + lr;
            const float4 x = pr_add(xr[i], sum(lc, sub));
            float ss = pr_dot(x, x);
#pragma unroll
            for (int o = SUBS / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lr < my_rows) {
                const size_t o = (size_t)t * HIDDEN + tile * BN + sub * 4;
                *reinterpret_cast<float4*>(p.x + o) = x;
                *reinterpret_cast<uint2*>(p.xn + o) = pr_pack4(pr_mul(x, g));
                if (sub == 0) p.ssq_out[(size_t)tile * p.ssq_ld + t] = ss;
            }
        }
    }
    if (C > 1) {
        pr_cluster_arrive();      // (matched before the exit: this block's copies have been counted by their receivers or given up)
        pr_cluster_wait();
        if (my_rows > 0 && !received && te == 0) tc_drain(&red_bar, 0);
    } else {
        asm volatile("bar.sync 3, 192;" ::: "memory");
    }
    }
}

// ------------------------------------------------------------------------------------------------------------------------------
// Long prompts: 256 tokens x BN weight rows on a PAIR of SMs (cta_group::2).  Each block of the pair loads its own 128 token rows and half of
// the weight rows; the tensor cores of both read both halves, so a multiply-add costs each SM two thirds of the shared-memory
// traffic and of the bytes from L2 that a 128 x 256 tile on one SM costs it.
//
// Persistent: the pairs walk the items (token tile, weight tile); the TMA ring never drains between items, two accumulators
// (2 x BN columns of TMEM) let the eight epilogue warps finish item i while the products of item i + 1 run.  One thread of the first
// block issues every product; commits reach both blocks' barriers.
//
// An epilogue warp takes its 32 rows 64 columns at a time through a piece of shared memory of its own: written a thread per row
// (where the row's scale and a head's norm are), read half a row per eight or sixteen lanes, so that global accesses are runs of 64 to
// 256 bytes.
//
// A wait that gives up ends the loops of its block; the peer's waits give up too.  The loads of both blocks are counted on the first one's
// barriers: it drains them, and the products, between its own last barrier and the pair's.
// ------------------------------------------------------------------------------------------------------------------------------
constexpr int PP_EPI_WARPS = 8;
constexpr int PP_THREADS = 64 + 32 * PP_EPI_WARPS;   // warp 0: TMA, warp 1: MMA and TMEM, warps 2..9: epilogue (two per TMEM quadrant, half the columns each)
constexpr int PP_MAX_STAGES = 8;
constexpr int PP_LD = 68;                            // floats a row takes in a warp's piece: 64 and padding against bank conflicts
constexpr uint32_t PP_PIECE = 32 * PP_LD * 4;

template <int BN> struct PpShape {
    static constexpr uint32_t A_BYTES = PR_BM * TC_BK * 2, B_BYTES = BN / 2 * TC_BK * 2, STAGE = A_BYTES + B_BYTES;
    static constexpr uint32_t PIECES = PP_EPI_WARPS * PP_PIECE;
    static constexpr int STAGES = (225 * 1024 - PIECES) / STAGE < PP_MAX_STAGES ? (225 * 1024 - PIECES) / STAGE : PP_MAX_STAGES;
    static constexpr size_t SMEM = STAGES * STAGE + PIECES;
    static constexpr uint32_t COLS = BN <= 128 ? 256 : 512;      // TMEM columns: two accumulators, a power of two
};

__device__ __forceinline__ void pp_load_box(uint32_t dst, const void* map, int k, int row, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(k), "r"(row), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ void pp_commit(uint64_t* bar) {   // arrives at the same barrier of both blocks
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(tc_smem(bar)), "h"((unsigned short)3) : "memory");
}

template <int KIND, int BN>
__global__ void __launch_bounds__(PP_THREADS, 1) prompt_pair_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
                                                                    const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_x,
                                                                    const PromptParams p) {
    using S = PpShape<BN>;
    constexpr int STAGES = S::STAGES;
    extern __shared__ __align__(1024) unsigned char pp_raw[];
    __shared__ __align__(8) uint64_t full_bar[PP_MAX_STAGES], empty_bar[PP_MAX_STAGES], acc_full[2], acc_empty[2], drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ int armed_s;
    __shared__ volatile int abort_flag;
    unsigned char* const base = pp_raw;

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { pr_mbar_init(&full_bar[s], 1); pr_mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { pr_mbar_init(&acc_full[b], 1); pr_mbar_init(&acc_empty[b], 2 * PP_EPI_WARPS); }
        pr_mbar_init(&drain_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(S::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pr_cluster_arrive();
    pr_cluster_wait();            // both blocks' barriers and columns are set up
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    pdl_launch();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            // (one thread's instructions are a serial chain: whatever does not change from stage to stage is computed once an item)
            const CUtensorMap* tm_w = &tm_w0;
            int r0 = 0, m0 = 0;
            auto decode = [&](int item) {
                const int tile = item % p.n_tiles;
                m0 = (item / p.n_tiles) * 2 * PR_BM + rank * PR_BM;
                r0 = tile * BN + rank * (BN / 2);
                if (KIND == PR_QKV) {
                    tm_w = &tm_w0;
                    if (tile >= Q_DIM / BN) { tm_w = &tm_w1; r0 -= Q_DIM; }
                    if (tile >= (Q_DIM + KV_DIM) / BN) { tm_w = &tm_w2; r0 -= KV_DIM; }
                }
                if (KIND == PR_SILU) { tm_w = rank ? &tm_w1 : &tm_w0; r0 = tile * (BN / 2); }   // columns [0, BN / 2): gate, the rest: up
            };
            const uint32_t bar0 = pr_map(tc_smem(&full_bar[0]), 0), st0 = tc_smem(base);
            uint32_t bar = bar0, st = st0;                   // the slot's barrier in the first block, its stage in this one
            auto weights = [&](int kb, int s) {
                if (rank == 0) pr_expect(&full_bar[s], 2 * S::STAGE);                            // both blocks' loads
                pp_load_box(st + S::A_BYTES, tm_w, kb * TC_BK, r0, bar);
            };
            int armed = 0;                                   // k blocks whose loads have been requested
            const int ahead = min(p.kb_total, STAGES);       // the first ring's weights before the wait
            decode(pair);
            for (int kb = 0; kb < ahead; ++kb, bar += 8, st += S::STAGE) weights(kb, kb);
            armed = ahead;
            pdl_wait();
            bar = bar0; st = st0;
            int s = 0, turn = 0;
            bool ok = true;
            for (int item = pair; item < p.n_items && ok; item += n_pairs) {
                if (item != pair) decode(item);
                for (int kb = 0; kb < p.kb_total; ++kb, ++s, bar += 8, st += S::STAGE) {
                    if (s == STAGES) { s = 0; ++turn; bar = bar0; st = st0; }
                    if (turn > 0) {
                        if (!tc_wait(&empty_bar[s], (turn - 1) & 1, &abort_flag, p.status, 65)) { ok = false; break; }
                        weights(kb, s);
                        ++armed;
                    } else if (kb >= ahead || item != pair) {
                        weights(kb, s);
                        ++armed;
                    }
                    pp_load_box(st, &tm_x, kb * TC_BK, m0, bar);
                }
            }
            armed_s = armed;
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer: the first block's, for both
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(2 * PR_BM >> 4) << 24);
            const uint64_t da0 = tc_desc(tc_smem(base)), db0 = tc_desc(tc_smem(base) + S::A_BYTES);
            uint64_t ds = 0;
            int s = 0, phase = 0, li = 0;
            bool ok = true;
            for (int item = pair; item < p.n_items && ok; item += n_pairs, ++li) {
                const int acc = li & 1;
                if (li >= 2) ok = tc_wait(&acc_empty[acc], ((li >> 1) - 1) & 1, &abort_flag, p.status, 66);   // its previous tenant was read out by both blocks
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < p.kb_total && ok; ++kb, ++s, ds += S::STAGE >> 4) {
                    if (s == STAGES) { s = 0; phase ^= 1; ds = 0; }
                    ok = tc_wait(&full_bar[s], phase, &abort_flag, p.status, 67);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k) {
                        const uint64_t da = da0 + ds + 2 * k, db = db0 + ds + 2 * k;
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                                     ::"r"(tmem_base + (uint32_t)(acc * BN)), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)(kb | k)) : "memory");
                    }
                    pp_commit(&empty_bar[s]);
                }
                if (ok) pp_commit(&acc_full[acc]);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quad = warp & 3, half = (warp - 2) >> 2;
        float* const piece = reinterpret_cast<float*>(base + (size_t)STAGES * S::STAGE + (size_t)(warp - 2) * PP_PIECE);
        const uint32_t trow = tmem_base + ((uint32_t)(quad * 32) << 16);
        pdl_wait();
        int li = 0;
        for (int item = pair; item < p.n_items; item += n_pairs, ++li) {
            const int tile = item % p.n_tiles, acc = li & 1;
            const int m0 = (item / p.n_tiles) * 2 * PR_BM + rank * PR_BM + quad * 32;     // this warp's first token
            const int rows = min(32, p.T - m0);                                           // (may be zero or less)
            float r = 0.f;
            constexpr int SUBS = KIND == PR_RESID ? 16 : 8, STEP = 32 / SUBS;             // lanes a row, rows an instruction
            const int sub = lane % SUBS, lr0 = lane / SUBS;
            float4 xr[KIND == PR_RESID ? 16 : 1];
            PrRope rope[KIND == PR_QKV ? 4 : 1];          // four rows' entries at a time
            auto rope_rows = [&](int i0, int c) {
#pragma unroll
                for (int i = 0; i < 4; ++i) rope[KIND == PR_QKV ? i : 0] = pr_rope(p, m0 + max(0, min(lr0 + STEP * (i0 + i), rows - 1)), c * 32 + sub * 4);
            };
            if (KIND != PR_RESID) {
                if (lane < rows) r = pr_scale(p, m0 + lane);
                if (KIND == PR_QKV && rows > 0) rope_rows(0, 0);
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int lr = lr0 + STEP * i;
                    xr[i] = lr < rows ? *reinterpret_cast<const float4*>(p.x + (size_t)(m0 + lr) * HIDDEN + tile * BN + half * 64 + sub * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            if (!tc_wait_warp(&acc_full[acc], (li >> 1) & 1, &abort_flag, p.status, 68)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tacc = trow + (uint32_t)(acc * BN);
            if (rows > 0) {
                if constexpr (KIND == PR_QKV) {
                    static_assert(KIND != PR_QKV || BN == 256, "a head a warp");
                    const int col0 = tile * BN + half * HEAD_DIM;
                    uint32_t v[4][32];                  // the head: every column of the row under one wait
#pragma unroll
                    for (int c = 0; c < 4; ++c) tc_ld32(v[c], tacc + (uint32_t)(half * 128 + c * 32));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float f = r;
                    if (col0 < Q_DIM + KV_DIM) {
                        float ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                        for (int j = 0; j < 32; ++j)
#pragma unroll
                            for (int c = 0; c < 4; ++c) { const float y = __uint_as_float(v[c][j]) * r; ss[c] = fmaf(y, y, ss[c]); }
                        f = r * rsqrtf(((ss[0] + ss[1]) + (ss[2] + ss[3])) / (float)HEAD_DIM + EPS);
                    }
                    const bf16_raw* gp = pr_head_gain(p, col0);
#pragma unroll
                    for (int c = 0; c < 2; ++c) {       // dims [32 c, 32 c + 32) and their partners 64 further
                        __syncwarp();                   // the piece's previous contents have been read
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            *reinterpret_cast<float4*>(piece + lane * PP_LD + 4 * j) = make_float4(__uint_as_float(v[c][4 * j]) * f, __uint_as_float(v[c][4 * j + 1]) * f, __uint_as_float(v[c][4 * j + 2]) * f, __uint_as_float(v[c][4 * j + 3]) * f);
                            *reinterpret_cast<float4*>(piece + lane * PP_LD + 32 + 4 * j) = make_float4(__uint_as_float(v[2 + c][4 * j]) * f, __uint_as_float(v[2 + c][4 * j + 1]) * f, __uint_as_float(v[2 + c][4 * j + 2]) * f, __uint_as_float(v[2 + c][4 * j + 3]) * f);
                        }
                        __syncwarp();
                        const int d = c * 32 + sub * 4;
                        const float4 glo = pr_unpack4(__ldg(reinterpret_cast<const uint2*>(gp + d))), ghi = pr_unpack4(__ldg(reinterpret_cast<const uint2*>(gp + 64 + d)));
#pragma unroll
                        for (int i0 = 0; i0 < 8; i0 += 4) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int lr = lr0 + STEP * (i0 + i);
                                if (lr < rows)
                                    pr_finish_head(p, col0, m0 + lr, d, *reinterpret_cast<const float4*>(piece + lr * PP_LD + sub * 4),
                                                   *reinterpret_cast<const float4*>(piece + lr * PP_LD + 32 + sub * 4), glo, ghi, rope[i]);
                            }
                            if (c == 0 || i0 == 0) rope_rows(i0 ? 0 : 4, i0 ? 1 : c);
                        }
                    }
                } else if constexpr (KIND == PR_RESID) {
                    static_assert(KIND != PR_RESID || BN == 128, "64 columns a warp");
                    uint32_t a[32], b[32];
                    tc_ld32(a, tacc + (uint32_t)(half * 64));
                    tc_ld32(b, tacc + (uint32_t)(half * 64 + 32));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        *reinterpret_cast<uint4*>(piece + lane * PP_LD + 4 * j) = make_uint4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]);
                        *reinterpret_cast<uint4*>(piece + lane * PP_LD + 32 + 4 * j) = make_uint4(b[4 * j], b[4 * j + 1], b[4 * j + 2], b[4 * j + 3]);
                    }
                    __syncwarp();
                    const int col = tile * BN + half * 64 + sub * 4;
                    const float4 g = pr_unpack4(*reinterpret_cast<const uint2*>(p.gain + col));
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int lr = lr0 + STEP * i;
                        const float4 x = pr_add(xr[i], *reinterpret_cast<const float4*>(piece + lr * PP_LD + sub * 4));
                        float ss = pr_dot(x, x);
#pragma unroll
                        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                        if (lr < rows) {
                            const size_t o = (size_t)(m0 + lr) * HIDDEN + col;
                            *reinterpret_cast<float4*>(p.x + o) = x;
                            *reinterpret_cast<uint2*>(p.xn + o) = pr_pack4(pr_mul(x, g));
                            if (sub == 0) p.ssq_out[(size_t)(tile * 2 + half) * p.ssq_ld + m0 + lr] = ss;
                        }
                    }
                } else if constexpr (BN == 256) {
                    uint32_t g[2][32], u[2][32], out[32];   // 64 columns of this lane's row, under one wait
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        tc_ld32(g[c], tacc + (uint32_t)(half * 64 + c * 32));
                        tc_ld32(u[c], tacc + (uint32_t)(BN / 2 + half * 64 + c * 32));
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            out[c * 16 + j] = pr_pack(pr_silu(__uint_as_float(g[c][2 * j]) * r, __uint_as_float(u[c][2 * j]) * r),
                                                      pr_silu(__uint_as_float(g[c][2 * j + 1]) * r, __uint_as_float(u[c][2 * j + 1]) * r));
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<uint4*>(piece + lane * PP_LD + 4 * j) = make_uint4(out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {       // eight lanes a row of 128 bytes
                        const int lr = lr0 + STEP * i;
                        if (lr < rows)
                            *reinterpret_cast<uint4*>(p.hid + (size_t)(m0 + lr) * INTER + tile * (BN / 2) + half * 64 + sub * 8) = *reinterpret_cast<const uint4*>(piece + lr * PP_LD + sub * 4);
                    }
                } else {
                    static_assert(BN == 192, "a warp reads 64 gate and 64 up columns, or 48");
                    constexpr int HC = BN / 4, UNITS = HC / 8;   // gate and up columns a warp, 16-byte units of a row's output
                    uint32_t g[2][32], u[2][32], out[32];        // of this lane's row, under one wait
                    const uint32_t tg = tacc + (uint32_t)(half * HC), tu = tg + (uint32_t)(BN / 2);
                    tc_ld32(g[0], tg);
                    tc_ld32(u[0], tu);
                    tc_ld16(g[1], tg + 32u);
                    tc_ld16(u[1], tu + 32u);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < HC / 2; ++j) {
                        const int c = j >> 4, k = 2 * (j & 15);
                        out[j] = pr_pack(pr_silu(__uint_as_float(g[c][k]) * r, __uint_as_float(u[c][k]) * r), pr_silu(__uint_as_float(g[c][k + 1]) * r, __uint_as_float(u[c][k + 1]) * r));
                    }
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < UNITS; ++j)
                        *reinterpret_cast<uint4*>(piece + lane * PP_LD + 4 * j) = make_uint4(out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
                    __syncwarp();
                    bf16_raw* const dst = p.hid + (size_t)m0 * INTER + tile * (BN / 2) + half * HC;
#pragma unroll
                    for (int i = 0; i < UNITS; ++i) {   // six lanes a row of 96 bytes
                        const int at = i * 32 + lane, lr = at / UNITS, j = at - lr * UNITS;
                        if (lr < rows) *reinterpret_cast<uint4*>(dst + (size_t)lr * INTER + j * 8) = *reinterpret_cast<const uint4*>(piece + lr * PP_LD + j * 4);
                    }
                }
            }
            // this accumulator may be overwritten by the item after next
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(pr_map(tc_smem(&acc_empty[acc]), 0)) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // After a wait gave up (nobody of this block waits any more, so the flag is what it will be): the loads land and the products end before the pair's
    // columns and memory go.
    if (warp < 2 && rank == 0 && abort_flag && elect_one()) {
        if (warp == 0) {
            for (int k = max(0, armed_s - STAGES); k < armed_s; ++k) tc_drain(&full_bar[k % STAGES], (k / STAGES) & 1);
        } else {
            asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&drain_bar)) : "memory");
            tc_drain(&drain_bar, 0);
        }
    }
    __syncwarp();
    pr_cluster_arrive();
    pr_cluster_wait();            // nothing of the pair is under way to this block any more
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::COLS) : "memory");
    }
}

// ---- embedding gather: a block per token -------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) prompt_embed_kernel(const long long* __restrict__ ids, const bf16_raw* __restrict__ embed, int vocab, float* __restrict__ x,
                                                           const bf16_raw* __restrict__ gain, bf16_raw* __restrict__ xn, float* __restrict__ ssq, int ssq_ld,
                                                           uint32_t* status) {
    pdl_launch();
    pdl_wait();
    const int b = blockIdx.x, tid = threadIdx.x;
    long long t = ids[b];
    if (t < 0 || t >= vocab) {
        if (tid == 0) report(status, ST_BAD_TOKEN, 0, (uint32_t)t);
        t = 0;
    }
    const float4 v = pr_unpack4(reinterpret_cast<const uint2*>(embed + (size_t)t * HIDDEN)[tid]), g = pr_unpack4(reinterpret_cast<const uint2*>(gain)[tid]);
    reinterpret_cast<float4*>(x + (size_t)b * HIDDEN)[tid] = v;
    reinterpret_cast<uint2*>(xn + (size_t)b * HIDDEN)[tid] = pr_pack4(pr_mul(v, g));
    float ss = pr_dot(v, v);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 15) == 0) ssq[(size_t)(tid >> 4) * ssq_ld + b] = ss;
}

cudaError_t launch_prompt_embed(const long long* ids, const bf16_raw* embed, int vocab, float* x, const bf16_raw* gain, bf16_raw* xn, float* ssq, int ssq_ld,
                                uint32_t* status, int T, cudaStream_t st) {
    return launch_chain(prompt_embed_kernel, dim3(T), dim3(256), 0, st, ids, embed, vocab, x, gain, xn, ssq, ssq_ld, status);
}

// ---- host side ---------------------------------------------------------------------------------------------------------------
template <typename K>
static cudaError_t pr_prepare(K kernel, size_t smem, bool (&done)[64]) {   // (a benign race between host threads: the same value is written)
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) done[dev] = true;
    return e;
}

template <int KIND, int BN, int C, int OCC>
static cudaError_t launch_split(const CUtensorMap* tw, const CUtensorMap& tx, const PromptParams& p, cudaStream_t st) {
    using S = PsShape<KIND, BN, C, OCC>;
    static bool done[64] = {};
    cudaError_t e = pr_prepare(prompt_split_kernel<KIND, BN, C, OCC>, S::SMEM, done);
    if (e != cudaSuccess) return e;
    constexpr int tiles = KIND == PR_QKV ? QKV_DIM / HEAD_DIM : KIND == PR_RESID ? HIDDEN / BN : 2 * INTER / BN;
    const dim3 grid(S::CL, tiles, (p.T + PR_BM - 1) / PR_BM);
    if constexpr (S::CL == 1) return launch_chain(prompt_split_kernel<KIND, BN, C, OCC>, grid, dim3(PS_THREADS), S::SMEM, st, tw[0], tw[1], tw[2], tx, p);
    else return launch_chain_cluster(prompt_split_kernel<KIND, BN, C, OCC>, grid, dim3(PS_THREADS), S::SMEM, S::CL, st, tw[0], tw[1], tw[2], tx, p);
}

template <int KIND, int BN>
static cudaError_t launch_pair(const CUtensorMap* tw, const CUtensorMap& tx, PromptParams p, int sm_count, cudaStream_t st) {
    using S = PpShape<BN>;
    static bool done[64] = {};
    cudaError_t e = pr_prepare(prompt_pair_kernel<KIND, BN>, S::SMEM, done);
    if (e != cudaSuccess) return e;
    p.n_tiles = KIND == PR_QKV ? QKV_DIM / BN : KIND == PR_RESID ? HIDDEN / BN : 2 * INTER / BN;
    p.n_items = p.n_tiles * ((p.T + 2 * PR_BM - 1) / (2 * PR_BM));
    const int pairs = p.n_items < sm_count / 2 ? p.n_items : sm_count / 2;
    return launch_chain_cluster(prompt_pair_kernel<KIND, BN>, dim3(2 * pairs), dim3(PP_THREADS), S::SMEM, 2, st, tw[0], tw[1], tw[2], tx, p);
}

cudaError_t launch_prompt_gemm(const PromptGemmCall& c, cudaStream_t st) {
    if (c.T < 1 || c.K % TC_BK || c.K < 8 * TC_BK || c.ssq_ld < c.T) return cudaErrorInvalidValue;
    PromptParams p{};
    p.a_rows = prompt_box_rows(c.T);
    p.T = c.T; p.kb_total = c.K / TC_BK; p.ssq_ld = c.ssq_ld; p.ssq_in = c.ssq; p.ssq_out = c.ssq;
    p.q_hi = c.q_hi; p.q_lo = c.q_lo; p.qkv = c.qkv; p.kc = c.kc; p.vc = c.vc; p.qn = c.qn; p.kn = c.kn; p.rope = c.rope;
    p.x = c.x; p.xn = c.xn; p.gain = c.gain; p.hid = c.hid; p.status = c.status;
    const int sm = tc_sm_count();
    if (sm < 2) return cudaErrorInvalidDevice;
    const int mt = (c.T + PR_BM - 1) / PR_BM;
    // The shape by the number of 128-token tiles: about one block an SM while tiles are narrow enough for that, then two an SM, then pairs.
    // Measured, us a prompt with every product as below but for one (128-row columns / slices / blocks an SM; 0: the pair kernel):
    //   q/k/v    128 tokens 32//1 970, 32//2 1010, 64//1 1007;  256: 64//1 1099, 32//2 1099, 64//2 1108;  300: 64//2 1292, 128//1 1316;  512: 64//2 1388, 128//1
    //            1411;  640: 128//2 1750, 0 1807, 64//2 1865;  1000: 2030, 0 2080;  1150: 2092, 0 2333;  1290: 0 2456, 128//2 2502
    //   gate/up  64 tokens 48//2 917, 48//1 933;  128: 970, 977, 96//1 1007;  256: 96//1 1101, 48//2 1098;  300: 128//1 1292, 192//1 1346;  512: 192//1 1388, 96//2
    //            1393, 0 1437;  520: 128//2 1733, 0 1742;  777: 0 1952, 192//1 1967;  1290: 0 2454, 128//2 2571
    //   Wo, down 64 tokens 32/8/2 917, 32/4/1 938;  128: 970, 972, 64/4/1 1032;  256: 64/4/1 1099, 32/4/2 1169;  300: 64/4/2 1292, 64/2/1 1306;  512: 1388, 1416;
    //            640: 64/2/2 1772, 0 1964;  1150: 64/2/2 2096, 0 2201;  1290: 0 2455, 64/1/2 2588
    const bool pair = mt > (c.kind == PR_SILU ? 4 : 9);
    const int bn = c.kind == PR_QKV ? (mt == 1 ? 32 : mt <= 4 ? 64 : 128) : c.kind == PR_RESID ? (mt == 1 ? 32 : 64) : mt == 1 ? 48 : mt == 2 ? 96 : mt == 3 ? 128 : 192;
    const int rows[3] = {c.kind == PR_QKV ? Q_DIM : c.kind == PR_RESID ? HIDDEN : INTER, c.kind == PR_QKV ? KV_DIM : INTER, KV_DIM};
    const int n_w = c.kind == PR_QKV ? 3 : c.kind == PR_RESID ? 1 : 2;
    // gate/up on pairs of SMs: items of 192 columns where their rounds are shorter than those of 256 by more than an eighth, which the products show: 769 to
    // 1024 tokens on 148 SMs (us a prompt, 256 / 192: 800 tokens 1868 / 1845, 1000 1995 / 1944; one round of 256, 640, 1656 / 1770; 1100 2020 / 2068; 1400 2520 / 2561).
    // Where the rounds are shorter by less, both take the same: 2320 3995 / 3954, 2400 4238 / 4190, 2560 4401 / 4413, 2700 4690 / 4717, 4000 6994 / 6957 (runs of one side 80 apart).
    const int pairs = sm / 2, mt2 = (mt + 1) / 2, rounds256 = (mt2 * (2 * INTER / 256) + pairs - 1) / pairs, rounds192 = (mt2 * (2 * INTER / 192) + pairs - 1) / pairs;
    const bool finer = c.kind == PR_SILU && rounds192 * 192 * 8 < rounds256 * 256 * 7;
    const uint32_t box = pair ? (c.kind == PR_RESID ? 64u : finer ? 96u : 128u) : c.kind == PR_RESID ? (uint32_t)bn : (uint32_t)bn / 2;
    CUtensorMap tw[3];
    for (int i = 0; i < 3; ++i) {
        if (i >= n_w) tw[i] = tw[0];
        else if (!tc_cached_map(c.w[i], (uint64_t)rows[i], (uint64_t)c.K, box, &tw[i])) return cudaErrorUnknown;
    }
    p.ssq_parts = *c.parts;
    if (c.kind == PR_RESID) *c.parts = pair ? HIDDEN / 64 : HIDDEN / bn;
    switch (c.kind) {
        case PR_QKV:
            if (pair) return launch_pair<PR_QKV, 256>(tw, *c.in, p, sm, st);
            if (mt == 1) return launch_split<PR_QKV, 32, 1, 1>(tw, *c.in, p, st);
            if (mt == 2) return launch_split<PR_QKV, 64, 1, 1>(tw, *c.in, p, st);
            if (mt <= 4) return launch_split<PR_QKV, 64, 1, 2>(tw, *c.in, p, st);
            return launch_split<PR_QKV, 128, 1, 2>(tw, *c.in, p, st);
        case PR_RESID:
            if (pair) return launch_pair<PR_RESID, 128>(tw, *c.in, p, sm, st);
            if (mt == 1) return launch_split<PR_RESID, 32, 8, 2>(tw, *c.in, p, st);
            if (mt == 2) return launch_split<PR_RESID, 64, 4, 1>(tw, *c.in, p, st);
            if (mt <= 4) return launch_split<PR_RESID, 64, 4, 2>(tw, *c.in, p, st);
            return launch_split<PR_RESID, 64, 2, 2>(tw, *c.in, p, st);
        case PR_SILU:
            if (pair) return finer ? launch_pair<PR_SILU, 192>(tw, *c.in, p, sm, st) : launch_pair<PR_SILU, 256>(tw, *c.in, p, sm, st);
            if (mt == 1) return launch_split<PR_SILU, 48, 1, 2>(tw, *c.in, p, st);
            if (mt == 2) return launch_split<PR_SILU, 96, 1, 1>(tw, *c.in, p, st);
            if (mt == 3) return launch_split<PR_SILU, 128, 1, 1>(tw, *c.in, p, st);
            return launch_split<PR_SILU, 192, 1, 1>(tw, *c.in, p, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace q3
