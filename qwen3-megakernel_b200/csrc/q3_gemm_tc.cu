// Tensor-core GEMM for decode batches of more than 64 sequences and for q3_linear_tc: out[t, n] (+)= sum_k W[n, k] * X[t, k]; and the
// LM head of smaller decode batches.  (A prompt's products: q3_prompt.cu.)
//
// Blackwell path: TMA (cp.async.bulk.tensor, 128-byte swizzle) stages W and X tiles in shared memory,
// one elected thread issues tcgen05.mma (kind::f16, bf16 operands, fp32 accumulator in TMEM), four
// warps read the accumulator back with tcgen05.ld and store it.  The weight matrix is the M operand
// (128 weight rows per tile) and the tokens are the N operand, so a decode batch of 32..256 tokens is
// one N tile and every weight byte crosses HBM once.
//
// Exact activations: the fp32 activations are passed as up to three bf16 planes (hi, mid, lo with
// X = hi + mid + lo); each W tile is multiplied with every plane into the same accumulator.  With
// three planes the result equals the fp32 product of the bf16 weights up to accumulation order;
// large-batch decode uses that (the extra MMAs are free while the weights stream from HBM).
#include <cuda.h>

#include <mutex>
#include <vector>

#include "q3_engine.h"
#include "q3_gemm_tc.h"
#include "q3_tc_ptx.cuh"

namespace q3 {

constexpr int MAX_DEVICES = 64;
static std::mutex& host_lock() { static std::mutex m; return m; }   // guards the per-device set-up flags and the tensor-map cache

constexpr int TC_THREADS = 192;    // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2..5: epilogue
constexpr int TC_BM = 128;         // weight rows per tile (UMMA M)

template <int BN>
__global__ void __launch_bounds__(TC_THREADS, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tm_w0,
                                                                const __grid_constant__ CUtensorMap tm_w1,
                                                                const __grid_constant__ CUtensorMap tm_w2,
                                                                const __grid_constant__ CUtensorMap tm_x, const GemmTcParams p) {
    extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[8], empty_bar[8], acc_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    // which weight matrix this tile belongs to (grouped launches), and its first row inside that matrix
    int grp = 0, tile = blockIdx.x;
    if (p.n_groups > 1) {
        if (tile >= p.g_tiles[0]) { tile -= p.g_tiles[0]; grp = 1; }
        if (grp == 1 && p.n_groups > 2 && tile >= p.g_tiles[1]) { tile -= p.g_tiles[1]; grp = 2; }
    }
    const CUtensorMap* tm_w = grp == 0 ? &tm_w0 : (grp == 1 ? &tm_w1 : &tm_w2);
    float* const out = p.n_groups > 1 ? (grp == 0 ? p.g_out[0] : grp == 1 ? p.g_out[1] : p.g_out[2]) : p.out;
    const int ldo = p.n_groups > 1 ? (grp == 0 ? p.g_ldo[0] : grp == 1 ? p.g_ldo[1] : p.g_ldo[2]) : p.ldo;
    const int n_rows = p.n_groups > 1 ? (grp == 0 ? p.g_tiles[0] : grp == 1 ? p.g_tiles[1] : p.g_tiles[2]) * TC_BM : p.n_rows;
    const int m0 = tile * TC_BM;                // first weight row of this tile
    const int n0 = blockIdx.y * BN;             // first token of this tile
    // split-K: grid.z slices of the k blocks; partial tiles are added into `out` with fp32 atomics
    const int kb_begin = blockIdx.z * p.kb_per_split;
    const int nkb = min(p.K / TC_BK - kb_begin, p.kb_per_split);
    const int nsplit = p.nsplit;
    const uint32_t a_bytes = TC_BM * TC_BK * 2, b_bytes = BN * TC_BK * 2;
    const uint32_t stage_bytes = a_bytes + nsplit * b_bytes;
    const int stages = p.stages;
    // 1024-byte aligned base (the swizzle pattern repeats every 1024 bytes)
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&full_bar[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&empty_bar[s])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&acc_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
    }
    // The planes of a stage lie one after the other in shared memory, each BN rows of 128 bytes: up to 256 rows they are
    // ONE B operand of nsplit * BN columns, so a k step is one tcgen05.mma instead of nsplit (an instruction costs about 150
    // clocks here whatever its N), and the epilogue adds the planes' column groups.  Beyond 256 columns: one MMA per plane
    // into the same BN columns.
    const bool wide = nsplit > 1 && nsplit * BN <= 256;
    const uint32_t tmem_cols = wide ? (nsplit * BN <= 128 ? 128u : 256u) : (uint32_t)(BN < 32 ? 32 : BN);
    if (warp == 1) {   // TMEM allocation: one warp, power-of-two column count >= 32
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    // Barriers and the accumulator are set up.  The successor may start its own set-up now; this kernel waits for its
    // predecessor only where it first touches what that one produced: the weights are nobody's output, so their tiles
    // are requested BEFORE the wait (their HBM latency overlaps the predecessor's tail), the activation planes and
    // the output stores come after it.
    pdl_launch();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            const int ahead = min(nkb, stages);   // the first ring of stages: weight tiles before the wait
            for (int kb = 0; kb < ahead; ++kb) {
                unsigned char* st = base + (size_t)kb * stage_bytes;
                asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&full_bar[kb])), "r"(stage_bytes) : "memory");
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                             ::"r"(tc_smem(st)), "l"(tm_w), "r"((kb_begin + kb) * TC_BK), "r"(m0), "r"(tc_smem(&full_bar[kb])) : "memory");
            }
            int armed = ahead;                    // k blocks whose loads have been requested
            pdl_wait();
            // (slot and phase are counted along: `stages` is no constant, and a division is longer than the rest of the loop)
            for (int kb = 0, s = 0, turn = 0; kb < nkb; ++kb, ++s) {
                if (s == stages) { s = 0; ++turn; }
                if (turn > 0 && !tc_wait(&empty_bar[s], (turn - 1) & 1, &abort_flag, p.status, 30)) break;
                unsigned char* st = base + (size_t)s * stage_bytes;
                if (kb >= ahead) {
                    armed = kb + 1;
                    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&full_bar[s])), "r"(stage_bytes) : "memory");
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(tc_smem(st)), "l"(tm_w), "r"((kb_begin + kb) * TC_BK), "r"(m0), "r"(tc_smem(&full_bar[s])) : "memory");
                }
                for (int sp = 0; sp < nsplit; ++sp)
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(tc_smem(st + a_bytes + sp * b_bytes)), "l"(&tm_x), "r"((kb_begin + kb) * TC_BK), "r"(sp * p.plane_rows + n0),
                                   "r"(tc_smem(&full_bar[s])) : "memory");
            }
            // Neither this thread nor the issuing one ends before the products have: in the shadow of the epilogue (a look behind the block's last barrier
            // cost 0.08 us a launch).  If a wait of theirs gave up, some of the last loads have no product: they land before this memory is somebody else's.
            tc_drain(&acc_bar, 0);
            if (abort_flag)
                for (int k = max(0, armed - stages); k < armed; ++k) tc_drain(&full_bar[k % stages], (k / stages) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            // instruction descriptor: D fp32, A and B bf16, both K-major, N = BN (or all planes side by side), M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((wide ? nsplit * BN : BN) >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
            const int n_mma = wide ? 1 : nsplit;
            bool ok = true;
            for (int kb = 0, s = 0, phase = 0; kb < nkb && ok; ++kb, ++s) {
                if (s == stages) { s = 0; phase ^= 1; }
                ok = tc_wait(&full_bar[s], phase, &abort_flag, p.status, 31);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t sa = tc_smem(base + (size_t)s * stage_bytes);
                for (int sp = 0; sp < n_mma; ++sp) {
                    const uint32_t sb = sa + a_bytes + sp * b_bytes;
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k) {
                        const uint64_t da = tc_desc(sa + k * 32), db = tc_desc(sb + k * 32);
                        const uint32_t accumulate = (kb | sp | k) ? 1u : 0u;
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                     ::"r"(tmem_base), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                    }
                }
                // the stage may be overwritten once these MMAs have read it
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&empty_bar[s])) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&acc_bar)) : "memory");
            tc_drain(&acc_bar, 0);
        }
    } else {
        // ------------------------------------------------------------------ epilogue: TMEM -> registers -> global
        const int quad = warp & 3;                      // TMEM lanes [32 quad, 32 quad + 32) belong to this warp
        const bool ok = tc_wait_warp(&acc_bar, 0, &abort_flag, p.status, 32);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        pdl_wait();   // before the first store (the output may be something the predecessor still reads)
        if (ok) {
            const int row = m0 + quad * 32 + lane;      // weight row = output column
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t r[32];
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c * 32);
                tc_ld32(r, taddr);
                if constexpr (BN >= 64) {
                    // all column groups of these tokens are requested before the one wait (a TMEM round trip each otherwise:
                    // batch 64 x 1024 2478 -> 2424 us per step).  Not for the 32-token tile: the 64 extra registers cost it
                    // two of its five CTAs per SM (batch 8 x 1024 1083 -> 1153 us).
                    uint32_t q1[32], q2[32];
                    if (wide) {
                        tc_ld32(q1, taddr + (uint32_t)BN);
                        if (nsplit > 2) tc_ld32(q2, taddr + (uint32_t)(2 * BN));
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (wide) {   // add the other planes' columns of the same tokens
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            float v = __uint_as_float(r[j]) + __uint_as_float(q1[j]);
                            if (nsplit > 2) v += __uint_as_float(q2[j]);
                            r[j] = __float_as_uint(v);
                        }
                    }
                } else {
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (wide) {
                        for (int sp = 1; sp < nsplit; ++sp) {
                            uint32_t q[32];
                            tc_ld32(q, taddr + (uint32_t)(sp * BN));
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(q[j]));
                        }
                    }
                }
                if (row < n_rows) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int t = n0 + c * 32 + j;
                        if (t < p.n_tok) {
                            float v = __uint_as_float(r[j]);
                            float* dst = out + (size_t)t * ldo + row;
                            if (p.epi == TC_EPI_ATOMIC) {
                                atomicAdd(dst, v);   // split-K: `out` already holds zero or the residual
                            } else {
                                if (p.epi == TC_EPI_RESID) v += p.resid[(size_t)t * p.ldr + row];
                                *dst = v;
                            }
                        }
                    }
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// The same GEMM for many tokens of one plane as a PERSISTENT kernel: one CTA per SM walks a list of work items (a tile of 128 weight rows x
// 256 tokens).  What the one-tile-per-CTA kernel does in
// series - fill the pipeline, the MMAs, the read-back of 128 KB of accumulator - overlaps here:
//   * the TMA ring never drains between items (the producer runs ahead into the next item's k blocks),
//   * two accumulators in TMEM (2 x 256 columns = all of it): the epilogue warps read item i out while the MMA thread
//     already accumulates item i + 1,
//   * N = 256 per tcgen05.mma halves the shared-memory operand traffic per flop against N = 128.
// Items are numbered with the weight tile fastest, so that the CTAs of a round share a few token tiles in L2.
// ------------------------------------------------------------------------------------------------
constexpr int TP_BN = 256;
constexpr int TP_THREADS = 64 + 256;   // warp 0: TMA, warp 1: MMA, warps 2..9: epilogue (two warps per TMEM lane quadrant, half the columns each)
struct GemmPersistItems {
    int n_items, m_tiles, n_ttiles;   // items = token tiles x weight tiles
};

__global__ void __launch_bounds__(TP_THREADS, 1) gemm_tc_persist_kernel(const __grid_constant__ CUtensorMap tm_w,
                                                                        const __grid_constant__ CUtensorMap tm_x, const GemmTcParams p,
                                                                        const GemmPersistItems w) {
    constexpr int BN = TP_BN;                       // tokens per item
    constexpr int ACC = BN;                         // TMEM columns of one accumulator buffer
    extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[8], empty_bar[8], acc_full[2], acc_empty[2], drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ int armed_s;
    __shared__ volatile int abort_flag;

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int nsplit = p.nsplit, stages = p.stages;
    const uint32_t a_bytes = TC_BM * TC_BK * 2, b_bytes = BN * TC_BK * 2;
    const uint32_t stage_bytes = a_bytes + nsplit * b_bytes;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&full_bar[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&empty_bar[s])) : "memory");
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&acc_full[b])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 256;" ::"r"(tc_smem(&acc_empty[b])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&drain_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"((uint32_t)(2 * ACC)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    pdl_launch();

    // item -> (token tile, weight tile)
    struct Item { int m0, n0; };
    auto decode = [&](int it) { return Item{it % w.m_tiles * TC_BM, it / w.m_tiles * BN}; };
    const int nkb = p.K / TC_BK;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            pdl_wait();
            int s = 0, turn = 0, armed = 0;      // armed: k blocks whose loads have been requested
            for (int it = blockIdx.x; it < w.n_items && !abort_flag; it += gridDim.x) {
                const Item r = decode(it);
                for (int kb = 0; kb < nkb; ++kb, ++s) {
                    if (s == stages) { s = 0; ++turn; }
                    if (turn > 0 && !tc_wait(&empty_bar[s], (turn - 1) & 1, &abort_flag, p.status, 36)) break;
                    unsigned char* st = base + (size_t)s * stage_bytes;
                    ++armed;
                    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&full_bar[s])), "r"(stage_bytes) : "memory");
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(tc_smem(st)), "l"(&tm_w), "r"(kb * TC_BK), "r"(r.m0), "r"(tc_smem(&full_bar[s])) : "memory");
                    for (int sp = 0; sp < nsplit; ++sp)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                     ::"r"(tc_smem(st + a_bytes + sp * b_bytes)), "l"(&tm_x), "r"(kb * TC_BK), "r"(sp * p.plane_rows + r.n0),
                                       "r"(tc_smem(&full_bar[s])) : "memory");
                }
            }
            armed_s = armed;
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
            int s = 0, phase = 0, li = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < w.n_items && ok; it += gridDim.x, ++li) {
                const int acc = li & 1;
                // the accumulator is free once the epilogue warps have read its previous tenant out
                if (li >= 2) ok = tc_wait(&acc_empty[acc], ((li >> 1) - 1) & 1, &abort_flag, p.status, 37);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < nkb && ok; ++kb, ++s) {
                    if (s == stages) { s = 0; phase ^= 1; }
                    ok = tc_wait(&full_bar[s], phase, &abort_flag, p.status, 38);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = tc_smem(base + (size_t)s * stage_bytes);
                    for (int sp = 0; sp < nsplit; ++sp) {
                        const uint32_t sb = sa + a_bytes + sp * b_bytes;
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k) {
                            const uint64_t da = tc_desc(sa + k * 32), db = tc_desc(sb + k * 32);
                            const uint32_t accumulate = (kb | sp | k) ? 1u : 0u;
                            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                         "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                         ::"r"(tmem_base + (uint32_t)(acc * ACC)), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                        }
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&empty_bar[s])) : "memory");
                }
                if (ok) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&acc_full[acc])) : "memory");
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue: TMEM -> registers -> global
        const int quad = warp & 3, half = (warp - 2) >> 2;   // TMEM lanes [32 quad, +32), columns [half BN / 2, + BN / 2)
        pdl_wait();   // before the first store (the output may be something the predecessor still reads)
        int li = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < w.n_items && ok; it += gridDim.x, ++li) {
            const Item r = decode(it);
            const int acc = li & 1;
            ok = tc_wait_warp(&acc_full[acc], (li >> 1) & 1, &abort_flag, p.status, 39);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row = r.m0 + quad * 32 + lane;    // weight row = output column (every tile is a full 128 rows)
#pragma unroll 1
            for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
                if (r.n0 + c * 32 >= p.n_tok) break;    // the rest of the token tile is padding
                uint32_t v[32];
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * ACC + c * 32);
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                             "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                             "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                               "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                               "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                               "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                             : "r"(taddr) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const int t = r.n0 + c * 32 + j;
                    if (t < p.n_tok) {
                        float x = __uint_as_float(v[j]);
                        float* dst = p.out + (size_t)t * p.ldo + row;
                        if (p.epi == TC_EPI_RESID) x += p.resid[(size_t)t * p.ldr + row];
                        *dst = x;
                    }
                }
            }
            // this accumulator may be overwritten by the item after next
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&acc_empty[acc])) : "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    // After a wait gave up (nobody waits any more, so the flag is what it will be): the loads land and the products end before the columns and this memory go.
    if (warp < 2 && abort_flag && elect_one()) {
        if (warp == 0) {
            for (int k = max(0, armed_s - stages); k < armed_s; ++k) tc_drain(&full_bar[k % stages], (k / stages) & 1);
        } else {
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&drain_bar)) : "memory");
            tc_drain(&drain_bar, 0);
        }
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(2 * ACC)) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// The LM head of a decode batch of 4..64 sequences: logits[t, n] = (planes[t] . W[n]) * rsqrt(sum of the 32 parts ssq[i * ssq_ld + t] /
// 1024 + eps).  PERSISTENT: a block per SM walks tiles of 128 words; a TMA ring of five to seven stages (the weight tile's 64 columns and
// the three planes' of all sequences, one B operand) never drains between tiles, and two accumulators let the epilogue of a tile
// run while the products of the next do.
//
// Bound by the weights' bytes: 311 MB, 48 us at the copy bandwidth.  The one-tile-per-block kernel this replaced had two stages a
// block, so a tile was two waits for memory, its products and its epilogue in series.  A one-layer step (LM head, arg-max and about 25 us
// of a layer) of 8 / 27 / 64 sequences, us: 88.9 / 98.8 / 139.9 before, 81.8 / 92.8 / 113.8 now.
// ------------------------------------------------------------------------------------------------
struct LmHeadParams {
    const float* ssq;
    int ssq_ld, n_tok, n_tiles;
    float* out;
    int ldo;
    uint32_t* status;
};
template <int BN> struct LmShape {
    static constexpr uint32_t A_BYTES = TC_BM * TC_BK * 2, STAGE = A_BYTES + 3 * BN * TC_BK * 2;
    static constexpr int STAGES = 200 * 1024 / STAGE;              // 7 or 5
    static constexpr int KB = HIDDEN / TC_BK;
    static constexpr uint32_t ACC = BN == 32 ? 128 : 256;          // TMEM columns of an accumulator
    static constexpr int EPI_WARPS = BN / 8;                       // a warp takes 32 words x 32 sequences
    static constexpr int THREADS = 64 + 32 * EPI_WARPS;
};

template <int BN>
__global__ void __launch_bounds__(LmShape<BN>::THREADS, 1) lm_head_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                                                                          const LmHeadParams p) {
    using S = LmShape<BN>;
    extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[S::STAGES], empty_bar[S::STAGES], acc_full[2], acc_empty[2], drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ int armed_s;
    __shared__ volatile int abort_flag;
    __shared__ float s_scale[BN];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~(uintptr_t)1023);

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&full_bar[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&empty_bar[s])) : "memory");
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&acc_full[b])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(&acc_empty[b])), "r"(S::EPI_WARPS) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&drain_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(2 * S::ACC) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    pdl_launch();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        int armed = 0;                                       // stages requested
        if (elect_one()) {
            const uint32_t st0 = tc_smem(base);
            auto weights = [&](int tile, int kb, int s) {
                asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&full_bar[s])), "r"(S::STAGE) : "memory");
                tc_load_box(st0 + s * S::STAGE, &tm_w, kb * TC_BK, tile * TC_BM, &full_bar[s]);
                ++armed;
            };
            for (int kb = 0; kb < S::STAGES; ++kb) weights(blockIdx.x, kb, kb);      // (KB > STAGES: the first tile's)
            pdl_wait();
            int s = 0, turn = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < p.n_tiles && ok; tile += gridDim.x)
                for (int kb = 0; kb < S::KB; ++kb, ++s) {
                    if (s == S::STAGES) { s = 0; ++turn; }
                    if (turn > 0) {
                        ok = tc_wait(&empty_bar[s], (turn - 1) & 1, &abort_flag, p.status, 70);
                        if (!ok) break;
                        weights(tile, kb, s);
                    }
                    tc_load_planes(st0 + s * S::STAGE + S::A_BYTES, &tm_x, kb * TC_BK, 0, &full_bar[s]);
                }
            armed_s = armed;
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(3 * BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
            const uint64_t da0 = tc_desc(tc_smem(base)), db0 = tc_desc(tc_smem(base) + S::A_BYTES);
            uint64_t ds = 0;
            int s = 0, phase = 0, li = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < p.n_tiles && ok; tile += gridDim.x, ++li) {
                const int acc = li & 1;
                if (li >= 2) ok = tc_wait(&acc_empty[acc], ((li >> 1) - 1) & 1, &abort_flag, p.status, 71);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < S::KB && ok; ++kb, ++s, ds += S::STAGE >> 4) {
                    if (s == S::STAGES) { s = 0; phase ^= 1; ds = 0; }
                    ok = tc_wait(&full_bar[s], phase, &abort_flag, p.status, 72);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                     ::"r"(tmem_base + (uint32_t)acc * S::ACC), "l"(da0 + ds + 2 * k), "l"(db0 + ds + 2 * k), "r"(idesc), "r"((uint32_t)(kb | k)), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&empty_bar[s])) : "memory");
                }
                if (ok) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&acc_full[acc])) : "memory");
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quad = warp & 3, t0 = ((warp - 2) >> 2) * 32;     // TMEM lanes [32 quad, + 32), sequences [t0, t0 + 32)
        pdl_wait();
        for (int j = warp - 2; j < BN; j += S::EPI_WARPS) {
            const float ss = warp_sum(j < p.n_tok ? p.ssq[(size_t)lane * p.ssq_ld + j] : 0.f);
            if (lane == 0) s_scale[j] = rsqrtf(ss / (float)HIDDEN + EPS);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * S::EPI_WARPS) : "memory");
        int li = 0;
        for (int tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x, ++li) {
            const int acc = li & 1;
            if (!tc_wait_warp(&acc_full[acc], (li >> 1) & 1, &abort_flag, p.status, 73) || __any_sync(0xffffffffu, abort_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t r[32], q1[32], q2[32];                  // the planes' columns of the same sequences, under one wait
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)acc * S::ACC + (uint32_t)t0;
            tc_ld32(r, taddr);
            tc_ld32(q1, taddr + BN);
            tc_ld32(q2, taddr + 2 * BN);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(tc_smem(&acc_empty[acc])) : "memory");
            float* dst = p.out + (size_t)t0 * p.ldo + tile * TC_BM + quad * 32 + lane;
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (t0 + j < p.n_tok) dst[(size_t)j * p.ldo] = (__uint_as_float(r[j]) + __uint_as_float(q1[j]) + __uint_as_float(q2[j])) * s_scale[t0 + j];
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    // After a wait gave up (nobody waits any more, so the flag is what it will be): the loads land and the products end before the columns and this memory go.
    if (warp < 2 && abort_flag && elect_one()) {
        if (warp == 0) {
            for (int k = max(0, armed_s - S::STAGES); k < armed_s; ++k) tc_drain(&full_bar[k % S::STAGES], (k / S::STAGES) & 1);
        } else {
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&drain_bar)) : "memory");
            tc_drain(&drain_bar, 0);
        }
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * S::ACC) : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// bf16 tensor [planes, rows, cols] row-major (two-dimensional when planes is 0), box [box_planes, box_rows, 64 columns],
// 128-byte swizzle
bool tc_make_map(CUtensorMap* m, const void* ptr, uint64_t planes, uint64_t rows, uint64_t cols, uint32_t box_planes, uint32_t box_rows, uint64_t plane_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {cols, rows, planes};
    const cuuint64_t strides[2] = {cols * 2, (plane_rows ? plane_rows : rows) * cols * 2};
    const cuuint32_t box[3] = {TC_BK, box_rows, box_planes};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, planes ? 3 : 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Few output tiles cannot fill the GPU: slice K so that about `fill` CTAs per SM stream weights, at least two k blocks per
// slice.  Measured with fill = 1 / 2 / 3 when prompts and all decode batches ran on this kernel: prompts of 2048 tokens 13.9 / 11.2 / 10.9 ms
// (Wo and down have 128 tiles of long K: one wave of long serial CTAs unless K is cut), steps of 8 sequences
// 1322 / 1250 / 1249 us, of 64 3017 / 3031 / 3000 us; 128 tokens (one 128-token tile) are the exception:
// 1.70 / 1.86 / 1.82 ms.  k blocks per slice at least 2 (batch 64 / batch 8 steps: 2 -> 3077 / 1433 us, 4 -> 3121 / 1477).
// Capping the slices of a batch-64 launch at two CTAs per SM (what its 256 TMEM columns per CTA allow at once) was slower:
// 2509 against 2479 us per step.
static int sm_count_of_current_device();
static int k_slices(int n_rows, int n_tok, int bn, int nkb, int sm_count) {
    const int tiles = ((n_rows + TC_BM - 1) / TC_BM) * ((n_tok + bn - 1) / bn);
    const int fill = (n_tok > 64 && n_tok < 256) ? 1 : 3;
    if (tiles >= fill * sm_count) return 1;
    int ksplit = fill * sm_count / tiles;
    if (ksplit > nkb / 2) ksplit = nkb / 2;   // (one / two / three k blocks per slice at least: batch 64 x 1024 2498 / 2369 / 2414 us per step)
    return ksplit < 1 ? 1 : ksplit;
}

// One plane and 128 x 256 items that occupy at least 0.6 of the SMs take the persistent kernel.  Measured when prompts ran on it, 2048 tokens: 4096
// weight rows of K = 1024 23.9 us against 32.3; a threshold of 1.0 / 0.6 / 0.4 of the SMs, whole prompts of 512 tokens 2.39 / 2.28 / 2.29 ms,
// 768 2.90 / 2.49 / 2.49.
static bool persist_serves(int n_rows, int n_tok, int nsplit, int sm_count) {
    // one activation plane: with more the 256-token stages no longer fit four deep
    return n_tok >= TP_BN && nsplit == 1 && (n_rows / TC_BM) * ((n_tok + TP_BN - 1) / TP_BN) * 10 >= sm_count * 6;
}

static cudaError_t launch_persist(const CUtensorMap& tw, const CUtensorMap& tx, GemmTcParams p, int n_rows, int n_tok, int sm_count, cudaStream_t st) {
    constexpr int BN = TP_BN;
    const uint32_t stage_bytes = TC_BM * TC_BK * 2 + p.nsplit * BN * TC_BK * 2;
    int stages = (int)((200u * 1024u) / stage_bytes);
    if (stages > 8) stages = 8;
    if (stages < 2) return cudaErrorInvalidValue;
    p.stages = stages;
    const size_t smem = (size_t)stages * stage_bytes + 1024;
    {
        static bool attr_set[MAX_DEVICES] = {};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> hold(host_lock());
        if (!attr_set[dev]) {
            e = cudaFuncSetAttribute(gemm_tc_persist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
            if (e != cudaSuccess) return e;
            attr_set[dev] = true;
        }
    }
    GemmPersistItems w{};
    w.m_tiles = n_rows / TC_BM;
    w.n_ttiles = (n_tok + BN - 1) / BN;
    w.n_items = w.m_tiles * w.n_ttiles;
    const int grid = w.n_items < sm_count ? w.n_items : sm_count;
    return launch_chain(gemm_tc_persist_kernel, dim3(grid), dim3(TP_THREADS), smem, st, tw, tx, p, w);
}

template <int BN>
static cudaError_t launch_bn(const CUtensorMap* tw, const CUtensorMap& tx, GemmTcParams p, int n_rows, int n_tok, int sm_count, cudaStream_t st) {
    // n_rows: all weight rows of the launch (the sum over the groups); tw: three maps (unused ones repeat the first)
    const int nkb = p.K / TC_BK;
    const int tiles = ((n_rows + TC_BM - 1) / TC_BM) * ((n_tok + BN - 1) / BN);
    int ksplit = 1;
    if (p.epi == TC_EPI_STORE || p.resid == p.out) ksplit = k_slices(n_rows, n_tok, BN, nkb, sm_count);
    p.kb_per_split = (nkb + ksplit - 1) / ksplit;
    ksplit = (nkb + p.kb_per_split - 1) / p.kb_per_split;
    if (ksplit > 1) {
        if (p.epi == TC_EPI_STORE && !p.out_is_zero) {   // partial sums are added onto zeros
            const int ng = p.n_groups > 1 ? p.n_groups : 1;
            for (int g = 0; g < ng; ++g) {
                float* o = p.n_groups > 1 ? p.g_out[g] : p.out;
                const int ld = p.n_groups > 1 ? p.g_ldo[g] : p.ldo, rows = p.n_groups > 1 ? p.g_tiles[g] * TC_BM : n_rows;
                // adjacent groups of one row-major buffer (q | k | v) are cleared by the first group's call
                if (g > 0 && p.g_out[g] == p.g_out[g - 1] + p.g_tiles[g - 1] * TC_BM && p.g_ldo[g] == p.g_ldo[g - 1]) continue;
                int span = rows;
                for (int h = g + 1; h < ng && p.g_out[h] == o + span && p.g_ldo[h] == ld; ++h) span += p.g_tiles[h] * TC_BM;
                cudaError_t e = cudaMemset2DAsync(o, (size_t)ld * 4, 0, (size_t)span * 4, (size_t)n_tok, st);
                if (e != cudaSuccess) return e;
            }
        }
        p.epi = TC_EPI_ATOMIC;         // in place on the residual otherwise
    }
    const uint32_t stage_bytes = TC_BM * TC_BK * 2 + p.nsplit * BN * TC_BK * 2;
    int stages = (int)((200u * 1024u) / stage_bytes);
    if (stages > 8) stages = 8;
    if (stages > p.kb_per_split) stages = p.kb_per_split;
    // Grids of more than two tiles per SM: two stages, so that two CTAs share an SM and the epilogue of one
    // overlaps the MMAs of the other (measured when prompts ran on this kernel, 2048 tokens: 14.0 ms against 15.6 ms with four stages).
    if (tiles * ksplit > 2 * sm_count && stages > 2) stages = 2;
    if (stages < 1) return cudaErrorInvalidValue;
    p.stages = stages;
    const size_t smem = (size_t)stages * stage_bytes + 1024;
    {   // the shared-memory limit of a function is a per-device attribute: set it once on every device that launches
        static bool attr_set[MAX_DEVICES] = {};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> hold(host_lock());
        if (!attr_set[dev]) {
            e = cudaFuncSetAttribute(gemm_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
            if (e != cudaSuccess) return e;
            attr_set[dev] = true;
        }
    }
    dim3 grid((n_rows + TC_BM - 1) / TC_BM, (n_tok + BN - 1) / BN, ksplit);
    return launch_chain(gemm_tc_kernel<BN>, grid, dim3(TC_THREADS), smem, st, tw[0], tw[1], tw[2], tx, p);
}

// Encoding a tensor map costs a few microseconds of host time; a step issues hundreds of GEMMs over the
// same few hundred (pointer, shape) pairs, so the maps are cached.
struct MapKey { const void* p; uint64_t planes, rows, cols; uint32_t box; };
struct MapEntry { MapKey k; CUtensorMap m; };
static std::vector<MapEntry>& map_cache() { static std::vector<MapEntry> c; return c; }
// (device addresses are unique across the GPUs of a process, so one cache serves them all; it is locked because
// engines on different host threads share it)
static bool cached_map(const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows, CUtensorMap* out, uint64_t planes = 0) {
    std::lock_guard<std::mutex> hold(host_lock());
    auto& c = map_cache();
    for (auto& e : c)
        if (e.k.p == ptr && e.k.planes == planes && e.k.rows == rows && e.k.cols == cols && e.k.box == box_rows) { *out = e.m; return true; }
    if (c.size() > 4096) c.clear();
    MapEntry e{{ptr, planes, rows, cols, box_rows}, {}};
    if (!tc_make_map(&e.m, ptr, planes, rows, cols, (uint32_t)planes, box_rows)) return false;
    c.push_back(e);
    *out = e.m;
    return true;
}
bool gemm_tc_splits_k(int n_rows, int n_tok, int K) {
    const int bn = n_tok <= 32 ? 32 : (n_tok <= 64 ? 64 : 128);
    return k_slices(n_rows, n_tok, bn, K / TC_BK, sm_count_of_current_device()) > 1;
}
bool tc_cached_map(const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows, CUtensorMap* out, uint64_t planes) {
    return cached_map(ptr, rows, cols, box_rows, out, planes);
}
int tc_sm_count() { return sm_count_of_current_device(); }
static int sm_count_of_current_device() {
    static int sms[MAX_DEVICES] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return 0;
    std::lock_guard<std::mutex> hold(host_lock());
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return sms[dev];
}

template <int BN>
static cudaError_t launch_lm(const CUtensorMap& tw, const CUtensorMap& tx, const LmHeadParams& p, int sm_count, cudaStream_t st) {
    using S = LmShape<BN>;
    constexpr size_t smem = (size_t)S::STAGES * S::STAGE + 1024;
    static bool attr_set[MAX_DEVICES] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> hold(host_lock());
        if (!attr_set[dev]) {
            e = cudaFuncSetAttribute(lm_head_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            attr_set[dev] = true;
        }
    }
    return launch_chain(lm_head_kernel<BN>, dim3(p.n_tiles < sm_count ? p.n_tiles : sm_count), dim3(S::THREADS), smem, st, tw, tx, p);
}

cudaError_t launch_lm_head(const LmHeadCall& c, cudaStream_t st) {
    const int bn = c.n_tok <= 32 ? 32 : 64, sm = sm_count_of_current_device();
    if (sm < 1) return cudaErrorInvalidDevice;
    if (c.vocab < TC_BM || c.vocab % TC_BM || c.n_tok < 1 || c.n_tok > 64 || c.prow < bn) return cudaErrorInvalidValue;
    CUtensorMap tw, tx;
    if (!cached_map(c.w, (uint64_t)c.vocab, (uint64_t)HIDDEN, TC_BM, &tw) || !cached_map(c.planes, (uint64_t)c.prow, (uint64_t)HIDDEN, (uint32_t)bn, &tx, 3)) return cudaErrorUnknown;
    const LmHeadParams p{c.ssq, c.ssq_ld, c.n_tok, c.vocab / TC_BM, c.out, c.vocab, c.status};
    return bn == 32 ? launch_lm<32>(tw, tx, p, sm, st) : launch_lm<64>(tw, tx, p, sm, st);
}

cudaError_t launch_gemm_tc(const GemmTcCall& c, cudaStream_t st) {
    if (c.K % TC_BK || c.n_rows % TC_BM || c.nsplit < 1 || c.nsplit > 3 || c.n_tok < 1) return cudaErrorInvalidValue;
    // token tile: the smallest of 32 / 64 / 128 that covers the tokens, 128 beyond
    const int bn = c.n_tok <= 32 ? 32 : (c.n_tok <= 64 ? 64 : 128);
    if (c.plane_rows % bn) return cudaErrorInvalidValue;
    CUtensorMap tw, tx;
    if (!cached_map(c.w, (uint64_t)c.n_rows, (uint64_t)c.K, TC_BM, &tw)) return cudaErrorUnknown;
    if (!cached_map(c.x_planes, (uint64_t)c.nsplit * c.plane_rows, (uint64_t)c.K, (uint32_t)bn, &tx)) return cudaErrorUnknown;
    GemmTcParams p{};
    p.out = c.out; p.resid = c.resid; p.ldo = c.ldo; p.ldr = c.ldr; p.n_rows = c.n_rows; p.n_tok = c.n_tok; p.K = c.K;
    p.nsplit = c.nsplit; p.plane_rows = c.plane_rows; p.epi = c.resid ? TC_EPI_RESID : TC_EPI_STORE; p.status = c.status;
    const int sm_count = sm_count_of_current_device();
    if (sm_count < 1) return cudaErrorInvalidDevice;
    const CUtensorMap maps[3] = {tw, tw, tw};
    if (persist_serves(c.n_rows, c.n_tok, c.nsplit, sm_count)) {
        CUtensorMap txp;
        if (!cached_map(c.x_planes, (uint64_t)c.nsplit * c.plane_rows, (uint64_t)c.K, (uint32_t)TP_BN, &txp)) return cudaErrorUnknown;
        return launch_persist(tw, txp, p, c.n_rows, c.n_tok, sm_count, st);
    }
    if (bn == 32) return launch_bn<32>(maps, tx, p, c.n_rows, c.n_tok, sm_count, st);
    if (bn == 64) return launch_bn<64>(maps, tx, p, c.n_rows, c.n_tok, sm_count, st);
    return launch_bn<128>(maps, tx, p, c.n_rows, c.n_tok, sm_count, st);
}

cudaError_t launch_gemm_tc_group(const GemmTcGroupCall& c, cudaStream_t st) {
    if (c.n_groups < 1 || c.n_groups > 3 || c.K % TC_BK || c.nsplit < 1 || c.nsplit > 3 || c.n_tok < 1) return cudaErrorInvalidValue;
    const int bn = c.n_tok <= 32 ? 32 : (c.n_tok <= 64 ? 64 : 128);
    if (c.plane_rows % bn) return cudaErrorInvalidValue;
    CUtensorMap maps[3];
    GemmTcParams p{};
    int rows = 0;
    for (int g = 0; g < c.n_groups; ++g) {
        if (c.n_rows[g] % TC_BM || c.n_rows[g] < TC_BM) return cudaErrorInvalidValue;
        if (!cached_map(c.w[g], (uint64_t)c.n_rows[g], (uint64_t)c.K, TC_BM, &maps[g])) return cudaErrorUnknown;
        p.g_tiles[g] = c.n_rows[g] / TC_BM; p.g_out[g] = c.out[g]; p.g_ldo[g] = c.ldo[g];
        rows += c.n_rows[g];
    }
    for (int g = c.n_groups; g < 3; ++g) maps[g] = maps[0];
    CUtensorMap tx;
    if (!cached_map(c.x_planes, (uint64_t)c.nsplit * c.plane_rows, (uint64_t)c.K, (uint32_t)bn, &tx)) return cudaErrorUnknown;
    p.n_groups = c.n_groups; p.out = c.out[0]; p.resid = nullptr; p.ldo = c.ldo[0]; p.ldr = 0; p.n_rows = rows; p.n_tok = c.n_tok; p.K = c.K;
    p.nsplit = c.nsplit; p.plane_rows = c.plane_rows; p.epi = TC_EPI_STORE; p.status = c.status; p.out_is_zero = c.out_is_zero;
    const int sm_count = sm_count_of_current_device();
    if (sm_count < 1) return cudaErrorInvalidDevice;
    if (bn == 32) return launch_bn<32>(maps, tx, p, rows, c.n_tok, sm_count, st);
    if (bn == 64) return launch_bn<64>(maps, tx, p, rows, c.n_tok, sm_count, st);
    return launch_bn<128>(maps, tx, p, rows, c.n_tok, sm_count, st);
}

}  // namespace q3
