// Causal attention for prefill on the 5th-generation tensor cores: tcgen05.mma with accumulators in TMEM, K/V tiles
// brought in by TMA (cp.async.bulk.tensor, 128-byte swizzle) through a two-stage mbarrier pipeline.
//
// One CTA owns 64 query positions of ONE KV HEAD GROUP: its M = 128 rows are the two query heads of the group (rows
// 0..63 head 2g, rows 64..127 head 2g + 1), so every K/V tile is fetched once for both heads (GQA sharing).  It walks
// the key tiles (128 keys) up to its diagonal:
//     S  = Q K^T      M 128 x N 128 keys x K 128 dims: Q as TWO bf16 planes (hi + lo, so the scores carry fp32-grade
//                     accuracy into the exponent), both K-major operands      -> TMEM columns [0, 128) / [128, 256)
//     P  = exp(S - m) two groups of eight warps, two threads per row (64 keys each); group g takes the key tiles t with t % 2 == g, so that
//                     one group's exponentials run while the tensor pipe and the hand-offs of the other's tile do.  P, rounded to
//                     bf16, takes the place of S in TMEM: the A operand of the second product
//     O += P V        M 128 x N 128 dims x K 128 keys; V is the MN-major B operand straight from its TMA tile.  Each group has an O of its own
//                     -> TMEM columns [256, 384) / [384, 512), summed by the tensor pipe over the group's tiles
// A group keeps its own running maximum and sum.  Its maximum is raised, and its O rescaled, only when a score exceeds it by 2^8: P
// then reaches at most 2^8, its bf16 rounding stays the same relative error and the fp32 sums have room.  At the end the two groups'
// O are combined under one maximum and written as the bf16 plane the Wo GEMM reads.
// The MMA thread issues S of tile t + 2 right behind the product of tile t, whose P it overwrites (the pipe works in order).
// One block per (query tile, kv group) in order of work (a query tile has 1..n key tiles), so that the SMs that finish early pick up the
// light tiles.  Where SMs would stay idle, two blocks of a cluster share a long query tile, half of the key tiles each, and finish half of its positions
// each (O, maxima and sums travel through distributed shared memory).  Every mbarrier wait is bounded.
//
// What bounds it: a key tile is 24 products of 128 x 128 x 16 (0.8 us at the measured bf16 rate) and 16 K exponentials and 8 K conversions on
// the XU pipe (0.8 us).  A tile takes 1.2 us: the products wait
// for the slowest of a group's warps (0.3 us) and for the exponentials that no other tile covers.  Measured, us a launch at 512 / 777 / 2048 tokens: sixteen
// warps on every tile with P in shared memory and O in registers 12.6 / 16.8 / 37.6, two groups 11.4 / 14.5 / 32.1.
//
// Replaces the [16, T, T] masked score matrix of the reference's prefill (qwen3mk/prefill.py:71-75).
#include <cuda.h>

#include "q3_engine.h"
#include "q3_gemm_tc.h"
#include "q3_prompt.h"
#include "q3_tc_ptx.cuh"

namespace q3 {

constexpr int AT_SOFT = 512;              // softmax / output threads: warps 0..15, group 0 the first eight
constexpr int AT_THREADS = AT_SOFT + 64;  // + warp 16 TMA producer, warp 17 MMA issuer and TMEM owner
constexpr int AT_QT = 64;                 // query positions per CTA pass
constexpr int AT_KT = 128;                // keys per tile
constexpr int AT_STAGES = 2;
constexpr uint32_t AT_BOX = 128 * 128;    // bytes of one [128 rows x 64 columns] bf16 box, 128-byte swizzle
constexpr uint32_t AT_Q_BYTES = 2 * AT_BOX, AT_KV_BYTES = 2 * AT_BOX;   // 128 x 128 bf16 = two boxes
constexpr size_t AT_SMEM = 2 * AT_Q_BYTES + AT_STAGES * 2 * AT_KV_BYTES;   // Q hi, Q lo, stages x (K, V) = 192 KB
constexpr int AT_SPLIT_MIN = 3;           // key tiles of a query tile that two blocks share, at least
constexpr float AT_LAG = 8.f;             // how far (in log2) scores may exceed the maximum that P is taken under
constexpr unsigned long long AT_WAIT_NS = 200ull * 1000 * 1000;

__device__ __forceinline__ uint32_t at_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long at_ns() { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }

__device__ __forceinline__ bool at_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t site) {
    unsigned it = 0;
    unsigned long long t0 = 0;
    for (;;) {
        uint32_t ok;
        // test_wait, not try_wait: a try_wait on a phase that is not complete yet parks the thread for a while, and a tile
        // has eight hand-offs between the MMA thread and the softmax warps
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(at_smem(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
        if ((++it & 63u) == 0) {
            const unsigned long long t = at_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > AT_WAIT_NS) {
                if (status) report(status, ST_MBAR_TIMEOUT, site, parity);
                *abort_flag = 1;
                return false;
            }
        }
    }
}
// One lane of a converged warp polls for all 32: the polls of 16 softmax warps, a request a lane, delay the MMA thread's own.
__device__ __forceinline__ bool at_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t site) {
    return one_lane_waits([&] { return at_wait(bar, parity, abort_flag, status, site); });
}

// K-major operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart (as in the GEMM)
__device__ __forceinline__ uint64_t at_desc_k(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// MN-major operand (V: rows = keys = the K index, 64 contiguous dims per 128-byte row), 128-byte swizzle: the next 64
// dims are one box further (leading byte offset), the next 8 keys 1024 bytes further (stride byte offset)
__device__ __forceinline__ uint64_t at_desc_mn(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);
    d |= (uint64_t)(AT_BOX >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// The special-function pipe (16 results a cycle and SM) is this kernel's bottleneck: a tile needs 16 K exponentials and
// the conversion of 16 K probabilities to bf16.  So: one ex2 per element (log2(e) is folded into the scale of Q) and one
// conversion per PAIR of elements.
__device__ __forceinline__ float at_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float at_max_nan(float a, float b) {   // NaN if either is
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}
__device__ __forceinline__ uint32_t at_pack_bf16(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

__device__ __forceinline__ void at_ld32(uint32_t (&r)[32], uint32_t taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}

__device__ __forceinline__ void at_ld16(uint32_t* r, uint32_t taddr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void at_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}

// both blocks of a cluster, all threads; writes to the other's shared memory before it are seen behind it
__device__ __forceinline__ void at_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t at_map(uint32_t smem_addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}

struct PrefillAttnTcArgs {
    bf16_raw* plane;      // [T][2048] bf16: the output, as the Wo GEMM reads it
    int T, layer;
    int shared;           // PAIR: query tiles (of a kv group, the longest) that two blocks share
    uint32_t* status;
};

template <bool PAIR>
__global__ void __launch_bounds__(AT_THREADS, 1) prefill_attn_tc_kernel(const __grid_constant__ CUtensorMap tm_qh, const __grid_constant__ CUtensorMap tm_ql,
                                                                        const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                                                                        const PrefillAttnTcArgs a) {
    extern __shared__ __align__(1024) unsigned char at_raw[];
    __shared__ __align__(8) uint64_t k_full[AT_STAGES], v_full[AT_STAGES], k_empty[AT_STAGES], v_empty[AT_STAGES], q_full, s_full[2], p_full[2], o_full[2], drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;
    __shared__ float s_max[2][2][2][128];           // per group and parity of its tiles: the tile's maximum of a row's two halves
    __shared__ float s_m[2][128], s_l[2][2][128];   // at the end: per group, a row's maximum and the two halves of its sum

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    // The query tiles with the most key tiles come first.  PAIR: a cluster of two blocks shares one of the `shared` longest, its key tiles cut in two, or
    // takes two tiles, a block each.
    const int tiles = (a.T + AT_QT - 1) / AT_QT, unit = PAIR ? (int)blockIdx.x >> 1 : (int)blockIdx.x, place = unit / KV_HEADS, rank = PAIR ? (int)blockIdx.x & 1 : 0;
    const int g = unit % KV_HEADS;                  // kv head; query heads 2g and 2g + 1
    const bool both = PAIR && place < a.shared;
    const int nth = !PAIR || both ? place : a.shared + 2 * (place - a.shared) + rank;
    if (PAIR && nth >= tiles) return;               // (an odd tile's other block)
    const int q0 = (tiles - 1 - nth) * AT_QT;
    const int all_kt = (q0 + AT_QT - 1) / AT_KT + 1;        // key tiles up to and including the diagonal one
    const int kt0 = both && rank ? (all_kt + 1) / 2 : 0, n_kt = both ? (rank ? all_kt / 2 : (all_kt + 1) / 2) : all_kt;     // this block's
    unsigned char* sQh = at_raw;
    unsigned char* sQl = sQh + AT_Q_BYTES;
    unsigned char* sKV = sQl + AT_Q_BYTES;          // stage s: K at s * 2 * AT_KV_BYTES, V right after it

    if (tid == 0) {
        for (int s = 0; s < AT_STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&k_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&v_full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&k_empty[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&v_empty[s])) : "memory");
        }
        for (int b = 0; b < 2; ++b) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&s_full[b])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&o_full[b])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(at_smem(&p_full[b])) : "memory");   // the group's warps
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&q_full)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(at_smem(&drain_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_flag = 0;
    }
    if (warp == AT_SOFT / 32 + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at_smem(&tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;

    pdl_launch();

    int armed_k = 0, armed_v = 0;                           // tiles whose K and V the producer has requested
    {
        if (warp == AT_SOFT / 32) {
            // ------------------------------------------------------------------ TMA producer
            if (elect_one()) {
                pdl_wait();
                // Q of both heads, hi and lo: boxes of 64 positions x 64 dims, rows past the prompt read as zeros
                asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(&q_full)), "r"(2 * AT_Q_BYTES) : "memory");
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int plane = i >> 2, head = (i >> 1) & 1, b = i & 1;
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(at_smem((plane ? sQl : sQh) + b * AT_BOX + head * (AT_BOX / 2))), "l"(plane ? &tm_ql : &tm_qh),
                                   "r"((2 * g + head) * HEAD_DIM + 64 * b), "r"(q0), "r"(at_smem(&q_full)) : "memory");
                }
                // K and V of a tile share a stage but are released separately: the K half is free as soon as S of its tile has
                // been computed, a whole tile before the V half (after PV), so the next K is on its way that much earlier
                for (int t = 0; t < n_kt; ++t) {
                    const int s = t % AT_STAGES;
                    unsigned char* sk = sKV + (size_t)s * 2 * AT_KV_BYTES;
                    unsigned char* sv = sk + AT_KV_BYTES;
                    if (t >= AT_STAGES && !at_wait(&k_empty[s], ((t / AT_STAGES) - 1) & 1, &abort_flag, a.status, 40)) break;
                    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(&k_full[s])), "r"(AT_KV_BYTES) : "memory");
#pragma unroll
                    for (int b = 0; b < 2; ++b)        // the two 64-dim halves of the head
                        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                                     ::"r"(at_smem(sk + b * AT_BOX)), "l"(&tm_k), "r"(g * HEAD_DIM + 64 * b), "r"((kt0 + t) * AT_KT), "r"(a.layer), "r"(at_smem(&k_full[s])) : "memory");
                    armed_k = t + 1;
                    if (t >= AT_STAGES && !at_wait(&v_empty[s], ((t / AT_STAGES) - 1) & 1, &abort_flag, a.status, 47)) break;
                    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(&v_full[s])), "r"(AT_KV_BYTES) : "memory");
#pragma unroll
                    for (int b = 0; b < 2; ++b)
                        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                                     ::"r"(at_smem(sv + b * AT_BOX)), "l"(&tm_v), "r"(g * HEAD_DIM + 64 * b), "r"((kt0 + t) * AT_KT), "r"(a.layer), "r"(at_smem(&v_full[s])) : "memory");
                    armed_v = t + 1;
                }
            }
        } else if (warp == AT_SOFT / 32 + 1) {
            // ------------------------------------------------------------------ MMA issuer
            if (elect_one()) {
                // D fp32, A and B bf16, M 128, N 128; bit 16: B is MN-major (V)
                const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
                const uint32_t idesc_o = idesc_s | (1u << 16);
                // (descriptors count 16-byte units; what a step adds to them is a constant)
                constexpr uint64_t BOX = AT_BOX >> 4, STAGE = 2 * AT_KV_BYTES >> 4;
                const uint64_t dq = at_desc_k(at_smem(sQh)), dk = at_desc_k(at_smem(sKV)), dv = at_desc_mn(at_smem(sKV + AT_KV_BYTES));
                static_assert(AT_STAGES == 2, "a tile's stage is its parity");
                auto issue_s = [&](int t) -> bool {    // S = (Q hi + Q lo) K^T of key tile t, into S buffer t & 1
                    const int s = t % AT_STAGES;
                    if (!at_wait(&k_full[s], (t / AT_STAGES) & 1, &abort_flag, a.status, 41)) return false;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t dks = dk + (uint64_t)s * STAGE;
#pragma unroll
                    for (int plane = 0; plane < 2; ++plane) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {  // 16 dims a step: four steps per 64-dim box
                            const uint64_t o = (uint64_t)(k >> 2) * BOX + (uint64_t)(k & 3) * 2;
                            const uint64_t da = dq + (uint64_t)plane * (AT_Q_BYTES >> 4) + o, db = dks + o;
                            const uint32_t acc = (plane | k) ? 1u : 0u;
                            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                         "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                         ::"r"(tmem_base + (uint32_t)(t & 1) * 128u), "l"(da), "l"(db), "r"(idesc_s), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                        }
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(at_smem(&s_full[t & 1])) : "memory");
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(at_smem(&k_empty[s])) : "memory");
                    return true;
                };
                bool ok = at_wait(&q_full, 0, &abort_flag, a.status, 48) && issue_s(0) && (n_kt == 1 || issue_s(1));
                for (int t = 0; t < n_kt && ok; ++t) {
                    const int b = t & 1, s = t % AT_STAGES;
                    ok = at_wait(&p_full[b], (t >> 1) & 1, &abort_flag, a.status, 42) && at_wait(&v_full[s], (t / AT_STAGES) & 1, &abort_flag, a.status, 43);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t dvs = dv + (uint64_t)s * STAGE;
                    const uint32_t tp = tmem_base + (uint32_t)b * 128u;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {      // 16 keys a step: eight columns of P (two bf16 each)
                        const uint64_t db = dvs + (uint64_t)k * (2048 >> 4);
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                     "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                     ::"r"(tp + 256u), "r"(tp + (uint32_t)k * 8u), "l"(db), "r"(idesc_o), "r"((t >= 2 || k) ? 1u : 0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(at_smem(&o_full[b])) : "memory");
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(at_smem(&v_empty[s])) : "memory");
                    if (t + 2 < n_kt) ok = issue_s(t + 2);
                }
            }
        } else {
            // ------------------------------------------------------------------ softmax and output: row = TMEM lane
            const int quad = warp & 3, row = quad * 32 + lane, grp = warp >> 3, part = (warp >> 2) & 1;   // part: 64 keys of a tile
            const int qpos = q0 + (row & 63);
            const uint32_t trow = tmem_base + ((uint32_t)(quad * 32) << 16);
            const uint32_t ts = trow + (uint32_t)(grp * 128), to = trow + 256u + (uint32_t)(grp * 128 + part * 64);
            float m = -INFINITY, lsum = 0.f;
            bool ok = true;
            // Two warps share their rows and wait for themselves, so one may give up where the other does not.  They stay together all the same: one that
            // gives up leaves NaN as its maxima (a maximum is never one) and both leave the loop behind the same barrier.  Maxima of alternate tiles
            // have places of their own: a warp that gave up on O is at the next barrier while the other still reads.
            for (int t = grp, i = 0; t < n_kt; t += 2, ++i) {
                ok = ok && at_wait_warp(&s_full[grp], i & 1, &abort_flag, a.status, 44);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t r[2][32];
                at_ld32(r[0], ts + (uint32_t)(part * 64));
                at_ld32(r[1], ts + (uint32_t)(part * 64 + 32));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (kt0 + t == all_kt - 1) {   // the diagonal tile: causal mask (it also hides keys past the prompt)
                    const int key0 = (kt0 + t) * AT_KT + part * 64;
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (key0 + j > qpos) r[0][j] = 0xff800000u;            // -inf
                        if (key0 + 32 + j > qpos) r[1][j] = 0xff800000u;
                    }
                }
                float x[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int j = 0; j < 32; ++j) { x[j & 1] = fmaxf(x[j & 1], __uint_as_float(r[0][j])); x[2 + (j & 1)] = fmaxf(x[2 + (j & 1)], __uint_as_float(r[1][j])); }
                const float x0 = ok ? fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3])) : NAN;
                // the row's other half is a thread of the warp four further; behind the barrier both have read their part of S, too
                s_max[grp][i & 1][part][row] = x0;
                asm volatile("bar.sync %0, 64;" ::"r"(1 + grp * 4 + quad) : "memory");
                const float top = at_max_nan(x0, s_max[grp][i & 1][part ^ 1][row]);   // finite: the first key of a tile is visible to every row
                const bool raise = !(top <= m + AT_LAG);
                if (__any_sync(0xffffffffu, raise)) {
                    if (top != top) { ok = false; break; }      // (here, where few tiles come: looking in every tile cost 0.3 us a launch)
                    const float mn = raise ? top : m, c = at_ex2(m - mn);
                    m = mn;
                    if (i > 0) {           // O of the tiles so far, once the last of them has been added
                        ok = at_wait_warp(&o_full[grp], (i - 1) & 1, &abort_flag, a.status, 45);
                        if (!ok) continue;      // (P of this tile is not handed over: its S is the last)
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        lsum *= c;
#pragma unroll 1
                        for (int h = 0; h < 64; h += 16) {
                            uint32_t o[16];
                            at_ld16(o, to + (uint32_t)h);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * c);
                            at_st16(to + (uint32_t)h, o);
                        }
                    }
                }
                float psum0 = 0.f, psum1 = 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t pk[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float e0 = at_ex2(__uint_as_float(r[h][2 * j]) - m), e1 = at_ex2(__uint_as_float(r[h][2 * j + 1]) - m);
                        psum0 += e0; psum1 += e1;
                        pk[j] = at_pack_bf16(e0, e1);
                    }
                    at_st16(ts + (uint32_t)(part * 32 + h * 16), pk);
                }
                lsum += psum0 + psum1;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(at_smem(&p_full[grp])) : "memory");
            }
            const int mine = (n_kt - grp + 1) / 2;      // tiles of this group
            if (ok && mine > 0) ok = at_wait_warp(&o_full[grp], (mine - 1) & 1, &abort_flag, a.status, 46);
            if (part == 0) s_m[grp][row] = m;
            s_l[grp][part][row] = lsum;
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            asm volatile("bar.sync 9, %0;" ::"n"(AT_SOFT) : "memory");
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const float m0 = s_m[0][row], m1 = s_m[1][row], mx = fmaxf(m0, m1);      // (a block of one tile has no second group: m1 is -inf)
            const float f0 = at_ex2(m0 - mx), f1 = at_ex2(m1 - mx);
            const float sum = (s_l[0][0][row] + s_l[0][1][row]) * f0 + (s_l[1][0][row] + s_l[1][1][row]) * f1;
            const float inv = both ? 1.f : 1.f / sum, w0 = f0 * inv, w1 = f1 * inv;
            const int dim0 = (warp >> 2) * 32;          // a quarter of the row's dims
            uint32_t o0[32], o1[32];
            at_ld32(o0, trow + 256u + (uint32_t)dim0);
            at_ld32(o1, trow + 384u + (uint32_t)dim0);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float o[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                o[j] = __uint_as_float(o0[j]) * w0;
                if (n_kt > 1) o[j] = fmaf(__uint_as_float(o1[j]), w1, o[j]);   // (TMEM that nothing was added to may hold anything)
            }
            const int pos = row & 63;
            const bool own = !both || (pos >> 5) == rank;
            if (both) {
                // Each block finishes 32 of the positions: the other's sums, and O under its maximum, come through distributed shared memory into the place
                // of Q hi (every product of both blocks has completed), the two numbers of a row into that of Q lo.
                const int slot = (row >> 6) * 4 + (warp >> 2);
                at_cluster_sync();
                if (!own) {
                    const uint32_t to_o = at_map(at_smem(sQh) + (uint32_t)(slot * 8 * 32 + lane) * 16u, rank ^ 1), to_n = at_map(at_smem(sQl) + (uint32_t)((row >> 6) * 32 + lane) * 8u, rank ^ 1);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to_o + (uint32_t)j * 512u), "f"(o[4 * j]), "f"(o[4 * j + 1]), "f"(o[4 * j + 2]), "f"(o[4 * j + 3]) : "memory");
                    // (a block that gave up sends NaN: the other does not pass its rows off as whole)
                    if (warp < 4) asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(to_n), "f"(mx), "f"(abort_flag ? NAN : sum) : "memory");
                }
                at_cluster_sync();
                if (own) {
                    const float2 n2 = reinterpret_cast<const float2*>(sQl)[(row >> 6) * 32 + lane];
                    const float top = fmaxf(mx, n2.x), a0 = at_ex2(mx - top), a1 = at_ex2(n2.x - top), r = 1.f / (sum * a0 + n2.y * a1), u0 = a0 * r, u1 = a1 * r;
                    const float4* in = reinterpret_cast<const float4*>(sQh) + slot * 8 * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 v = in[j * 32];
                        o[4 * j] = fmaf(v.x, u1, o[4 * j] * u0); o[4 * j + 1] = fmaf(v.y, u1, o[4 * j + 1] * u0);
                        o[4 * j + 2] = fmaf(v.z, u1, o[4 * j + 2] * u0); o[4 * j + 3] = fmaf(v.w, u1, o[4 * j + 3] * u0);
                    }
                }
            }
            // Through shared memory (Q's: all products have completed), so that a warp writes a position's 512 bytes (a thread per row: 1 us more a block).
            // 16-byte chunks of a position's row are XORed by the position.
            uint4* const so = reinterpret_cast<uint4*>(both ? sQl + 1024 : sQh);
            if (own) {
                const int at = both ? pos & 31 : pos, chunk = (row >> 6) * 16 + dim0 / 8;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    so[at * 32 + ((chunk + j) ^ (pos & 7))] = make_uint4(at_pack_bf16(o[8 * j], o[8 * j + 1]), at_pack_bf16(o[8 * j + 2], o[8 * j + 3]),
                                                                          at_pack_bf16(o[8 * j + 4], o[8 * j + 5]), at_pack_bf16(o[8 * j + 6], o[8 * j + 7]));
            }
            asm volatile("bar.sync 9, %0;" ::"n"(AT_SOFT) : "memory");
            if (!abort_flag) {
                const int p0 = both ? q0 + 32 * rank : q0, count = both ? 2 : 4;
                bf16_raw* const dst = a.plane + (size_t)p0 * Q_DIM + 2 * g * HEAD_DIM + lane * 8;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int at = warp + 16 * i;
                    if (i < count && p0 + at < a.T) *reinterpret_cast<uint4*>(dst + (size_t)at * Q_DIM) = so[at * 32 + (lane ^ (at & 7))];
                }
            }
        }
        if (both && warp >= AT_SOFT / 32) { __syncwarp(); at_cluster_sync(); at_cluster_sync(); }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // After a wait gave up (nobody waits any more, so the flag is what it will be): the loads land and the products end before this block's memory and
    // columns are somebody else's.
    if (warp == AT_SOFT / 32 && abort_flag && elect_one()) {
        tc_drain(&q_full, 0);
        for (int t = max(0, armed_k - AT_STAGES); t < armed_k; ++t) tc_drain(&k_full[t % AT_STAGES], (t / AT_STAGES) & 1);
        for (int t = max(0, armed_v - AT_STAGES); t < armed_v; ++t) tc_drain(&v_full[t % AT_STAGES], (t / AT_STAGES) & 1);
    }
    if (warp == AT_SOFT / 32 + 1) {
        if (abort_flag && elect_one()) {
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(at_smem(&drain_bar)) : "memory");
            tc_drain(&drain_bar, 0);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

cudaError_t launch_prefill_attn_tc(const CUtensorMap& q_hi, const CUtensorMap& q_lo, const CUtensorMap& k, const CUtensorMap& v, int layer, void* plane, int T,
                                   uint32_t* status, cudaStream_t st) {
    {
        static bool attr_set[64] = {};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
        if (!attr_set[dev]) {   // (a benign race between host threads: the attribute is set to the same value)
            e = cudaFuncSetAttribute(prefill_attn_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(prefill_attn_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM);
            if (e != cudaSuccess) return e;
            attr_set[dev] = true;
        }
    }
    // A launch takes as long as its longest query tile.  While there are SMs without a block, pairs of blocks share the longest ones, as many as still leave
    // every block resident at once (us a prompt, shared / not: 512 tokens 1379 / 1413, 777 1817 / 1874, 1088 1985 / 2013; tiles of two key tiles as well: 256
    // tokens 1099 / 1080; in two waves 1090 tokens 2105 / 2019, 1400 2606 / 2506).
    const int tiles = (T + AT_QT - 1) / AT_QT;
    const int long_ones = tiles - 2 * (AT_SPLIT_MIN - 1);        // query tiles of at least AT_SPLIT_MIN key tiles (every key tile is the last of two)
    const int one_wave = tc_sm_count() / KV_HEADS;               // blocks of a kv group that are resident at once, one on an SM: 18 of 148
    const int shared = min(one_wave - tiles, long_ones);
    if (shared > 0) {
        PrefillAttnTcArgs a{reinterpret_cast<bf16_raw*>(plane), T, layer, shared, status};
        return launch_chain_cluster(prefill_attn_tc_kernel<true>, dim3(2 * (shared + (tiles - shared + 1) / 2) * KV_HEADS), dim3(AT_THREADS), AT_SMEM, 2, st, q_hi, q_lo, k, v, a);
    }
    // one block per (query tile, kv group), dispatched in the order of their work (a query tile has 1..n key tiles), so that the
    // SMs that finish early pick up the light tiles: greedy longest-first over all SMs
    PrefillAttnTcArgs a{reinterpret_cast<bf16_raw*>(plane), T, layer, 0, status};
    return launch_chain(prefill_attn_tc_kernel<false>, dim3(tiles * KV_HEADS), dim3(AT_THREADS), AT_SMEM, st, q_hi, q_lo, k, v, a);
}

}  // namespace q3
