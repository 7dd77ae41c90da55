// The dense products of a layer for decode batches of at most 64 sequences: tcgen05 GEMMs whose k slices are the blocks of a
// cluster.
//
// With 1..64 tokens a layer's weights are a few megabytes per product, so what a launch costs is latency, and what a
// layer costs is the number of launches that wait for one another.  A product whose tiles are cut along K to occupy
// the GPU has to add its slices up again.  Adding them with fp32 atomics to global memory leaves the finished row to
// the NEXT launch, so every product drags a second launch behind it that normalises or applies SiLU, writes the bf16
// planes of the following product and clears the next sums.  Here the slices are the blocks of a cluster: each
// block sends its partial tile to the owners of the tokens (token t belongs to block t mod C) with bulk copies through
// distributed shared memory, and the owner adds the C partials in a fixed order and finishes the row: no atomics, no cleared
// buffers, the same result on every run, and five launches per layer (q/k/v, attention, Wo, gate/up, down) instead of
// eight or nine.
//
// The RMS norm commutes with the product: the planes hold x * gain, the producer of x (CL_RESID) also leaves 32 partial sums of
// squares per row, and the consumer's epilogue multiplies by rsqrt(mean + eps).
//
//   CL_QKV    128-row tiles of [Wq; Wk; Wv]: 32 tiles        qkv = (planes . W) * r
//   CL_RESID  64-row tiles of Wo or Wd: 16 tiles             x += planes . W; planes of x * gain; sums of squares
//   CL_SILU   64 rows of Wg and the same 64 of Wu: 48 tiles  planes of silu(gate * r) * (up * r)
//
// NACC: accumulators the k steps of a slice go to in turn.  The tensor core truncates every sum it adds to an accumulator, so the
// result is short by about half a unit in the last place a step; the epilogue adds the accumulators with rounding.  Fewer than
// Q3_TC_MIN_BATCH sequences take four, because the kernels that serve them otherwise add in fp32 or exactly: logits rel-L2 against
// fp64, two sequences at 16 / 1000 positions and three at 900, with two accumulators 1.31, 1.84 and 1.79e-6, with four 1.16, 1.66 and
// 1.66e-6 (with one, and the LM head truncating as well, 2.16, 2.70 and 2.68e-6); the persistent kernel, one sequence after the other,
// 1.23, 1.76 and 1.83e-6.  In larger batches the two planes of the attention leave 1.7e-5 whatever the products do.
//
// Measured (one B200, us per step, before -> after): 8 sequences x 1024 positions 984 -> 720, 64 x 1024 2333 -> 2055, one at
// 5000 positions 1606 -> 800.  What bounds it: a launch is about 3.4 us of latencies in series (8 sequences, medians of the blocks: release
// of the wait to the first stage 0.6, products 1.0, partial tile out 0.3, to the owners 0.5, finished row 0.3, end of the grid to the
// next release 1.0, each a little longer for the time stamps) beside 1..2 us of weight bytes that overlap them.
//
// Weight tiles are requested before the wait for the previous launch, so that their latency overlaps its tail.
//
// A wait that gives up (status words).  A block whose accumulator is not complete sends nothing and stores nothing; one that does
// not receive every partial stores nothing.  Whoever gave up still meets its cluster at every barrier, and a partial tile is only
// ever sent before the last one: behind it nobody sends any more, and a block that still lacks a partial waits once more, for
// copies that were on their way when it gave up, before it leaves.  The receivers' limit is twice the senders', so a
// late sender has given up or delivered before a receiver gives up.  The stages and TMEM are drained the same way.
#include <cuda.h>

#include "q3_engine.h"
#include "q3_gemm_cl.h"
#include "q3_gemm_tc.h"
#include "q3_tc_ptx.cuh"

namespace q3 {

constexpr int CL_THREADS = 192;   // warp 0: TMA, warp 1: MMA and TMEM, warps 2..5: epilogue
constexpr int CL_MAX_STAGES = 6;
constexpr unsigned long long CL_RED_WAIT_NS = 2 * TC_WAIT_NS;
constexpr int CL_FEW = 4;          // most tokens of the kernels with several accumulators
static_assert(Q3_TC_MIN_BATCH <= CL_FEW, "a batch below it fits");

struct ClusterGemmParams {
    int kb_total;                 // k blocks of 64
    int prow, n_tok, stages;
    int tiles_q, tiles_k;         // CL_QKV: tiles of the first two matrices
    float* out;
    int ldo;
    bf16_raw* planes;
    int ldp;
    const bf16_raw* gain;
    float* ssq;
    int ssq_ld;
    uint32_t* status;
};

__device__ __forceinline__ uint32_t cl_map(uint32_t smem_addr, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
    return a;
}
// (relaxed: no data is handed over by the cluster's barrier, only the mbarriers' initialisation, which has its own fence)
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

__device__ __forceinline__ void cl_store_planes(bf16_raw* p, size_t plane, float v) {
    const bf16_raw h = f_to_bf(v);
    const float r1 = v - bf_to_f(h);
    const bf16_raw m = f_to_bf(r1), l = f_to_bf(r1 - bf_to_f(m));
    p[0] = h;
    p[plane] = m;
    p[2 * plane] = l;
}

template <int KIND, int BN> struct ClShape {
    static constexpr int TM = KIND == CL_RESID ? 64 : 128;                                // rows of the weight tile
    static constexpr int C = KIND == CL_RESID ? 8 : 4;                                      // k slices = blocks of the cluster
    static constexpr int SLOTS = (BN + C - 1) / C;                                        // tokens a block owns
    static constexpr uint32_t ACC_COLS = CL_PLANES * BN <= 64 ? 64 : 128;                 // TMEM columns of an accumulator
    static constexpr int RED_BYTES = C * SLOTS * TM * 4;                                  // partial tiles of the owned tokens
};

template <int KIND, int BN, int NACC>
__global__ void __launch_bounds__(CL_THREADS, 1) gemm_cluster_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
                                                                     const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_x,
                                                                     const ClusterGemmParams p) {
    using S = ClShape<KIND, BN>;
    constexpr int TM = S::TM, C = S::C, SLOTS = S::SLOTS;
    constexpr uint32_t A_BYTES = TM * TC_BK * 2, B_BYTES = BN * TC_BK * 2;
    extern __shared__ __align__(1024) unsigned char cl_raw[];
    __shared__ __align__(8) uint64_t full_bar[CL_MAX_STAGES], empty_bar[CL_MAX_STAGES], acc_bar, red_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag;
    __shared__ float s_r[SLOTS];

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x;                 // the cluster spans x
    const int tile = blockIdx.y, n0 = blockIdx.z * BN;
    const int stages = p.stages;
    const int base_kb = p.kb_total / C, rem_kb = p.kb_total % C;
    const int kb0 = rank * base_kb + min(rank, rem_kb), nkb = base_kb + (rank < rem_kb ? 1 : 0);
    constexpr uint32_t stage_bytes = A_BYTES + CL_PLANES * B_BYTES;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(cl_raw) + 1023) & ~(uintptr_t)1023);
    float* red = reinterpret_cast<float*>(base + (size_t)stages * stage_bytes);      // [C][SLOTS][TM]: what the blocks send to this one
    auto slots_of = [&](int owner) { return max(0, (min(p.n_tok - n0, BN) - owner + C - 1) / C); };   // tokens of this tile that `owner` finishes
    const int my_slots = slots_of(rank);

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&full_bar[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&empty_bar[s])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&acc_bar)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&red_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (my_slots > 0)
            asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&red_bar)), "r"((uint32_t)(C * my_slots * TM * 4)) : "memory");
        abort_flag = 0;
    }
    // the planes of a stage lie side by side: columns of one B operand
    constexpr uint32_t cols = CL_PLANES * BN, acc_cols = S::ACC_COLS, tmem_cols = NACC * acc_cols;
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tmem_base_s)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    // The attention launch that follows q/k/v reads lengths and cache rows before it waits: it may start only once everything
    // before this launch has completed (below).  The others' successors read nothing but weights early.
    if (KIND != CL_QKV) pdl_launch();
    cl_arrive();      // (matched before the first remote copy: every block of the cluster has set its barriers up by then)

    const int te = (int)threadIdx.x - 64;        // 0..127 in the epilogue warps
    constexpr int OSTEP = KIND == CL_QKV ? 1 : 2;                   // threads finish `OSTEP` owned tokens side by side
    constexpr int PER = (SLOTS + OSTEP - 1) / OSTEP;                // owned tokens a thread finishes
    const int orow = KIND == CL_QKV ? te : te & 63, osub = KIND == CL_QKV ? 0 : te >> 6;
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        int armed = 0;                           // k blocks whose loads have been requested
        const bool one = elect_one();
        if (one) {
            const CUtensorMap* tm_w = &tm_w0;
            int m0 = tile * TM;
            if (KIND == CL_QKV) {
                if (tile >= p.tiles_q) { tm_w = &tm_w1; m0 -= p.tiles_q * TM; }
                if (tile >= p.tiles_q + p.tiles_k) { tm_w = &tm_w2; m0 -= p.tiles_k * TM; }
            }
            if (KIND == CL_SILU) m0 = tile * (TM / 2);
            auto weights = [&](int kb, int s) {
                const uint32_t st = tc_smem(base + (size_t)s * stage_bytes);
                asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(&full_bar[s])), "r"(stage_bytes) : "memory");
                tc_load_box(st, tm_w, (kb0 + kb) * TC_BK, m0, &full_bar[s]);
                if (KIND == CL_SILU) tc_load_box(st + A_BYTES / 2, &tm_w1, (kb0 + kb) * TC_BK, m0, &full_bar[s]);
                armed = kb + 1;
            };
            const int ahead = min(nkb, stages);
            for (int kb = 0; kb < ahead; ++kb) weights(kb, kb);
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_x) : "memory");
            pdl_wait();
            if (KIND == CL_QKV) pdl_launch();
            for (int kb = 0, s = 0, turn = 0; kb < nkb; ++kb, ++s) {
                if (s == stages) { s = 0; ++turn; }
                if (turn > 0) {
                    if (!tc_wait(&empty_bar[s], (turn - 1) & 1, &abort_flag, p.status, 50)) break;
                    weights(kb, s);
                }
                tc_load_planes(tc_smem(base + (size_t)s * stage_bytes) + A_BYTES, &tm_x, (kb0 + kb) * TC_BK, n0, &full_bar[s]);
            }
        }
        __syncwarp();
        cl_wait();
        cl_arrive();
        cl_wait();
        if (one && abort_flag)                   // (the last `stages` of them may still be on their way)
            for (int kb = max(0, armed - stages); kb < armed; ++kb) tc_drain(&full_bar[kb % stages], (kb / stages) & 1);
        return;
    }
    if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((cols >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
            // (descriptors count 16-byte units: a k step of 16 elements is 2 of them, a stage stage_bytes / 16)
            const uint64_t da0 = tc_desc(tc_smem(base)), db0 = tc_desc(tc_smem(base) + A_BYTES);
            uint64_t ds = 0;
            for (int kb = 0, s = 0, phase = 0; kb < nkb; ++kb, ++s, ds += stage_bytes >> 4) {
                if (s == stages) { s = 0; phase ^= 1; ds = 0; }
                if (!tc_wait(&full_bar[s], phase, &abort_flag, p.status, 51)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k) {
                    const uint64_t da = da0 + ds + 2 * k, db = db0 + ds + 2 * k;
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                                 ::"r"(tmem_base + (uint32_t)(k % NACC) * acc_cols), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)(kb | (k / NACC))), "r"(0u), "r"(0u), "r"(0u), "r"(0u) : "memory");
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&empty_bar[s])) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&acc_bar)) : "memory");
        }
        __syncwarp();
        cl_wait();
        asm volatile("bar.sync 2, 160;" ::: "memory");              // the epilogue warps have read the accumulator
        if (abort_flag) tc_drain(&acc_bar, 0);                      // ... or gave it up: the products that were issued end first
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
        cl_arrive();
        cl_wait();
        return;
    }

    // ---------------------------------------------------------------------- epilogue
    const float gain = KIND == CL_RESID ? bf_to_f(p.gain[tile * TM + orow]) : 0.f;
    const int quad = warp & 3;                   // TMEM lanes [32 quad, 32 quad + 32) belong to this warp
    const size_t plane = (size_t)p.prow * p.ldp;
    float xr[KIND == CL_RESID ? PER : 1];
    pdl_wait();
    // while the products run: the scale of the owned rows, or the residual they are added to
    if (KIND != CL_RESID) {
#pragma unroll 4
        for (int s = warp - 2; s < my_slots; s += 4) {
            const float ss = warp_sum(p.ssq[(size_t)lane * p.ssq_ld + n0 + s * C + rank]);
            if (lane == 0) s_r[s] = rsqrtf(ss / (float)HIDDEN + EPS);
        }
    } else {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int s = osub + i * OSTEP;
            xr[i] = s < my_slots ? p.out[(size_t)(n0 + s * C + rank) * p.ldo + tile * TM + orow] : 0.f;
        }
    }
    // (the MMA thread commits to acc_bar after a wait of its own gave up, too, so that its products can be drained: the flag tells)
    const bool summed = __all_sync(0xffffffffu, tc_wait_warp(&acc_bar, 0, &abort_flag, p.status, 52) && !abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // The partial tile goes to this block's staging area (the stages are free: every MMA has completed), token by token and
    // grouped by owner, and from there to the owners with one bulk copy each, counted on the owner's mbarrier.
    // (a tile of 64 rows occupies the first 16 lanes of every 32-lane quarter)
    if (summed) {
        const bool live = TM == 128 || lane < 16;
        float* stage = reinterpret_cast<float*>(base) + (TM == 128 ? quad * 32 + lane : quad * 16 + (lane & 15));   // [C][SLOTS][TM]
        if constexpr (NACC > 1) {            // at most CL_FEW tokens: their columns of every accumulator and plane under one wait
            uint32_t r[NACC][CL_PLANES][CL_FEW];
#pragma unroll
            for (int ac = 0; ac < NACC; ++ac)
#pragma unroll
                for (int sp = 0; sp < 3; ++sp) tc_ld4(r[ac][sp], tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)ac * acc_cols + sp * BN);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < CL_FEW; ++j) {
                float v[3];
#pragma unroll
                for (int sp = 0; sp < 3; ++sp) {
                    v[sp] = __uint_as_float(r[0][sp][j]);
#pragma unroll
                    for (int ac = 1; ac < NACC; ++ac) v[sp] += __uint_as_float(r[ac][sp][j]);
                }
                if (live) stage[((j % C) * SLOTS + j / C) * TM] = v[0] + (v[1] + v[2]);
            }
        } else {
        constexpr int STEP = BN < 32 ? BN : 32;
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += STEP) {
            if (n0 + c0 >= p.n_tok) break;
            uint32_t r[32], q1[32], q2[32];
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
            if constexpr (STEP == 16) {
                tc_ld16(r, taddr);
                tc_ld16(q1, taddr + BN);
                tc_ld16(q2, taddr + 2 * BN);
            } else {
                tc_ld32(r, taddr);
                tc_ld32(q1, taddr + BN);
                tc_ld32(q2, taddr + 2 * BN);
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < STEP; ++j) {
                const float v = __uint_as_float(r[j]) + __uint_as_float(q1[j]) + __uint_as_float(q2[j]);
                if (live) stage[(((c0 + j) % C) * SLOTS + (c0 + j) / C) * TM] = v;
            }
        }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.arrive 2, 160;" ::: "memory");
    cl_wait();                                   // every block of the cluster has set its mbarrier up
    asm volatile("bar.sync 1, 128;" ::: "memory");
    const bool whole = !abort_flag;               // no warp of this block gave up on the accumulator
    if (whole && te < C && slots_of(te) > 0) {
        const uint32_t src = tc_smem(base) + (uint32_t)(te * SLOTS * TM * 4);
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(cl_map(tc_smem(red + (size_t)rank * SLOTS * TM), te)), "r"(src), "r"((uint32_t)(slots_of(te) * TM * 4)), "r"(cl_map(tc_smem(&red_bar), te)) : "memory");
    }
    __syncwarp();
    const bool received = my_slots > 0 && whole && tc_wait_warp(&red_bar, 0, &abort_flag, p.status, 53, CL_RED_WAIT_NS);
    cl_arrive();      // (matched before the exit: this block sends nothing any more)

    // the owned tokens: add the slices in order and finish the row
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int s = osub + i * OSTEP, t = n0 + s * C + rank;
        if (s >= my_slots || !received) break;
        const float* src = red + s * TM + orow;
        float v = src[0];
#pragma unroll
        for (int c = 1; c < C; ++c) v += src[c * SLOTS * TM];
        if (KIND == CL_QKV) {
            p.out[(size_t)t * p.ldo + tile * TM + orow] = v * s_r[s];
        } else if (KIND == CL_RESID) {
            const float x = xr[i] + v;
            const size_t col = (size_t)tile * TM + orow;
            p.out[(size_t)t * p.ldo + col] = x;
            cl_store_planes(p.planes + (size_t)t * p.ldp + col, plane, x * gain);
            const float ss = warp_sum(x * x);
            if (lane == 0) p.ssq[(size_t)(tile * 2 + (orow >> 5)) * p.ssq_ld + t] = ss;
        } else {
            float u = src[TM / 2];
#pragma unroll
            for (int c = 1; c < C; ++c) u += src[c * SLOTS * TM + TM / 2];
            const float g = v * s_r[s];
            u *= s_r[s];
            cl_store_planes(p.planes + (size_t)t * p.ldp + tile * (TM / 2) + orow, plane, (g / (1.f + expf(-g))) * u);
        }
    }
    cl_wait();
    if (my_slots > 0 && !received && te == 0) tc_drain(&red_bar, 0);
}

// ---- embedding gather with the first layer's planes: one block per sequence ----------------------------------------
__global__ void __launch_bounds__(256) embed_planes_kernel(const long long* __restrict__ token, const bf16_raw* __restrict__ embed, int vocab, float* __restrict__ x,
                                                           const bf16_raw* __restrict__ gain, bf16_raw* __restrict__ planes, int prow,
                                                           float* __restrict__ ssq, int ssq_ld, uint32_t* status, unsigned long long* argmax_keys,
                                                           unsigned* argmax_tickets, const int* __restrict__ seq_len, int len_bound) {
    pdl_launch();
    pdl_wait();
    const int b = blockIdx.x, tid = threadIdx.x;
    if (tid == 0 && seq_len != nullptr && (seq_len[b] > len_bound || seq_len[b] < 0)) report(status, ST_BAD_LEN, 1000, (uint32_t)seq_len[b]);
    if (tid == 0 && argmax_keys != nullptr) { argmax_keys[b] = 0ull; argmax_tickets[b] = 0u; }
    long long t = token[b];
    if (t < 0 || t >= vocab) {
        if (tid == 0) report(status, ST_BAD_TOKEN, 0, (uint32_t)t);
        t = 0;
    }
    const uint2 v = reinterpret_cast<const uint2*>(embed + (size_t)t * HIDDEN)[tid], g = reinterpret_cast<const uint2*>(gain)[tid];   // 4 bf16 each
    const float4 o = make_float4(bf_lo(v.x), bf_hi(v.x), bf_lo(v.y), bf_hi(v.y));
    reinterpret_cast<float4*>(x + (size_t)b * HIDDEN)[tid] = o;
    const float y[4] = {o.x * bf_lo(g.x), o.y * bf_hi(g.x), o.z * bf_lo(g.y), o.w * bf_hi(g.y)};
#pragma unroll
    for (int i = 0; i < 4; ++i) cl_store_planes(planes + (size_t)b * HIDDEN + tid * 4 + i, (size_t)prow * HIDDEN, y[i]);
    float ss = fmaf(o.x, o.x, fmaf(o.y, o.y, fmaf(o.z, o.z, o.w * o.w)));
#pragma unroll
    for (int sh = 4; sh > 0; sh >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, sh);   // eight threads make a part of 32 elements
    if ((tid & 7) == 0) ssq[(size_t)(tid >> 3) * ssq_ld + b] = ss;
}

cudaError_t launch_embed_planes(const long long* token, const bf16_raw* embed, int vocab, float* x, const bf16_raw* gain, bf16_raw* planes, int prow,
                                float* ssq, int ssq_ld, uint32_t* status, int batch, cudaStream_t st, unsigned long long* argmax_keys,
                                unsigned* argmax_tickets, const int* seq_len, int len_bound) {
    return launch_chain(embed_planes_kernel, dim3(batch), dim3(256), 0, st, token, embed, vocab, x, gain, planes, prow, ssq, ssq_ld, status,
                        argmax_keys, argmax_tickets, seq_len, len_bound);
}

// ---- host side ------------------------------------------------------------------------------------------------------
// Tokens per tile.  Wider tiles need more shared memory than the neighbouring launches leave: batch 64 x 1024 with tiles of 16 / 32 /
// 64: 2419 / 2075 / 2349 us per step.
static int cl_tile(int n_tok) { return n_tok <= 16 ? 16 : 32; }

// (a plane's rows are the LM head's token tile, which reads the last planes)
int gemm_cluster_rows(int n_tok) { return n_tok <= 32 ? 32 : CL_MAX_TOK; }

template <int KIND, int BN, int NACC>
static cudaError_t launch_cl(const CUtensorMap* tw, const CUtensorMap& tx, ClusterGemmParams p, int tiles, cudaStream_t st) {
    using S = ClShape<KIND, BN>;
    constexpr int MAX_SMEM = 220 * 1024;
    static bool attr_set[64] = {};   // (a benign race between host threads: the same value is written)
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        if ((e = cudaFuncSetAttribute(gemm_cluster_kernel<KIND, BN, NACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM)) != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    constexpr int stage_bytes = S::TM * TC_BK * 2 + CL_PLANES * BN * TC_BK * 2;
    // Half of an SM's shared memory, so that the next launch's blocks find room while this one's are still there: they set up
    // and fetch their weights before they wait (batch 64 x 1024, 75 / 90 / 112 KB: 2118 / 2104 / 2075 us per step; 27 ragged
    // up to 2048: 1460 / 1437 / 1383 us).
    int stages = (112 * 1024 - S::RED_BYTES - 1024) / stage_bytes;
    const int nkb = (p.kb_total + S::C - 1) / S::C;
    if (stages > nkb) stages = nkb;
    if (stages > CL_MAX_STAGES) stages = CL_MAX_STAGES;
    const int need = (S::RED_BYTES + stage_bytes - 1) / stage_bytes;   // the stages also hold the outgoing partial tile
    if (stages < need) stages = need;
    p.stages = stages;
    // A block holds its TMEM columns until its whole cluster has met, so every block on an SM has to get its columns without waiting
    // for another's: whatever cluster products share an SM, of this launch, of its neighbours in the stream or of an engine on
    // another stream, their columns never exceed the SM's 512.  Every block asks for so much shared memory that at most three fit, and one with
    // 256 columns for so much that no third fits beside two of them: 3 x 128 or 256 + 2 x 128 or 2 x 256 at most.  The
    // layer kernel (q3_layer_tc.cu), whose blocks wait for one another too, leaves room for one block of 128 columns beside its
    // 128.  The other kernels with TMEM wait for nothing but their predecessor in the stream, which has all its columns by then.
    constexpr int SM_SMEM = 228 * 1024, THIRD = 58 * 1024, HALF = 88 * 1024;
    static_assert(4 * THIRD > SM_SMEM && 2 * HALF + THIRD > SM_SMEM && NACC * S::ACC_COLS <= 256, "TMEM columns of an SM");
    int smem = stages * stage_bytes + S::RED_BYTES + 1024;
    constexpr int least = NACC * S::ACC_COLS > 128 ? HALF : THIRD;
    if (smem < least) smem = least;
    return launch_chain_cluster(gemm_cluster_kernel<KIND, BN, NACC>, dim3(S::C, tiles, (p.n_tok + BN - 1) / BN), dim3(CL_THREADS), (size_t)smem, S::C, st,
                                tw[0], tw[1], tw[2], tx, p);
}

template <int KIND>
static cudaError_t launch_kind(const CUtensorMap* tw, const CUtensorMap& tx, const ClusterGemmParams& p, int tiles, int bn, cudaStream_t st) {
    if (p.n_tok < Q3_TC_MIN_BATCH) return launch_cl<KIND, 16, 4>(tw, tx, p, tiles, st);
    if (bn == 16) return launch_cl<KIND, 16, 1>(tw, tx, p, tiles, st);
    return launch_cl<KIND, 32, 1>(tw, tx, p, tiles, st);
}

cudaError_t launch_gemm_cluster(const ClusterGemmCall& c, cudaStream_t st) {
    const int bn = cl_tile(c.n_tok);
    if (c.n_tok < 1 || c.n_tok > CL_MAX_TOK || c.K % TC_BK || c.K < 8 * TC_BK || c.prow < gemm_cluster_rows(c.n_tok) || c.prow % bn)
        return cudaErrorInvalidValue;
    ClusterGemmParams p{};
    p.kb_total = c.K / TC_BK; p.prow = c.prow; p.n_tok = c.n_tok;
    p.out = c.out; p.planes = c.planes; p.gain = c.gain; p.ssq = c.ssq; p.ssq_ld = c.ssq_ld; p.status = c.status;
    CUtensorMap tw[3], tx;
    if (!tc_cached_map(c.in, (uint64_t)c.prow, (uint64_t)c.K, (uint32_t)bn, &tx, (uint64_t)CL_PLANES)) return cudaErrorUnknown;
    const int rows[3] = {c.kind == CL_QKV ? Q_DIM : c.kind == CL_RESID ? HIDDEN : INTER, c.kind == CL_QKV ? KV_DIM : INTER, KV_DIM};
    const int n_w = c.kind == CL_QKV ? 3 : c.kind == CL_RESID ? 1 : 2;
    const uint32_t box = c.kind == CL_QKV ? 128u : 64u;
    for (int i = 0; i < 3; ++i) {
        if (i >= n_w) tw[i] = tw[0];
        else if (!tc_cached_map(c.w[i], (uint64_t)rows[i], (uint64_t)c.K, box, &tw[i])) return cudaErrorUnknown;
    }
    switch (c.kind) {
        case CL_QKV:
            p.tiles_q = Q_DIM / 128; p.tiles_k = KV_DIM / 128; p.ldo = QKV_DIM;
            return launch_kind<CL_QKV>(tw, tx, p, QKV_DIM / 128, bn, st);
        case CL_RESID:
            p.ldo = HIDDEN; p.ldp = HIDDEN;
            return launch_kind<CL_RESID>(tw, tx, p, HIDDEN / 64, bn, st);
        case CL_SILU:
            p.ldp = INTER;
            return launch_kind<CL_SILU>(tw, tx, p, INTER / 64, bn, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace q3
