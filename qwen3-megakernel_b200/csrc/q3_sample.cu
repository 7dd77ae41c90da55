// Temperature / top-k sampling over the fp32 logits a decode step writes.
//
// The reference decodes greedily inside its kernel and leaves sampling to the caller, who gets the fp32
// logits for that purpose (csrc/qwen3_step.cu:175 writes them, qwen3mk/kernel.py:44-50 returns them).  This is
// that next step on the GPU, so that a sampled token can feed the following launch without a trip to the host.
//
// A CLUSTER of blocks per row: block r of C owns a contiguous slice of the row, warp w of it a contiguous run of the
// slice, so that sums over (block, warp, group of 32) follow the index order and every load is coalesced.  What the
// blocks of a row have to agree on travels through distributed shared memory, one cluster barrier each:
//   1. every block finds its maximum.  Where the whole vocabulary takes part, it sums its weights exp((l_i - max) / T) under its own maximum,
//      in the same pass over memory where a thread's words do not fit its registers (a thread's sum is scaled when its maximum
//      grows); maxima and sums are exchanged together and the blocks' sums scaled to the row's maximum;
//   2. top-k: a block whose threads have at least k elements bins its THREADS' maxima linearly between the smallest and
//      the largest of them; the bins that hold the k largest maxima bound its own k largest elements from below, so the
//      few elements at or above that bound (about 1.1 k of them) are the block's candidates, in the order of their indices.  The union of all blocks'
//      candidates contains every word that is kept; every block finds the threshold among them (binary search over the bits of
//      the keys, held in registers, below the bits they share and until exactly k are above it) and adds up the weights of the kept
//      ones, list by list, in the same order as every other block.  A row whose candidates do not fit (large k, many equal values) goes
//      through a radix select instead: three passes of 11, 11 and 10 bits over the order-preserving integer image of the
//      floats, histograms summed over the cluster, then the weights' sums.  Every logit >= the k-th value is kept, so ties are all kept;
//   3. the token is the first index whose inclusive prefix sum exceeds u * total, u in [0, 1) supplied per row
//      by the caller (a seeded generator on the host side keeps runs reproducible); the block whose words
//      bracket the target finds it among its candidates, a thread each, or walks the run of the warp that brackets it.  Only a word with a
//      weight above zero (in fp32, under the row's maximum) is drawn, and the same numbers draw the same word on every run.
// T <= 0 or k == 1 degenerate to the arg-max (ties -> lowest index), like the decode kernels.
//
// A single row is bound by latency (0.6 MB, but a dozen dependent block-wide steps), a full batch by the row's bytes and the same steps.
// Measured, us: 1 row, k = 50: 10.8 to 11.6 from box to box on changing logits (11.4 to 12.2 before a warp took its largest value in one instruction); 15 / 36 / 64 rows, whole vocabulary: 12.6 / 18.9 / 18.6 (before a run's last loads left together, four words a thread
// in the walk, and up to 64 rows the next loads under way behind the ones at work: 13.8 / 20.7 / 20.7); 15 / 36 / 64 rows, k = 50: 15.1 / 18.7 / 18.7 (before
// lanes shared the second look at the row: 16.6 / 22.8 / 24.8).
#include <cooperative_groups.h>

#include <cfloat>

#include "q3_engine.h"

namespace cg = cooperative_groups;

namespace q3 {

constexpr int SAMPLE_THREADS = 1024;
constexpr int SAMPLE_WARPS = SAMPLE_THREADS / 32;
constexpr int SAMPLE_MAX_CLUSTER = 16;
constexpr int SAMPLE_BINS = 2048;
constexpr int SAMPLE_CAND = 1024;     // candidates a block publishes
constexpr int SAMPLE_KEYS = 4;        // candidates of all blocks a thread holds in the search: 4096 in all

__device__ __forceinline__ unsigned ordered_key(float f) {   // monotonic in the float's value
    const unsigned b = __float_as_uint(f);
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}

__device__ __forceinline__ float key_value(unsigned k) { return __uint_as_float((k >> 31) ? k ^ 0x80000000u : ~k); }   // the inverse

// the largest of a warp's values (one instruction; a NaN loses to any number, as in fmaxf)
__device__ __forceinline__ float row_max(float v) {
    float m;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(v));
    return m;
}

// elements of a warp's run when a row of `vocab` words goes to `cluster` blocks
__host__ __device__ inline int sample_run(int vocab, int cluster) {
    return ((vocab + cluster * SAMPLE_WARPS - 1) / (cluster * SAMPLE_WARPS) + 127) / 128 * 128;
}

struct SampleShared {
    float bmax[SAMPLE_MAX_CLUSTER];         // per block of the cluster: its maximum, ...
    int bidx[SAMPLE_MAX_CLUSTER];           // ... where it is, ...
    int ncand[SAMPLE_MAX_CLUSTER];          // ... how many candidates it has (-1: they did not fit), ...
    float bsum[SAMPLE_MAX_CLUSTER];         // ... and the sum of its weights
    float wf[SAMPLE_WARPS], wg[SAMPLE_WARPS];
    int wi[SAMPLE_WARPS];
    unsigned wcount[2][SAMPLE_WARPS];
    unsigned hist[SAMPLE_BINS];
    unsigned cand[SAMPLE_CAND];             // keys
    int candi[SAMPLE_CAND];                 // and where they are
    __align__(16) float weight[SAMPLE_KEYS * SAMPLE_THREADS];   // weights of all blocks' candidates, the lists one after the other (before that, the block's own list unordered)
    unsigned sel, need, cand_n, cmin;
};

// Block-wide: the bin, counted from the largest, in which the running count of hist[] reaches `need`, and what is still
// needed inside it (sh.sel, sh.need).  from_top: bins run from SAMPLE_BINS - 1 down, else from 0 up.
__device__ __forceinline__ void find_bin(SampleShared& sh, unsigned c0, unsigned c1, unsigned need, bool from_top) {
    // thread t holds the counts of the bins of rank 2 t and 2 t + 1 in walking order
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned mine = c0 + c1;
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) sh.wcount[0][warp] = incl;
    if (tid == 0) { sh.sel = from_top ? 0u : (unsigned)SAMPLE_BINS - 1u; sh.need = need; }   // (fewer than `need` keys in all: everything)
    __syncthreads();
    const unsigned w = sh.wcount[0][lane];
    unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + incl - mine;
    if (before < need && before + mine >= need) {
        const bool second = before + c0 < need;
        const int rank = 2 * tid + (second ? 1 : 0);
        if (second) before += c0;
        sh.sel = (unsigned)(from_top ? SAMPLE_BINS - 1 - rank : rank);
        sh.need = need - before;
    }
    __syncthreads();
}

// Elements are dealt out in groups of 128 per warp, four neighbours a lane: element 4 lane + q of group j.  NQ > 0: a thread's
// elements of the row (at most NQ groups) stay in registers; NQ == 0: every pass reads the row again (from L2).  TWO: two blocks an SM (32 registers a
// thread).  SHARE: the threads with candidates read again with the help of their warp.
template <int NQ, bool TWO, bool SHARE>
__global__ void __launch_bounds__(SAMPLE_THREADS, TWO ? 2 : 1) sample_kernel(const float* __restrict__ logits, int vocab, float temperature, int top_k,
                                                                             const float* __restrict__ uniform, long long* __restrict__ out) {
    constexpr int WALK = NQ > 0 || (TWO && !SHARE) ? 1 : 4;     // words a thread takes of the run that is walked (a run of up to 640, and where registers are short: one)
    __shared__ SampleShared sh;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row_id = blockIdx.x / C;
    const float* row = logits + (size_t)row_id * vocab;
    // warp w of block r: elements [i0, i1), `per` of them but for the last runs of the row
    const int per = sample_run(vocab, C);
    const int i0 = (int)min((long long)vocab, (long long)(rank * SAMPLE_WARPS + warp) * per), i1 = min(vocab, i0 + per);
    // 0: the arg-max, 1: the k largest words take part, 2: all do.  (Opaque to the compiler: built by nvcc 12.9 from flags whose
    // terms it could see, an earlier form of this kernel failed every top-k test, as if the threshold had been skipped.  Why is not known: neither a
    // smaller case nor a fault in the source was found.)
    int mode = !(temperature > 0.f) || top_k == 1 ? 0 : top_k > 1 && top_k < vocab ? 1 : 2;
    asm volatile("" : "+r"(mode));
    const bool greedy = mode == 0, select = mode == 1;
    const bool vec = ((vocab & 3) | (int)(reinterpret_cast<uintptr_t>(logits) & 15)) == 0;
    cluster.barrier_arrive();   // (a peer's shared memory may be written once the peer runs: waited for before the first exchange)

    auto fetch = [&](int j, int of) -> float4 {  // group j of lane `of`; elements past the run are -inf, which no pass below counts
        const int i = i0 + 128 * j + 4 * of;
        if (vec && i + 3 < i1) return *reinterpret_cast<const float4*>(row + i);
        float4 v;
        v.x = i < i1 ? row[i] : -INFINITY; v.y = i + 1 < i1 ? row[i + 1] : -INFINITY;
        v.z = i + 2 < i1 ? row[i + 2] : -INFINITY; v.w = i + 3 < i1 ? row[i + 3] : -INFINITY;
        return v;
    };
    float4 x[NQ > 0 ? NQ : 1];
    if constexpr (NQ > 0) {
#pragma unroll
        for (int j = 0; j < NQ; ++j) x[j] = fetch(j, lane);
    }
    const int groups = (i1 - i0 + 127) / 128, whole = vec ? (i1 - i0) / 128 : 0;
    // NQ == 0: f(first group, four groups' elements) over the run.  The loads of the next four groups are under way while these are at work where the
    // registers allow it (a block an SM), and the last ones leave together.
    auto batches = [&](auto&& f) {
        auto load = [&](int j, float4 (&v)[4]) {
            if (j + 4 <= whole) {                  // (no guards)
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = *reinterpret_cast<const float4*>(row + i0 + 128 * (j + q) + 4 * lane);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = fetch(j + q, lane);
            }
        };
        float4 v[2][4];
        if (groups > 0) load(0, v[0]);
        for (int j = 0; j < groups; j += 8) {
            if (j + 4 < groups) load(j + 4, v[1]);
            f(j, v[0]);
            if (j + 8 < groups) load(j + 8, v[0]);
            if (j + 4 < groups) f(j + 4, v[1]);
        }
    };
    auto each = [&](auto&& f) {          // f(index, value) over this thread's elements, in ascending order
        auto four = [&](int j, const float4& v) {
            const int i = i0 + 128 * j + 4 * lane;
            f(i, v.x); f(i + 1, v.y); f(i + 2, v.z); f(i + 3, v.w);
        };
        if constexpr (NQ > 0) {
#pragma unroll
            for (int j = 0; j < NQ; ++j) four(j, x[j]);
        } else {
            if constexpr (TWO) {
                int j = 0;
                for (; j + 4 <= whole; j += 4) {   // (no guards: the four loads leave together)
                    float4 v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = *reinterpret_cast<const float4*>(row + i0 + 128 * (j + q) + 4 * lane);
#pragma unroll
                    for (int q = 0; q < 4; ++q) four(j + q, v[q]);
                }
                for (; j < groups; ++j) four(j, fetch(j, lane));
            } else {
                batches([&](int j, const float4 (&v)[4]) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) four(j + q, v[q]);
                });
            }
        }
    };

    // ---- 1. the block's maximum, and the smallest of its threads' maxima ----
    const bool any = i0 + 4 * lane < i1;
    const float inv_t = 1.f / temperature;
    const bool whole_row = mode == 2;
    float mine = -INFINITY, wsum = 0.f;
    bool nan = false;
    // (a logit that is no number makes a sum one, too: below; a word masked with -inf weighs nothing at any temperature, and so does what
    // lies past the end of a run: with 1 / T = 0 the exponential of the product would be NaN, not 0)
    auto weight = [&](float v, float top) { return v < -FLT_MAX ? 0.f : __expf((v - top) * inv_t); };
    if (NQ == 0 && whole_row) {
        // maximum and sum of weights in one pass over memory: the sum is taken under the running maximum and scaled when that grows
        auto raise = [&](float top) {
            if (top > mine) { if (mine > -INFINITY) wsum *= __expf((mine - top) * inv_t); mine = top; }
        };
        auto top4 = [&](const float4& v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); };
        auto add4 = [&](const float4& v) { wsum += (weight(v.x, mine) + weight(v.y, mine)) + (weight(v.z, mine) + weight(v.w, mine)); };
        auto sixteen = [&](const float4 (&v)[4]) {
            raise(fmaxf(fmaxf(top4(v[0]), top4(v[1])), fmaxf(top4(v[2]), top4(v[3]))));
#pragma unroll
            for (int q = 0; q < 4; ++q) add4(v[q]);
        };
        if constexpr (TWO) {
            int j = 0;
            for (; j + 4 <= whole; j += 4) {
                float4 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = *reinterpret_cast<const float4*>(row + i0 + 128 * (j + q) + 4 * lane);
                sixteen(v);
            }
            for (; j < groups; ++j) { const float4 v = fetch(j, lane); raise(top4(v)); add4(v); }
        } else {
            batches([&](int, const float4 (&v)[4]) { sixteen(v); });
        }
    } else {
        each([&](int, float v) { mine = fmaxf(mine, v); nan = nan || v != v; });
    }
    {
        const float bv = row_max(mine), lo = -row_max(any ? -mine : -INFINITY);
        if (lane == 0) { sh.wf[warp] = bv; sh.wg[warp] = lo; }
    }
    if (select)
        for (int b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) sh.hist[b] = 0u;
    if (tid == 0) { sh.cand_n = 0u; sh.need = 0x7fffffffu; sh.cmin = 0xffffffffu; }
    const int n_thr = __syncthreads_count(any);     // threads that have an element
    const float bmax = row_max(sh.wf[lane]), blo = -row_max(-sh.wg[lane]);

    // ---- 2a. the block's candidates for the k largest ----
    int n_cand = -1;
    if (select) {
        const float scale = (float)(SAMPLE_BINS - 1) / (bmax - blo);
        auto bin = [&](float v) -> int {            // non-increasing in v; anything odd (an infinite range) lands inside the bounds
            const float d = (bmax - v) * scale;
            return d >= 0.f ? (int)fminf(d, (float)(SAMPLE_BINS - 1)) : 0;
        };
        if (top_k <= n_thr) {
            unsigned* const raw = reinterpret_cast<unsigned*>(sh.weight);    // the candidates as they come: keys, then indices
            raw[SAMPLE_CAND + tid] = 0xffffffffu;
            if (any) atomicAdd(&sh.hist[bin(mine)], 1u);
            __syncthreads();
            find_bin(sh, sh.hist[2 * tid], sh.hist[2 * tid + 1], (unsigned)top_k, false);
            const int last = (int)sh.sel;
            auto take = [&](int i, float v) {
                if (bin(v) <= last && i < i1) {
                    const unsigned n = atomicAdd(&sh.cand_n, 1u), key = ordered_key(v);
                    if (n < SAMPLE_CAND) { raw[n] = key; raw[SAMPLE_CAND + n] = (unsigned)i; }
                    atomicMin(&sh.cmin, key);
                }
            };
            const bool has = any && bin(mine) <= last;          // (a thread whose maximum is below the bound has no candidate)
            if constexpr (!SHARE) {
                if (has) each(take);
            } else {
                // The few threads that have some read their elements again, all of a thread's groups at once: a lane a group, four threads' loads
                // under way.
                for (unsigned m = __ballot_sync(0xffffffffu, has); m; ) {
                    int of[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) { of[q] = m ? __ffs(m) - 1 : -1; m &= m - 1; }
                    for (int j = lane; j < groups; j += 32) {
                        float4 v[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (of[q] >= 0) v[q] = fetch(j, of[q]);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int i = i0 + 128 * j + 4 * of[q];
                            if (of[q] >= 0) { take(i, v[q].x); take(i + 1, v[q].y); take(i + 2, v[q].z); take(i + 3, v[q].w); }
                        }
                    }
                }
            }
            __syncthreads();
            // In the order of their indices: sums of weights must not depend on which thread came first.  (A list is about 1.1 k words long.)
            const int n = (int)sh.cand_n;
            if (n <= SAMPLE_CAND && tid < n) {
                const unsigned at = raw[SAMPLE_CAND + tid];
                int place = 0;
#pragma unroll 4
                for (int j = 0; j < n; j += 4) {
                    const uint4 o = *reinterpret_cast<const uint4*>(raw + SAMPLE_CAND + j);
                    place += (o.x < at) + (o.y < at) + (o.z < at) + (o.w < at);
                }
                sh.cand[place] = raw[tid]; sh.candi[place] = (int)at;
            }
            n_cand = n <= SAMPLE_CAND ? n : -1;
        } else {
            // fewer threads with elements than k: every element is a candidate, if they fit
            const int s0 = rank * SAMPLE_WARPS * per, slice = min(vocab, s0 + SAMPLE_WARPS * per) - min(vocab, s0);
            if (slice <= SAMPLE_CAND)
                each([&](int i, float v) { if (i < i1) { sh.cand[i - s0] = ordered_key(v); sh.candi[i - s0] = i; } });
            if (tid == 0) sh.cmin = 0u;
            n_cand = slice <= SAMPLE_CAND ? slice : -1;
        }
    }
    // ---- the block's sum of weights: over all its words under its own maximum, or (select) whether it has a NaN ----
    float lo = 0.f, hi = 0.f, bsum = 0.f;           // this warp's bracket inside the block, and the block's sum
    auto warp_sums = [&](float ws) {
        ws = warp_sum(ws);
        __syncthreads();
        if (lane == 0) sh.wf[warp] = ws;
        __syncthreads();
        bsum = 0.f;
        for (int w = 0; w < SAMPLE_WARPS; ++w) {    // (the same order everywhere: brackets meet without gaps)
            if (w == warp) lo = bsum;
            bsum += sh.wf[w];
            if (w == warp) hi = bsum;
        }
    };
    if (whole_row) {
        if constexpr (NQ > 0) each([&](int, float v) { wsum += weight(v, bmax); });
        else if (mine > -INFINITY) wsum *= __expf((mine - bmax) * inv_t);
        warp_sums(wsum);
    } else if (select) {
        bsum = __syncthreads_or(nan) ? NAN : 0.f;
    }
    cluster.barrier_wait();
    if (tid < C) {
        SampleShared* peer = cluster.map_shared_rank(&sh, tid);
        peer->bmax[rank] = bmax; peer->ncand[rank] = n_cand; peer->bsum[rank] = bsum;
    }
    cluster.sync();
    const float vmax = row_max(lane < C ? sh.bmax[lane] : -INFINITY);
    // the row's lowest index that holds the maximum (every block of the cluster takes part)
    auto write_argmax = [&]() {
        __syncthreads();
        if (tid == 0) sh.need = 0x7fffffffu;
        __syncthreads();
        if (mine == vmax) {
            int first = 0x7fffffff;
            each([&](int i, float v) { if (v == vmax && i < i1) first = min(first, i); });
            atomicMin(&sh.need, (unsigned)first);
        }
        __syncthreads();
        if (tid == 0) cluster.map_shared_rank(&sh, 0)->bidx[rank] = (int)sh.need;
        cluster.sync();
        if (rank == 0 && tid == 0) {
            int best = sh.bidx[0];
            for (int r = 1; r < C; ++r) best = min(best, sh.bidx[r]);
            out[row_id] = best < vocab ? best : 0;  // (a row of NaNs has no maximum)
        }
    };
    if (greedy) { write_argmax(); return; }

    const float u = uniform[row_id];
    float least = -FLT_MAX, base = 0.f, next = 0.f, total = 0.f, scale = 1.f;      // the block's bracket and the total; what its own sums are scaled by
    if (select) {
        // ---- 2b. threshold: the k-th largest key ----
        auto for_blocks = [&](auto&& f) {           // (without a loop where it would be the longest: one row, k = 50, 12.4 us with it, 12.2 without)
            if (C == SAMPLE_MAX_CLUSTER) {
#pragma unroll
                for (int r = 0; r < SAMPLE_MAX_CLUSTER; ++r) f(r);
            } else {
                for (int r = 0; r < C; ++r) f(r);
            }
        };
        // a lane per block: how many candidates it has, where its list begins in the union and where that ends
        const int listed = lane < C ? sh.ncand[lane] : 0;
        int list_end = listed;
#pragma unroll
        for (int o = 1; o < SAMPLE_MAX_CLUSTER; o <<= 1) {
            const int p = __shfl_up_sync(0xffffffffu, list_end, o);
            if (lane >= o) list_end += p;
        }
        const int count = __shfl_sync(0xffffffffu, list_end, SAMPLE_MAX_CLUSTER - 1), mine0 = __shfl_sync(0xffffffffu, list_end - listed, rank);
        const bool fits = __all_sync(0xffffffffu, listed >= 0) && count <= SAMPLE_KEYS * SAMPLE_THREADS;
        const float odd = __any_sync(0xffffffffu, lane < C && sh.bsum[lane] != 0.f) ? NAN : 0.f;      // (a block's is 0 or NaN)
        if (fits) {
            // this thread's share of the union: the blocks' lists one after the other (0 is below every key of a number)
            unsigned key[SAMPLE_KEYS];
#pragma unroll
            for (int q = 0; q < SAMPLE_KEYS; ++q) {
                const int e = q * SAMPLE_THREADS + tid;
                key[q] = 0u;
                if (q * SAMPLE_THREADS < count) {
                    int r = 0;
                    for_blocks([&](int k) { r += e >= __shfl_sync(0xffffffffu, list_end, k); });
                    const int at = e - __shfl_sync(0xffffffffu, list_end - listed, r & (SAMPLE_MAX_CLUSTER - 1));
                    if (e < count) key[q] = cluster.map_shared_rank(&sh, r)->cand[at];
                }
            }
            // Every block has read every list when it may leave; this one's own lists stay until then.
            cluster.barrier_arrive();
            const bool one = count <= SAMPLE_THREADS;
            // The largest t with at least k keys >= t, or any t with exactly k of them.  This block's candidates are at least k, so the k-th
            // largest key lies between the smallest of them and the maximum: only the bits below their common ones are searched.
            const unsigned diff = ordered_key(vmax) ^ sh.cmin;
            int bit = diff ? 31 - __clz(diff) : -1;
            unsigned t = bit < 0 ? sh.cmin : bit == 31 ? 0u : sh.cmin & ~((2u << bit) - 1u);
            for (; bit >= 0; --bit) {
                const unsigned trial = t | (1u << bit);
                unsigned n;
                if (one) n = (unsigned)__syncthreads_count(key[0] >= trial);
                else {
                    unsigned c = 0;
#pragma unroll
                    for (int q = 0; q < SAMPLE_KEYS; ++q) c += key[q] >= trial ? 1u : 0u;
                    c = __reduce_add_sync(0xffffffffu, c);
                    if (lane == 0) sh.wcount[bit & 1][warp] = c;
                    __syncthreads();                // (two buffers: the next round's writers cannot overtake this one's readers)
                    n = __reduce_add_sync(0xffffffffu, sh.wcount[bit & 1][lane]);
                }
                if (n >= (unsigned)top_k) t = trial;
                if (n == (unsigned)top_k) break;
            }
            // ---- 3. and 4. from the candidates alone: all kept words are among them, and every block adds the same weights in the same order, so
            // the blocks' brackets meet without another exchange.  A warp sums a list, and the lists' sums follow one another: a list without a
            // kept word adds exactly nothing, its block's bracket is empty (prefix sums of one scan over all lists would differ in the
            // last place where nothing but zeros lies between them) ----
            auto key_weight = [&](unsigned k) { return k >= t ? weight(key_value(k), vmax) : 0.f; };
#pragma unroll
            for (int q = 0; q < SAMPLE_KEYS; ++q) {
                const int e = q * SAMPLE_THREADS + tid;
                if (e < count) sh.weight[e] = key_weight(key[q]);
            }
            if (tid == 0) { sh.need = 0xffffffffu; sh.cand_n = 0u; }
            __syncthreads();
            if (warp < C) {
                const int end = __shfl_sync(0xffffffffu, list_end, warp);
                float ws = 0.f;
                for (int j = __shfl_sync(0xffffffffu, list_end - listed, warp) + lane; j < end; j += 32) ws += sh.weight[j];
                ws = warp_sum(ws);
                if (lane == 0) sh.wf[warp] = ws;
            }
            __syncthreads();
            const float list_sum = lane < C ? sh.wf[lane] : 0.f;
            for_blocks([&](int r) {
                if (r == rank) base = total;
                total += __shfl_sync(0xffffffffu, list_sum, r);
                if (r == rank) next = total;
            });
            total += odd;
            // Weights that are not numbers (infinite logits, or a NaN in the row), or a u outside [0, 1): no draw, the arg-max.
            if (!(total > 0.f && total < INFINITY && u >= 0.f && u < 1.f)) { cluster.barrier_wait(); write_argmax(); return; }
            float target = u * total;
            if (!(target < total)) target = __uint_as_float(__float_as_uint(total) - 1u);   // u * total rounded up to the total: the last word with a weight
            if (base <= target && target < next) {
                // the first of this block's kept words, in the order of their indices, whose inclusive prefix sum exceeds the target.  (next > base:
                // one of them has a weight)
                const float own = tid < n_cand ? sh.weight[mine0 + tid] : 0.f;
                float p = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float v = __shfl_up_sync(0xffffffffu, p, o);
                    if (lane >= o) p += v;
                }
                if (lane == 31) sh.wg[warp] = p;
                __syncthreads();
                if (warp > 0 && 32 * warp < n_cand) p += warp_sum(lane < warp ? sh.wg[lane] : 0.f);
                if (own > 0.f) {
                    const unsigned at = (unsigned)sh.candi[tid];
                    if (base + p > target) atomicMin(&sh.need, at);
                    atomicMax(&sh.cand_n, at);
                }
                __syncthreads();
                // rounding may leave the target a hair beyond the block's own sum: then its last word with a weight
                if (tid == 0) out[row_id] = sh.need != 0xffffffffu ? (long long)sh.need : (long long)sh.cand_n;
            }
            cluster.barrier_wait();
            return;
        } else {
            unsigned prefix = 0u, need = (unsigned)top_k;
            for (int pass = 0; pass < 3; ++pass) {
                const int shift = pass == 0 ? 21 : (pass == 1 ? 10 : 0), width = pass == 2 ? 10 : 11;
                const unsigned mask = pass == 0 ? 0u : 0xffffffffu << (shift + width);
                for (int b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) sh.hist[b] = 0u;
                __syncthreads();
                each([&](int i, float v) {
                    const unsigned k = ordered_key(v);
                    if (i < i1 && (k & mask) == prefix) atomicAdd(&sh.hist[(k >> shift) & ((1u << width) - 1u)], 1u);
                });
                cluster.sync();
                unsigned c0 = 0u, c1 = 0u;          // bins SAMPLE_BINS - 1 - 2 tid and the one below it, over the cluster
                for (int r = 0; r < C; ++r) {
                    const unsigned* h = cluster.map_shared_rank(&sh, r)->hist;
                    c0 += h[SAMPLE_BINS - 1 - 2 * tid]; c1 += h[SAMPLE_BINS - 2 - 2 * tid];
                }
                find_bin(sh, c0, c1, need, true);
                prefix |= sh.sel << shift;
                need = sh.need;
                cluster.sync();                     // every block has read this pass's histograms
            }
            least = fmaxf(key_value(prefix), -FLT_MAX);
        }
        // ---- 3. weights of the kept logits: sums per warp, per block, over the row, in index order ----
        float ws = 0.f;
        each([&](int, float v) { if (!(v < least)) ws += __expf((v - vmax) * inv_t); });
        warp_sums(ws);
        if (tid < C) cluster.map_shared_rank(&sh, tid)->bsum[rank] = bsum;
        cluster.sync();
        for (int r = 0; r < C; ++r) {
            if (r == rank) base = total;
            total += sh.bsum[r];
            if (r == rank) next = total;
        }
    } else {
        // ---- 3. every block's sum was taken under its own maximum ----
        const float own = lane < C ? sh.bsum[lane] : 0.f, f = own == 0.f ? 0.f : __expf((sh.bmax[lane < C ? lane : 0] - vmax) * inv_t);
        const float part = __fmul_rn(f, own);       // a lane per block
        scale = __shfl_sync(0xffffffffu, f, rank);
        for (int r = 0; r < C; ++r) {
            if (r == rank) base = total;
            total = __fadd_rn(total, __shfl_sync(0xffffffffu, part, r));
            if (r == rank) next = total;
        }
    }
    // ---- 4. the first index whose inclusive prefix exceeds u * total ----
    // Weights that are not numbers (infinite logits, or a NaN among them), or a u outside [0, 1): no draw, the arg-max.
    if (!(total > 0.f && total < INFINITY && u >= 0.f && u < 1.f)) { write_argmax(); return; }
    float target = u * total;
    if (!(target < total)) target = __uint_as_float(__float_as_uint(total) - 1u);   // u * total rounded up to the total: the last word with a weight
    if (!(base <= target && target < next)) return;
    // Inside the block: `from` of the first warp is base, `to` of the last one is next (the same roundings), and both are the same sums for
    // the neighbouring warps, so exactly one warp's run takes it.  The whole block walks that run, WALK words a thread.
    const float from = __fadd_rn(base, __fmul_rn(scale, lo)), to = __fadd_rn(base, __fmul_rn(scale, hi));
    if (lane == 0 && from <= target && target < to) { sh.sel = (unsigned)warp; sh.wg[0] = from; }
    if (tid == 0) { sh.need = 0xffffffffu; sh.cand_n = 0u; }
    __syncthreads();
    // The run was chosen by weights under the block's own maximum, its words are weighed under the row's: where those underflow the run may have no
    // word with a weight.  Then it is the next one behind the run, or the block's first: its maximum has a weight, or its sum would be nothing.
    auto run_start = [&](int w) { return (int)min((long long)vocab, (long long)(rank * SAMPLE_WARPS + w) * per); };
    const int s0 = run_start(0), s1 = run_start(SAMPLE_WARPS), r0 = run_start((int)sh.sel), r1 = run_start((int)sh.sel + 1);
    float run = sh.wg[0];
    int first = r0, end = r1, span = 0;             // 0: the run, 1: what follows it, 2: what is before it
    for (;;) {
        const int i = first + WALK * tid;
        float own[WALK], incl[WALK];
#pragma unroll
        for (int q = 0; q < WALK; ++q) own[q] = i + q < end ? row[i + q] : -INFINITY;
        // (the scan adds the same weights in another order for every lane, so a word without weight may see a larger prefix than the
        // word before it: only one with a weight is a candidate)
#pragma unroll
        for (int q = 0; q < WALK; ++q) {
            own[q] = own[q] >= least ? __expf((own[q] - vmax) * inv_t) : 0.f;
            incl[q] = q ? incl[q - 1] + own[q] : own[q];
        }
        float sum = incl[WALK - 1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float p = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += p;
        }
        if (lane == 31) sh.wf[warp] = sum;
        float lower = __shfl_up_sync(0xffffffffu, sum, 1);     // of the lanes before this one
        if (lane == 0) lower = 0.f;
        __syncthreads();
        float before = run;
        for (int w = 0; w < SAMPLE_WARPS; ++w) {
            if (w == warp) before = run;
            run += sh.wf[w];
        }
        unsigned hit = 0xffffffffu, last = 0u;
#pragma unroll
        for (int q = WALK - 1; q >= 0; --q) {
            if (own[q] > 0.f && (span > 0 || before + (lower + incl[q]) > target)) hit = (unsigned)(i + q);
            if (own[q] > 0.f && last == 0u) last = (unsigned)(i + q + 1);
        }
        hit = __reduce_min_sync(0xffffffffu, hit); last = __reduce_max_sync(0xffffffffu, last);
        if (lane == 0 && hit != 0xffffffffu) atomicMin(&sh.need, hit);
        if (lane == 0 && last) atomicMax(&sh.cand_n, last);    // (0: none so far)
        __syncthreads();
        if (sh.need != 0xffffffffu) break;
        first += WALK * SAMPLE_THREADS;
        if (first >= end) {
            if (sh.cand_n > 0u || span == 2) break;
            ++span;
            first = span == 1 ? r1 : s0; end = span == 1 ? s1 : r0;
        }
    }
    // rounding may leave the target a hair beyond the run's own sum: then its last element with a weight
    if (tid == 0) out[row_id] = sh.need != 0xffffffffu ? (long long)sh.need : (long long)sh.cand_n - 1;
}

template <int NQ, bool TWO, bool SHARE>
static cudaError_t launch_sample(int cluster, const float* logits, int batch, int vocab, float temperature, int top_k, const float* uniform,
                                 long long* out, cudaStream_t st) {
    if (cluster > 8) {   // sizes above 8 are opt-in, per device and function (setting it again changes nothing)
        const cudaError_t e = cudaFuncSetAttribute(sample_kernel<NQ, TWO, SHARE>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)batch * (unsigned)cluster); cfg.blockDim = dim3(SAMPLE_THREADS); cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, sample_kernel<NQ, TWO, SHARE>, logits, vocab, temperature, top_k, uniform, out);
}

}  // namespace q3

extern "C" int q3_sample(const float* logits, int32_t batch, int32_t vocab, float temperature, int32_t top_k,
                         const float* uniform, int64_t* out_tokens, void* stream) {
    if (!logits || !out_tokens) return q3::engine_fail(nullptr, Q3_ERR_INVALID, "q3_sample: logits and out_tokens are required");
    if (batch < 1 || vocab < 1 || top_k < 0) return q3::engine_fail(nullptr, Q3_ERR_INVALID, "q3_sample: batch=%d vocab=%d top_k=%d out of range", batch, vocab, top_k);
    if (temperature > 0.f && top_k != 1 && !uniform) return q3::engine_fail(nullptr, Q3_ERR_INVALID, "q3_sample: sampling needs one uniform number per row");
    // Blocks per row: as many as keep all rows' clusters resident at once, and at least 1024 words a block.  Measured with the
    // full vocabulary, us with clusters of 1 / 2 / 4 / 8 / 16 blocks, before lists were put in order (those in use, k = 50, with it: 1 and 8 rows 12.3, 16
    // rows 16.4, 64 rows 24.6): 1 row, k = 50: 24.4 / 18.5 / 15.8 / 12.3 / 12.1; 8 rows, k = 50:
    // 24.7 / 19.1 / 16.4 / 12.3 / 20.2; 16 rows, k = 50: 25.3 / 19.5 / 16.4 / 20.5 / 29.1; 33 rows, all words: 25.1 / 18.5 / 14.4 / 20.5 / 32.8;
    // 40 rows, all words: 26.7 / 19.2 / 20.7 / 22.6; 64 rows, all words: 27.5 / 20.5 / 21.6 / 35.0; 64 rows, k = 50: 30.7 / 24.6 / 26.6 / 48.1.
    // A thread keeps its elements in registers where it has at most three groups of four, or five.
    // One block an SM, with registers for eight loads, where that is room for every cluster: pairs of blocks for up to 64 rows (64 rows 18.6 us, with two
    // blocks an SM 20.4; clusters of four do not fit 148 SMs one by one: 36 rows, k = 50, 31.0 and 22.8).
    // The candidates' threads are read by a lane a group, four threads at a time, while a warp (k / 32 such threads) has few of them for its groups: k =
    // 50, 15 / 64 rows 15.1 / 18.7 us, each thread by itself 16.6 / 22.8; k = 200, 64 rows 23.0 / 26.8, but 36 rows 28.9 / 26.9 and 15 rows 21.0 / 18.9.
    int cluster = batch <= 4 ? 16 : batch <= 14 ? 8 : batch <= 36 ? 4 : batch <= 148 ? 2 : 1;
    while (cluster > 1 && vocab < cluster * q3::SAMPLE_THREADS) cluster /= 2;
    const int groups = q3::sample_run(vocab, cluster) / 128;
    cudaStream_t st = (cudaStream_t)stream;
    long long* out = reinterpret_cast<long long*>(out_tokens);
    const bool share = top_k <= 12 * groups || top_k >= vocab, deep = cluster == 2 && batch <= 64;
    auto* const launch = groups <= 3 ? q3::launch_sample<3, false, false> : groups <= 5 ? q3::launch_sample<5, false, false>
                         : deep ? (share ? q3::launch_sample<0, false, true> : q3::launch_sample<0, false, false>)
                                : (share ? q3::launch_sample<0, true, true> : q3::launch_sample<0, true, false>);
    const cudaError_t err = launch(cluster, logits, batch, vocab, temperature, top_k, uniform, out, st);
    if (err != cudaSuccess) return q3::engine_fail(nullptr, Q3_ERR_CUDA, "q3_sample: %s", cudaGetErrorString(err));
    return Q3_OK;
}
