// C ABI of the engine (declared in include/q3mk.h): engine life cycle, argument checks, path
// selection and the per-step launch sequence of the layered path.
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include <cuda.h>

#include "q3_engine.h"
#include "q3_gemm_cl.h"
#include "q3_gemm_tc.h"
#include "q3_layer_tc.h"
#include "q3_prompt.h"

using namespace q3;

static char g_create_error[512] = "";

int q3::engine_fail(q3_engine* e, int code, const char* fmt, ...) {
    char* dst = e ? e->err : g_create_error;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(dst, 512, fmt, ap);
    va_end(ap);
    return code;
}
#define fail q3::engine_fail

#define CU(e, call)                                                                                  \
    do {                                                                                             \
        cudaError_t err__ = (call);                                                                  \
        if (err__ != cudaSuccess)                                                                    \
            return fail(e, Q3_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(err__), __FILE__, __LINE__); \
    } while (0)

// ------------------------------------------------------------------------------------------------
// CUDA graphs for the layered step: a step is hundreds of small launches whose arguments all live in
// device memory, so a call with the same argument block can replay a captured graph instead of
// re-issuing them.  A key's first uses are plain launches (which also perform one-time function attribute
// set-up), then it is captured, and replayed afterwards.  Weights, RoPE table or trace changes
// drop the cache.
// ------------------------------------------------------------------------------------------------
// The key holds the addresses of one bind, so every bind captures anew.  A capture costs the host 450 to 850 us, beside 360 for the
// plain launches of a step; after three steps that are launched without waiting the GPU is far enough behind to hide it (8 x 1024, a fresh
// bind of 8 steps, capture on the 2nd / 4th: 6070 / 5910 us; of 2 steps 1680 / 1540).  Three sequences, whose steps before the capture are launches of the
// persistent kernel, and two of a caller who names the chain wait until the ninth: a replay saves them only 10 to 25 us a step, and a caller who waits for every
// step pays for the whole capture.  us of a fresh bind of 8 / 16 / 40 steps, capture on the 4th / the 9th / never: three at 16 positions, waiting for every
// step, 5370 / 10800 / 24610, 5080 / 11000 / 25700, 4990 / 9890 / 24630, without waiting 4730 / 9290 / 23060, 4880 / 9480 / 23420, 4900 / 9670 / 24080; three ragged
// up to 900 5690 / 10830 / 25890, 5230 / 10830 / 25940, 5210 / 10380 / 25960 and 5050 / 9990 / 24810, 5140 / 10060 / 24880, 5100 / 10150 / 25420; the chain at two
// of 16 5390 / 10040 / 24960, 5110 / 10610 / 25380, 5130 / 10290 / 25500 and 4760 / 9320 / 23160, 5010 / 9560 / 23640, 5000 / 9960 / 24630.  So the ninth costs 1 to 5
// per cent where nobody waits, and is worth 5 to 9 per cent of a short turn where somebody does.
static int plain_uses(int batch, bool persist) { return batch == 2 || persist ? 8 : 3; }
struct GraphEntry {
    q3_decode_args key;
    int n_splits;
    int chunk_pad;         // the attention kernel's padded chunk length is baked into the captured arguments
    int seen;
    int64_t launches;      // kernels inside the graph
    cudaGraphExec_t exec;
};
static std::vector<GraphEntry>* graph_cache(q3_engine* e) {
    if (!e->graphs) e->graphs = new std::vector<GraphEntry>();
    return static_cast<std::vector<GraphEntry>*>(e->graphs);
}
static void drop_graphs(q3_engine* e) {
    if (!e->graphs) return;
    auto* v = static_cast<std::vector<GraphEntry>*>(e->graphs);
    for (auto& g : *v)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    v->clear();
}

extern "C" const char* q3_version(void) { return "q3mk-b200 0.1 sm_100a"; }

extern "C" const char* q3_last_error(const q3_engine* e) { return e ? e->err : g_create_error; }

extern "C" int q3_create(int device, const q3_config* cfg, q3_engine** out) {
    if (!cfg || !out) return fail(nullptr, Q3_ERR_INVALID, "q3_create: null argument");
    *out = nullptr;
    if (cfg->n_layers < 1 || cfg->vocab < 1 || cfg->max_batch < 1 || cfg->max_tokens < 0 || cfg->grid_limit < 0 || cfg->wait_limit_us < 0)
        return fail(nullptr, Q3_ERR_INVALID, "q3_create: n_layers=%d vocab=%d max_batch=%d max_tokens=%d grid_limit=%d out of range",
                    cfg->n_layers, cfg->vocab, cfg->max_batch, cfg->max_tokens, cfg->grid_limit);
    CU(nullptr, cudaSetDevice(device));
    cudaDeviceProp prop;
    CU(nullptr, cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10)
        return fail(nullptr, Q3_ERR_UNSUPPORTED, "q3_create: device %d is sm_%d%d; this library holds sm_100a code only", device, prop.major, prop.minor);

    q3_engine* e = new (std::nothrow) q3_engine();
    if (!e) return fail(nullptr, Q3_ERR_INVALID, "q3_create: out of host memory");
    memset(e, 0, sizeof(*e));
    e->device = device;
    e->cfg = *cfg;
    e->sm_count = prop.multiProcessorCount;
    e->max_splits = Q3_MAX_SPLITS;
    e->lm_grid = e->sm_count * 8;
    e->cap = cfg->max_batch > cfg->max_tokens ? cfg->max_batch : cfg->max_tokens;
    const size_t B = (size_t)e->cap;
    // attention partials: up to 64 splits for small batches, at least 2 per token for large ones
    e->part_slots = (int)((B < 16 ? B : 16) * Q3_MAX_SPLITS > 2 * B ? (B < 16 ? B : 16) * Q3_MAX_SPLITS : 2 * B);
    const bool tc = e->cap >= Q3_TC_MIN_BATCH;
    const size_t cap_pad = (B + 127) / 128 * 128;
    e->chain_rows = gemm_cluster_rows(cfg->max_batch < CL_MAX_TOK ? cfg->max_batch : CL_MAX_TOK);
    // one allocation for all of it: every cudaMalloc and cudaFree of an engine's life costs its caller about a millisecond
    struct Part { void** p; size_t bytes; };
    const Part parts[] = {
        {(void**)&e->x, B * HIDDEN * 4}, {(void**)&e->qkv, B * QKV_DIM * 4}, {(void**)&e->attn, B * Q_DIM * 4}, {(void**)&e->hid, B * INTER * 4},
        {(void**)&e->part, (size_t)e->part_slots * Q_HEADS * ATTN_PART_STRIDE * 4},
        {(void**)&e->pval, (size_t)cfg->max_batch * e->lm_grid * 4}, {(void**)&e->pidx, (size_t)cfg->max_batch * e->lm_grid * 4},
        {(void**)&e->status, Q3_STATUS_WORDS * 4}, {(void**)&e->sync, Q3_SYNC_WORDS * 4}, {&e->pf_desc, 64 + B * 32},
        {&e->planes, 3 * cap_pad * INTER * 2}, {&e->xplanes, (size_t)3 * e->chain_rows * HIDDEN * 2}, {(void**)&e->ssq, (size_t)CL_SSQ_PARTS * e->chain_rows * 4},
        {(void**)&e->logits_tc, cfg->max_batch >= Q3_TC_MIN_BATCH ? (size_t)cfg->max_batch * cfg->vocab * 4 : 0},
        {(void**)&e->gate, tc ? B * INTER * 4 : 0}, {(void**)&e->up, tc ? B * INTER * 4 : 0}, {&e->lk_state, tc ? (size_t)LK_STATE_BYTES : 0}};
    auto padded = [](size_t n) { return (n + 1023) / 1024 * 1024; };
    size_t total = 0;
    for (const Part& p : parts) total += padded(p.bytes);
    cudaError_t err = cudaMalloc(&e->scratch, total);
    if (err == cudaSuccess) err = cudaMemset(e->scratch, 0, total);
    if (err != cudaSuccess) {
        q3_destroy(e);
        return fail(nullptr, Q3_ERR_CUDA, "q3_create: scratch of %zu bytes: %s", total, cudaGetErrorString(err));
    }
    char* at = static_cast<char*>(e->scratch);
    for (const Part& p : parts) {
        *p.p = p.bytes ? at : nullptr;
        at += padded(p.bytes);
    }
    int rc;
    {
        cudaStream_t cs = nullptr;
        if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) {
            fail(nullptr, Q3_ERR_CUDA, "q3_create: cudaStreamCreateWithFlags failed");
            q3_destroy(e);
            return Q3_ERR_CUDA;
        }
        e->capture_stream = cs;
    }
    rc = persist_setup(e);
    if (rc != Q3_OK) {
        strncpy(g_create_error, e->err, sizeof(g_create_error) - 1);
        q3_destroy(e);
        return rc;
    }
    *out = e;
    return Q3_OK;
}

extern "C" void q3_destroy(q3_engine* e) {
    if (!e) return;
    cudaSetDevice(e->device);
    drop_graphs(e);
    delete static_cast<std::vector<GraphEntry>*>(e->graphs);
    if (e->capture_stream) cudaStreamDestroy(static_cast<cudaStream_t>(e->capture_stream));
    persist_teardown(e);
    if (e->scratch) cudaFree(e->scratch);
    delete e;
}

extern "C" int q3_set_weights(q3_engine* e, const q3_weights* w) {
    if (!e || !w) return fail(e, Q3_ERR_INVALID, "q3_set_weights: null argument");
    const void* const* p = reinterpret_cast<const void* const*>(w);
    static const char* names[13] = {"ln1", "wq", "wk", "wv", "qn", "kn", "wo", "ln2", "wg", "wu", "wd", "fnorm", "embed"};
    for (int i = 0; i < 13; ++i) {
        if (!p[i]) return fail(e, Q3_ERR_INVALID, "q3_set_weights: %s is null", names[i]);
        if (reinterpret_cast<uintptr_t>(p[i]) & 15) return fail(e, Q3_ERR_INVALID, "q3_set_weights: %s is not 16-byte aligned", names[i]);
    }
    drop_graphs(e);
    e->w = *w;
    e->have_weights = 1;
    CU(e, cudaSetDevice(e->device));
    return persist_weights_changed(e);
}

extern "C" int q3_invalidate_weights(q3_engine* e) {
    if (!e) return Q3_ERR_INVALID;
    persist_invalidate_weights(e);
    return Q3_OK;
}

extern "C" int q3_tp_export(q3_engine* e, void* handle) {
    if (!e || !handle) return fail(e, Q3_ERR_INVALID, "q3_tp_export: null argument");
    CU(e, cudaSetDevice(e->device));
    return persist_tp_export(e, handle);
}

extern "C" int q3_tp_attach(q3_engine* e, int32_t rank, int32_t size, const void* handles) {
    if (!e) return fail(e, Q3_ERR_INVALID, "q3_tp_attach: null argument");
    CU(e, cudaSetDevice(e->device));
    drop_graphs(e);
    return persist_tp_attach(e, rank, size, handles);
}

extern "C" int q3_set_rope(q3_engine* e, const float* table, int32_t n_positions) {
    if (!e || !table || n_positions < 1) return fail(e, Q3_ERR_INVALID, "q3_set_rope: bad argument");
    drop_graphs(e);
    e->rope = table;
    e->rope_n = n_positions;
    return Q3_OK;
}

extern "C" int q3_set_trace(q3_engine* e, uint64_t* buf, int64_t n_words) {
    if (!e || n_words < 0) return fail(e, Q3_ERR_INVALID, "q3_set_trace: bad argument");
    e->trace = reinterpret_cast<unsigned long long*>(buf);
    e->trace_words = buf ? n_words : 0;
    return Q3_OK;
}

extern "C" int64_t q3_launch_count(const q3_engine* e) { return e ? e->launches : 0; }

extern "C" int q3_grid_info(const q3_engine* e, int32_t* ctas, int32_t* threads, int32_t* smem_bytes) {
    if (!e) return Q3_ERR_INVALID;
    if (ctas) *ctas = e->p_grid;
    if (threads) *threads = e->p_threads;
    if (smem_bytes) *smem_bytes = e->p_smem;
    return Q3_OK;
}

extern "C" int q3_scratch(const q3_engine* e, const char* name, void** ptr, int64_t* bytes) {
    if (!e || !name || !ptr || !bytes) return Q3_ERR_INVALID;
    const int64_t B = e->cap;
    if (!strcmp(name, "x")) { *ptr = e->x; *bytes = B * HIDDEN * 4; }
    else if (!strcmp(name, "qkv")) { *ptr = e->qkv; *bytes = B * QKV_DIM * 4; }
    else if (!strcmp(name, "attn")) { *ptr = e->attn; *bytes = B * Q_DIM * 4; }
    else if (!strcmp(name, "hid")) { *ptr = e->hid; *bytes = B * INTER * 4; }
    else if (!strcmp(name, "status")) { *ptr = e->status; *bytes = Q3_STATUS_WORDS * 4; }
    else if (!strcmp(name, "persist_acc")) { *ptr = persist_accumulators(e, bytes); if (!*ptr) return Q3_ERR_UNSUPPORTED; }
    else return Q3_ERR_INVALID;
    return Q3_OK;
}

extern "C" int q3_status(q3_engine* e, void* stream, uint32_t* words, int32_t n) {
    if (!e) return Q3_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t h[Q3_STATUS_WORDS];
    CU(e, cudaStreamSynchronize(st));
    CU(e, cudaMemcpy(h, e->status, sizeof(h), cudaMemcpyDeviceToHost));
    for (int i = 0; words && i < n && i < Q3_STATUS_WORDS; ++i) words[i] = h[i];
    if (h[0] == 0) return Q3_OK;
    // leave the engine reusable: clear the status and the barrier words
    CU(e, cudaMemset(e->status, 0, Q3_STATUS_WORDS * 4));
    CU(e, cudaMemset(e->sync, 0, Q3_SYNC_WORDS * 4));
    if (e->lk_state) CU(e, cudaMemset(e->lk_state, 0, LK_STATE_BYTES));
    if (persist_recover(e) != Q3_OK) return Q3_ERR_CUDA;
    return fail(e, Q3_ERR_DEVICE_WAIT, "device status: code %u at site %u, CTA %u, value %u", h[0], h[1], h[2], h[3]);
}

// ------------------------------------------------------------------------------------------------
// layered decode step
// ------------------------------------------------------------------------------------------------
// positions a split's block may take, rounded up to 32: with the split count it fixes the attention launch
static int chunk_pad_for(int max_len, int ns) { return (((max_len + 1 + ns - 1) / ns) + 31) / 32 * 32; }

// Decode steps of up to CL_MAX_TOK sequences run as five launches per layer (q3_gemm_cl.h); larger ones, and a step without an
// engine (q3_decode_noalloc, which has no planes), keep one launch per phase.
static bool chain_serves(const q3_engine* e, int batch) { return e->xplanes != nullptr && batch <= CL_MAX_TOK; }

static int splits_for(const q3_engine* e, int batch, int max_len, bool chain) {
    const double merge_us = chain ? 1.0 : 5.0;   // what more than one split costs beyond its blocks
    const int n = max_len + 1;
    int by_len = (n + 31) / 32;                                   // at least 32 positions per split
    // The split count with the shortest estimated launch.  A launch takes `waves` rounds of blocks; a block costs a fixed
    // 4 us (prologue with the head preparation, combine) plus its positions at the block's share of an SM's part of the copy
    // bandwidth; more than one split adds the merge launch (5 us), one split writes the output planes itself.
    //   Batches whose (sequence, kv head) pairs fill the GPU: four-warp blocks, two per SM, 23 ns per position.  Fitted to,
    //   per step: batch 64 x 1024, 1 / 2 / 3 / 4 splits: 2524 / 2623 / 2691 / 2716 us; batch 32 x 2048, 1 / 2: 2057 / 2149;
    //   batch 24 x 1024, 1 / 3: 1336 / 1463; batch 48 x 1024, 1 / 2: 2235 / 2214; batch 20 x 4096, 2 / 3: 2814 / 2415.
    //   Smaller batches: eight-warp blocks, one per SM, 6 ns per position.  Batch 8 x 1024, 1 / 2 splits: 1000 / 1035 us;
    //   batch 4 x 512: 882 / 920; batch 16 x 2048: 1446 / 1597.
    //   The chain: four-warp blocks for every batch (two of them, or one and a block of a neighbouring product, share an SM), a cluster
    //   costs 1 us, and blocks beyond the first round start as others end.  Batch 8 x 1024, 1 / 2 / 3 / 4 / 8 splits: 889 / 785 / 744 /
    //   734 / 913 us; 27 ragged up to 2048: 1429 / 1381 / 1496 / 1596 / 1958; 64 x 1024: 2344 / 2631 / 2682 / 2841 / 3916; three at 900
    //   (eight steps): 6329 / 5786 / 5473 / 5337 / 5139.
    const bool big = chain || KV_HEADS * batch >= e->sm_count;
    const int slots = (big ? 2 : 1) * e->sm_count, pairs = KV_HEADS * batch;
    const double per_pos = big ? 0.023 : 0.006;
    double best = 1e30;
    int s = 1;
    for (int c = 1; c <= (chain ? ATTN_CLUSTER_MAX : 16) && c <= by_len; ++c) {
        const int waves = (pairs * c + slots - 1) / slots, per = (n + c - 1) / c;
        const double rounds = chain ? fmax(1.0, (double)pairs * c / slots) : waves;
        const double t = 4.0 * waves + per_pos * per * rounds + (c > 1 ? merge_us : 0.0);
        if (t < best - 1e-9) { best = t; s = c; }
    }
    if (s < 1) s = 1;
    const int by_chunk = (n + ATTN_CHUNK_MAX - 1) / ATTN_CHUNK_MAX;   // a split takes at most ATTN_CHUNK_MAX positions (the launchers check it)
    if (s < by_chunk) s = by_chunk;
    if (s > e->max_splits) s = e->max_splits;
    if (e->part_slots > 0 && s * batch > e->part_slots) s = e->part_slots / batch;
    if (s < 1) s = 1;
    return s;
}

int q3::decode_layered(q3_engine* e, const q3_decode_args* a, cudaStream_t st, bool prompt, bool layer_kernel) {
    const bool last_token_only = prompt;
    const int B = a->batch, L = e->cfg.n_layers, V = e->cfg.vocab;
    const q3_weights& w = e->w;
    const int append = (a->flags & Q3_F_APPEND_KV) ? 1 : 0;
    const bool chain = !prompt && !layer_kernel && chain_serves(e, B);
    const int ns = splits_for(e, B, a->max_len, chain);
    // From Q3_TC_MIN_BATCH tokens on, the projections are tensor-core GEMMs over three bf16 planes of the
    // activations (exact to fp32); below that, CUDA-core matrix-vector kernels.
    constexpr int tc_planes = 3;
    const bool tc = B >= Q3_TC_MIN_BATCH && e->planes != nullptr;
    const int tile = B <= 32 ? 32 : (B <= 64 ? 64 : 128);
    const int prow = (B + tile - 1) / tile * tile;
    bf16_raw* planes = reinterpret_cast<bf16_raw*>(e->planes);
    auto bf = [](const void* p) { return reinterpret_cast<const bf16_raw*>(p); };
#define LAUNCH(call)                                                                                   \
    do {                                                                                               \
        cudaError_t err__ = (call);                                                                    \
        ++e->launches;                                                                                 \
        if (err__ != cudaSuccess) return fail(e, Q3_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(err__)); \
    } while (0)
    // out[:, col0 : col0 + rows] (+)= planes @ wmat^T
    auto gemm = [&](const bf16_raw* wmat, int rows, int K, float* out, int ldo, const float* resid, int ldr) -> cudaError_t {
        GemmTcCall c{wmat, planes, out, resid, ldo, ldr, rows, B, K, tc_planes, prow, e->status};
        return launch_gemm_tc(c, st);
    };

    // the row argmax of the tensor-core LM head meets in e->pval (64-bit keys) and e->pidx (tickets): both are scratch
    // of the matrix-vector LM head otherwise, and at least 8 bytes a sequence
    // (only a decode step of at most max_batch sequences uses them: a prompt's tokens would overrun the buffers)
    const bool row_argmax = !last_token_only && B <= e->cfg.max_batch;
    unsigned long long* arg_keys = row_argmax ? reinterpret_cast<unsigned long long*>(e->pval) : nullptr;
    unsigned* arg_tickets = row_argmax ? reinterpret_cast<unsigned*>(e->pidx) : nullptr;
    // what the launches of this step can serve: the attention split covers n_splits * chunk_pad positions (the new one
    // included) and the RoPE table has rope_n rows; both are fixed by (n_splits, chunk_pad), like a captured graph
    const int pad = chunk_pad_for(a->max_len, ns);
    long long cover = (long long)ns * pad - 1;
    if (cover > e->rope_n - 1) cover = e->rope_n - 1;
    const int len_bound = (int)cover;
    if (chain) {
        // q/k/v | attention | Wo | gate/up | down: each product finishes its rows and writes the planes of the next one, so
        // that nothing stands between them; the residual's planes and the others alternate between two buffers
        const int rows = gemm_cluster_rows(B), ssq_ld = e->chain_rows;
        bf16_raw* xp = reinterpret_cast<bf16_raw*>(e->xplanes);
        LAUNCH(launch_embed_planes(reinterpret_cast<const long long*>(a->token), bf(w.embed), V, e->x, bf(w.ln1), xp, rows, e->ssq, ssq_ld, e->status, B, st,
                                   arg_keys, arg_tickets, a->seq_len, len_bound));
        for (int l = 0; l < L; ++l) {
            ClusterGemmCall c{};
            c.prow = rows; c.n_tok = B; c.ssq = e->ssq; c.ssq_ld = ssq_ld; c.status = e->status;
            ClusterGemmCall q = c;
            q.kind = CL_QKV; q.K = HIDDEN; q.in = xp; q.out = e->qkv;
            q.w[0] = bf(w.wq) + (size_t)l * Q_DIM * HIDDEN; q.w[1] = bf(w.wk) + (size_t)l * KV_DIM * HIDDEN; q.w[2] = bf(w.wv) + (size_t)l * KV_DIM * HIDDEN;
            LAUNCH(launch_gemm_cluster(q, st));

            AttnArgs t{};
            t.qkv = e->qkv; t.seq_k = a->seq_k; t.seq_v = a->seq_v;
            t.seq_layer_stride = reinterpret_cast<const long long*>(a->seq_layer_stride);
            t.seq_len = a->seq_len; t.part = e->part; t.layer = l; t.n_splits = ns; t.chunk_pad = pad; t.len_bound = len_bound;
            t.fused_prep = 1; t.qn = bf(w.qn); t.kn = bf(w.kn); t.rope = e->rope;
            t.k_write = reinterpret_cast<bf16_raw*>(a->k_write); t.v_write = reinterpret_cast<bf16_raw*>(a->v_write);
            t.n_layers = L; t.append = append; t.qp_planes = B < Q3_TC_MIN_BATCH ? 3 : 2;
            if (ns <= ATTN_CLUSTER_MAX) {
                t.planes_out = planes; t.plane_rows = rows; t.cluster = ns > 1; t.early = 1;
                LAUNCH(launch_attn_split(t, B, st));
            } else {   // caches longer than a cluster's splits hold: partials in memory and a merge launch
                LAUNCH(launch_attn_planes(t, planes, rows, 3, B, st));
                ++e->launches;
            }

            ClusterGemmCall o = c;
            o.kind = CL_RESID; o.K = Q_DIM; o.in = planes; o.out = e->x; o.planes = xp; o.gain = bf(w.ln2) + (size_t)l * HIDDEN;
            o.w[0] = bf(w.wo) + (size_t)l * HIDDEN * Q_DIM;
            LAUNCH(launch_gemm_cluster(o, st));
            ClusterGemmCall g = c;
            g.kind = CL_SILU; g.K = HIDDEN; g.in = xp; g.planes = planes;
            g.w[0] = bf(w.wg) + (size_t)l * INTER * HIDDEN; g.w[1] = bf(w.wu) + (size_t)l * INTER * HIDDEN;
            LAUNCH(launch_gemm_cluster(g, st));
            ClusterGemmCall d = c;
            d.kind = CL_RESID; d.K = INTER; d.in = planes; d.out = e->x; d.planes = xp;
            d.gain = l + 1 < L ? bf(w.ln1) + (size_t)(l + 1) * HIDDEN : bf(w.fnorm);
            d.w[0] = bf(w.wd) + (size_t)l * HIDDEN * INTER;
            LAUNCH(launch_gemm_cluster(d, st));
        }
        // The LM head reads the last planes and applies the final norm's scale itself.  Few sequences keep the matrix-vector one: a tile's
        // 64 additions into one accumulator, each truncated, leave logits 9.8e-7 from fp64, fp32 FMAs 1.2e-7 (19 us a step more for three).
        if (V % 128 == 0 && B >= Q3_TC_MIN_BATCH) {
            float* logits = a->logits ? a->logits : e->logits_tc;
            LAUNCH(launch_lm_head(LmHeadCall{bf(w.embed), xp, rows, B, V, e->ssq, ssq_ld, logits, e->status}, st));
            LAUNCH(launch_argmax_rows(logits, V, reinterpret_cast<long long*>(a->next_token), a->seq_len, append, B, st, arg_keys, arg_tickets));
            return Q3_OK;
        }
    } else {
        LAUNCH(launch_embed(reinterpret_cast<const long long*>(a->token), bf(w.embed), V, e->x, e->status, B, st, arg_keys, arg_tickets, a->seq_len, len_bound));
    }
    // The fused path, decode batches of 4..64 sequences: two launches per layer, the split attention and the persistent layer kernel
    // (everything between two attentions: merge, Wo, norm, gate/up, SiLU, down, norm, q/k/v of the next layer).
    const bool lk = layer_kernel && tc && !prompt && layer_tc_supports(e, B);
    if (lk) LAUNCH(launch_layer_tc(e, LK_MODE_FIRST, 0, B, st));
    for (int l = 0; lk && l < L; ++l) {
        AttnArgs t{};
        t.qkv = e->qkv; t.seq_k = a->seq_k; t.seq_v = a->seq_v;
        t.seq_layer_stride = reinterpret_cast<const long long*>(a->seq_layer_stride);
        t.seq_len = a->seq_len; t.part = e->part; t.layer = l; t.n_splits = ns;
        t.chunk_pad = pad; t.len_bound = len_bound;
        t.fused_prep = 1; t.qn = bf(w.qn); t.kn = bf(w.kn); t.rope = e->rope;
        t.k_write = reinterpret_cast<bf16_raw*>(a->k_write); t.v_write = reinterpret_cast<bf16_raw*>(a->v_write);
        t.n_layers = L; t.append = append;
        t.row_ssq = reinterpret_cast<const float*>(e->lk_state);   // the q/k/v rows still lack their norm's scale
        t.merged = e->attn;                                        // the last block of a (sequence, kv head) merges its splits
        t.merge_count = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(e->lk_state) + LK_STATE_MERGE_OFFSET);
        LAUNCH(launch_attn_split(t, B, st));
        LAUNCH(launch_layer_tc(e, l + 1 < L ? LK_MODE_MID : LK_MODE_LAST, l, B, st));
    }
    for (int l = 0; !lk && !chain && l < L; ++l) {
        GemvArgs g{};
        // qkv = rms(x, ln1) @ [wq; wk; wv]^T
        if (tc) {
            // a split-K launch adds its partial tiles onto zeros, which the producer of its input planes writes on the side
            const ZeroRows zq{{e->qkv, nullptr}, {QKV_DIM, 0}, {QKV_DIM, 0}};
            LAUNCH(launch_act_split(e->x, HIDDEN, HIDDEN, bf(w.ln1) + (size_t)l * HIDDEN, planes, prow, tc_planes, B, st,
                                    gemm_tc_splits_k(QKV_DIM, B, HIDDEN) ? &zq : nullptr));
            {   // the three projections in one launch: 32 weight tiles instead of 16 + 8 + 8
                GemmTcGroupCall c{};
                c.n_groups = 3;
                c.w[0] = bf(w.wq) + (size_t)l * Q_DIM * HIDDEN; c.n_rows[0] = Q_DIM; c.out[0] = e->qkv; c.ldo[0] = QKV_DIM;
                c.w[1] = bf(w.wk) + (size_t)l * KV_DIM * HIDDEN; c.n_rows[1] = KV_DIM; c.out[1] = e->qkv + Q_DIM; c.ldo[1] = QKV_DIM;
                c.w[2] = bf(w.wv) + (size_t)l * KV_DIM * HIDDEN; c.n_rows[2] = KV_DIM; c.out[2] = e->qkv + Q_DIM + KV_DIM; c.ldo[2] = QKV_DIM;
                c.x_planes = planes; c.n_tok = B; c.K = HIDDEN; c.nsplit = tc_planes; c.plane_rows = prow; c.status = e->status;
                c.out_is_zero = 1;   // act_split has cleared the rows
                LAUNCH(launch_gemm_tc_group(c, st));
            }
        } else {
            g.seg[0] = {bf(w.wq) + (size_t)l * Q_DIM * HIDDEN, Q_DIM};
            g.seg[1] = {bf(w.wk) + (size_t)l * KV_DIM * HIDDEN, KV_DIM};
            g.seg[2] = {bf(w.wv) + (size_t)l * KV_DIM * HIDDEN, KV_DIM};
            g.x = e->x; g.ldx = HIDDEN; g.gain = bf(w.ln1) + (size_t)l * HIDDEN;
            g.out = e->qkv; g.ldo = QKV_DIM; g.n_rows = QKV_DIM; g.batch = B;
            LAUNCH(launch_gemv(1024, EPI_STORE, g, QKV_DIM / 16, st));
        }

        HeadPrepArgs h{};
        h.qkv = e->qkv; h.qn = bf(w.qn); h.kn = bf(w.kn); h.rope = e->rope; h.seq_len = a->seq_len;
        h.k_write = reinterpret_cast<bf16_raw*>(a->k_write); h.v_write = reinterpret_cast<bf16_raw*>(a->v_write);
        h.seq_k = a->seq_k; h.seq_v = a->seq_v; h.seq_layer_stride = reinterpret_cast<const long long*>(a->seq_layer_stride);
        h.layer = l; h.n_layers = L; h.append = append; h.len_bound = len_bound;
        // A prompt's tokens attend rows that earlier tokens of the same launch append: those need the separate kernel.
        // A decode step prepares the heads inside the attention kernel (one launch less per layer).
        const bool fused_prep = !prompt;
        if (!fused_prep) LAUNCH(launch_head_prep(h, B, st));

        AttnArgs t{};
        t.qkv = e->qkv; t.seq_k = a->seq_k; t.seq_v = a->seq_v;
        t.seq_layer_stride = reinterpret_cast<const long long*>(a->seq_layer_stride);
        t.seq_len = a->seq_len; t.part = e->part; t.layer = l; t.n_splits = ns;
        t.chunk_pad = pad; t.len_bound = len_bound;
        t.fused_prep = fused_prep ? 1 : 0; t.qn = h.qn; t.kn = h.kn; t.rope = h.rope; t.k_write = h.k_write; t.v_write = h.v_write;
        t.n_layers = L; t.append = append;
        if (tc && ns == 1 && fused_prep) {
            // one split: the attention blocks write the Wo GEMM's input planes themselves, no merge launch (the padding rows of the
            // token tile keep whatever they held: their columns of the product are never stored)
            t.planes_out = planes; t.plane_rows = prow;
            LAUNCH(launch_attn_split(t, B, st));
        } else if (tc) {
            LAUNCH(launch_attn_planes(t, planes, prow, tc_planes, B, st));   // the merge writes the Wo GEMM's input planes
            ++e->launches;  // two kernels
        } else {
            LAUNCH(launch_attn(t, e->attn, B, st));
            ++e->launches;  // launch_attn is two kernels
        }

        if (tc) {
            // x += attn @ wo^T
            LAUNCH(gemm(bf(w.wo) + (size_t)l * HIDDEN * Q_DIM, HIDDEN, Q_DIM, e->x, HIDDEN, e->x, HIDDEN));
            // hid = silu(rms(x, ln2) @ wg^T) * (rms(x, ln2) @ wu^T)
            const ZeroRows zf{{e->gate, e->up}, {INTER, INTER}, {INTER, INTER}};
            LAUNCH(launch_act_split(e->x, HIDDEN, HIDDEN, bf(w.ln2) + (size_t)l * HIDDEN, planes, prow, tc_planes, B, st,
                                    gemm_tc_splits_k(2 * INTER, B, HIDDEN) ? &zf : nullptr));
            {   // gate and up in one launch
                GemmTcGroupCall c{};
                c.n_groups = 2;
                c.w[0] = bf(w.wg) + (size_t)l * INTER * HIDDEN; c.n_rows[0] = INTER; c.out[0] = e->gate; c.ldo[0] = INTER;
                c.w[1] = bf(w.wu) + (size_t)l * INTER * HIDDEN; c.n_rows[1] = INTER; c.out[1] = e->up; c.ldo[1] = INTER;
                c.x_planes = planes; c.n_tok = B; c.K = HIDDEN; c.nsplit = tc_planes; c.plane_rows = prow; c.status = e->status;
                c.out_is_zero = 1;   // act_split has cleared the rows
                LAUNCH(launch_gemm_tc_group(c, st));
            }
            // x += (silu(gate) * up) @ wd^T
            LAUNCH(launch_silu_planes(e->gate, e->up, planes, prow, tc_planes, B, st));
            LAUNCH(gemm(bf(w.wd) + (size_t)l * HIDDEN * INTER, HIDDEN, INTER, e->x, HIDDEN, e->x, HIDDEN));
        } else {
            // x += attn @ wo^T
            g = GemvArgs{};
            g.seg[0] = {bf(w.wo) + (size_t)l * HIDDEN * Q_DIM, HIDDEN};
            g.x = e->attn; g.ldx = Q_DIM; g.out = e->x; g.ldo = HIDDEN; g.resid = e->x; g.ldr = HIDDEN;
            g.n_rows = HIDDEN; g.batch = B;
            LAUNCH(launch_gemv(2048, EPI_RESID, g, HIDDEN / 16, st));

            // hid = silu(rms(x, ln2) @ wg^T) * (rms(x, ln2) @ wu^T)
            g = GemvArgs{};
            g.seg[0] = {bf(w.wg) + (size_t)l * INTER * HIDDEN, INTER};
            g.w2 = bf(w.wu) + (size_t)l * INTER * HIDDEN;
            g.x = e->x; g.ldx = HIDDEN; g.gain = bf(w.ln2) + (size_t)l * HIDDEN;
            g.out = e->hid; g.ldo = INTER; g.n_rows = INTER; g.batch = B;
            LAUNCH(launch_gemv(1024, EPI_SILU, g, INTER / 8, st));

            // x += hid @ wd^T
            g = GemvArgs{};
            g.seg[0] = {bf(w.wd) + (size_t)l * HIDDEN * INTER, HIDDEN};
            g.x = e->hid; g.ldx = INTER; g.out = e->x; g.ldo = HIDDEN; g.resid = e->x; g.ldr = HIDDEN;
            g.n_rows = HIDDEN; g.batch = B;
            LAUNCH(launch_gemv(3072, EPI_RESID, g, HIDDEN / 16, st));
        }
    }
    // logits = rms(x, fnorm) @ embed^T ; next_token = argmax
    if (tc && row_argmax && V % 128 == 0 && (a->logits != nullptr || e->logits_tc != nullptr)) {
        float* logits = a->logits ? a->logits : e->logits_tc;
        LAUNCH(launch_act_split(e->x, HIDDEN, HIDDEN, bf(w.fnorm), planes, prow, tc_planes, B, st));
        LAUNCH(gemm(bf(w.embed), V, HIDDEN, logits, V, nullptr, 0));
        LAUNCH(launch_argmax_rows(logits, V, reinterpret_cast<long long*>(a->next_token), a->seq_len, append, B, st, arg_keys, arg_tickets));
    } else {
        // matrix-vector LM head: every sequence, or only the last token of a prompt
        const int nb = last_token_only ? 1 : B;
        if (nb > e->cfg.max_batch) return fail(e, Q3_ERR_INVALID, "decode: %d sequences exceed max_batch %d", nb, e->cfg.max_batch);
        GemvArgs g{};
        g.seg[0] = {bf(w.embed), V};
        g.x = e->x + (last_token_only ? (size_t)(B - 1) * HIDDEN : 0); g.ldx = HIDDEN; g.gain = bf(w.fnorm);
        g.out = a->logits; g.ldo = V; g.n_rows = V; g.batch = nb; g.pval = e->pval; g.pidx = e->pidx;
        int lm_grid = (V + 15) / 16;
        if (lm_grid > e->lm_grid) lm_grid = e->lm_grid;
        LAUNCH(launch_gemv(1024, EPI_LOGITS, g, lm_grid, st));
        LAUNCH(launch_argmax_final(e->pval, e->pidx, lm_grid, reinterpret_cast<long long*>(a->next_token), a->seq_len,
                                   last_token_only ? 0 : append, nb, st));
    }
#undef LAUNCH
    return Q3_OK;
}

extern "C" int q3_decode(q3_engine* e, const q3_decode_args* a, void* stream) {
    if (!e || !a) return fail(e, Q3_ERR_INVALID, "q3_decode: null argument");
    if (!e->have_weights) return fail(e, Q3_ERR_INVALID, "q3_decode: call q3_set_weights first");
    if (!e->rope) return fail(e, Q3_ERR_INVALID, "q3_decode: call q3_set_rope first");
    if (a->batch < 1 || a->batch > e->cfg.max_batch)
        return fail(e, Q3_ERR_INVALID, "q3_decode: batch %d outside 1..%d", a->batch, e->cfg.max_batch);
    if (a->max_len < 0 || a->max_len >= e->rope_n)
        return fail(e, Q3_ERR_INVALID, "q3_decode: max_len %d needs a RoPE table of more than %d rows (have %d)", a->max_len, a->max_len, e->rope_n);
    if (!a->token || !a->seq_k || !a->seq_v || !a->seq_layer_stride || !a->seq_len || !a->next_token)
        return fail(e, Q3_ERR_INVALID, "q3_decode: token, seq_k, seq_v, seq_layer_stride, seq_len and next_token are required");
    CU(e, cudaSetDevice(e->device));
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t path = a->flags & Q3_F_PATH_MASK;
    // One launch of the persistent kernel for one or two sequences, a chain of launches for more; three take the kernel as long as the chain would
    // be plain launches (the times stand at q3_persist.cu's limits).  What a caller captures is replayed without this code: only the chain sees weights that are
    // written in place between two replays, and serves lengths that grow within its split, so it has the captured launches but for those of one sequence up
    // to the length that always was the kernel's.
    bool until_captured = false;
    if (path == Q3_F_PATH_AUTO) {
        path = persist_supports(e, a) ? Q3_F_PATH_PERSIST : Q3_F_PATH_LAYERED;
        if (path == Q3_F_PATH_PERSIST && !persist_serves_replays(a)) {
            cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
            CU(e, cudaStreamIsCapturing(st, &capture));
            if (capture != cudaStreamCaptureStatusNone) path = Q3_F_PATH_LAYERED;
        }
        until_captured = path == Q3_F_PATH_PERSIST && a->batch == 3 && (a->flags & Q3_F_GRAPH);
        if (until_captured) path = Q3_F_PATH_LAYERED;
    }
    if (path == Q3_F_PATH_PERSIST) {
        if (!persist_supports(e, a))
            return fail(e, Q3_ERR_UNSUPPORTED, "q3_decode: the persistent kernel does not serve batch %d at length %d with a RoPE table at %p", a->batch, a->max_len, (const void*)e->rope);
        return persist_decode(e, a, st);
    }
    if (path != Q3_F_PATH_LAYERED && path != Q3_F_PATH_FUSED) return fail(e, Q3_ERR_INVALID, "q3_decode: unknown path flag 0x%x", path);
    const bool layer_kernel = path == Q3_F_PATH_FUSED;
    if (!(a->flags & Q3_F_GRAPH)) return decode_layered(e, a, st, false, layer_kernel);

    // graph replay: the key is the argument block with max_len replaced by what it determines in the captured
    // launches: the split count and the padded chunk length (which also sizes the attention kernel's shared memory)
    q3_decode_args key = *a;
    key.max_len = 0;
    key.reserved = 0;
    const int ns = splits_for(e, a->batch, a->max_len, !layer_kernel && chain_serves(e, a->batch));
    const int pad = chunk_pad_for(a->max_len, ns);
    auto* cache = graph_cache(e);
    GraphEntry* hit = nullptr;
    for (auto& g : *cache)
        if (g.n_splits == ns && g.chunk_pad == pad && !memcmp(&g.key, &key, sizeof(key))) { hit = &g; break; }
    if (!hit) {
        if (cache->size() >= 64) drop_graphs(e);
        cache->push_back(GraphEntry{key, ns, pad, 0, 0, nullptr});
        hit = &cache->back();
    }
    if (hit->exec) {
        CU(e, cudaGraphLaunch(hit->exec, st));
        e->launches += hit->launches;
        return Q3_OK;
    }
    if (hit->seen++ < plain_uses(a->batch, until_captured)) return until_captured ? persist_decode(e, a, st) : decode_layered(e, a, st, false, layer_kernel);
    const int64_t before = e->launches;
    // capture on the engine's own stream (the legacy default stream cannot be captured); nothing runs during capture
    cudaStream_t cs = static_cast<cudaStream_t>(e->capture_stream);
    CU(e, cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    const int rc = decode_layered(e, a, cs, false, layer_kernel);
    cudaGraph_t graph = nullptr;
    const cudaError_t end = cudaStreamEndCapture(cs, &graph);
    if (rc != Q3_OK) { if (graph) cudaGraphDestroy(graph); return rc; }
    if (end != cudaSuccess || !graph) return fail(e, Q3_ERR_CUDA, "q3_decode: stream capture failed: %s", cudaGetErrorString(end));
    hit->launches = e->launches - before;
    e->launches = before;
    const cudaError_t inst = cudaGraphInstantiate(&hit->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (inst != cudaSuccess) { hit->exec = nullptr; return fail(e, Q3_ERR_CUDA, "q3_decode: cudaGraphInstantiate: %s", cudaGetErrorString(inst)); }
    CU(e, cudaGraphLaunch(hit->exec, st));
    e->launches += hit->launches;
    return Q3_OK;
}

// A prompt: five launches a layer (q3_prompt.h).  The activations enter the tensor cores rounded to bf16, like the weights and like
// the cached K/V rows that the prompt's later positions attend anyway.  Measured at 2048 tokens, full model, against the fp32 CPU
// oracle: K/V rows rel-L2 6.6e-3 and logits 5.6e-3 with one plane, 4.0e-3 and 3.2e-3 with two (the cache rounding dominates
// both; the gates are 1e-2 and 2e-2).
// From 64 tokens on the attention is the tiled one over cached rows; fewer tokens keep the split attention, whose own row and
// probabilities are more precise than bf16.
static int prefill_chain(q3_engine* e, const q3_prefill_args* a, const q3_decode_args& s, cudaStream_t st) {
    const int T = a->n_tokens, L = e->cfg.n_layers, V = e->cfg.vocab;
    const q3_weights& w = e->w;
    const bool tiled = T >= 64;
    auto bf = [](const void* p) { return reinterpret_cast<const bf16_raw*>(p); };
    // one plane each of the residual rows, the FFN's hidden rows and the attention's output (three for the split attention, which writes
    // them for its other callers); q's two planes take the place of the fp32 q/k/v rows
    const size_t cap = (size_t)(e->cap + 127) / 128 * 128;
    bf16_raw* xn = reinterpret_cast<bf16_raw*>(e->planes);
    bf16_raw *hid = xn + cap * HIDDEN, *attn = hid + cap * INTER;
    bf16_raw *q_hi = reinterpret_cast<bf16_raw*>(e->qkv), *q_lo = q_hi + (size_t)T * Q_DIM;
    float* ssq = e->gate;
    int parts = PR_SSQ_PARTS;
    CUtensorMap m_xn, m_hid, m_attn, m_qh, m_ql, m_k, m_v;
    const uint32_t box = (uint32_t)prompt_box_rows(T);
    bool ok = tc_make_map(&m_xn, xn, 0, T, HIDDEN, 1, box) && tc_make_map(&m_hid, hid, 0, T, INTER, 1, box) && tc_make_map(&m_attn, attn, 0, T, Q_DIM, 1, box);
    if (tiled)
        ok = ok && tc_make_map(&m_qh, q_hi, 0, T, Q_DIM, 1, 64) && tc_make_map(&m_ql, q_lo, 0, T, Q_DIM, 1, 64) &&
             tc_make_map(&m_k, a->kcache, L, T, KV_DIM, 1, 128, a->cache_capacity) && tc_make_map(&m_v, a->vcache, L, T, KV_DIM, 1, 128, a->cache_capacity);
    if (!ok) return fail(e, Q3_ERR_CUDA, "q3_prefill: a tensor map could not be encoded");
    const int ns = tiled ? 1 : splits_for(e, T, s.max_len, false);
#define LAUNCH(call)                                                                                   \
    do {                                                                                               \
        cudaError_t err__ = (call);                                                                    \
        ++e->launches;                                                                                 \
        if (err__ != cudaSuccess) return fail(e, Q3_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(err__)); \
    } while (0)
    // The products read the RoPE table 16 bytes at a time.  A caller's table may be aligned to a float only: its rows are then copied to a buffer that
    // prompts do not use otherwise.  (A test of the address in the kernel cost 5 us of 1700 at 640 tokens.)
    const float* rope = e->rope;
    if (reinterpret_cast<uintptr_t>(rope) & 15) {
        CU(e, cudaMemcpyAsync(e->up, rope, (size_t)T * HEAD_DIM * sizeof(float), cudaMemcpyDeviceToDevice, st));
        rope = e->up;
    }
    LAUNCH(launch_prompt_embed(reinterpret_cast<const long long*>(a->ids), bf(w.embed), V, e->x, bf(w.ln1), xn, ssq, T, e->status, T, st));
    for (int l = 0; l < L; ++l) {
        PromptGemmCall c{};
        c.T = T; c.ssq = ssq; c.ssq_ld = T; c.parts = &parts; c.status = e->status;
        PromptGemmCall q = c;
        q.kind = PR_QKV; q.K = HIDDEN; q.in = &m_xn;
        q.w[0] = bf(w.wq) + (size_t)l * Q_DIM * HIDDEN; q.w[1] = bf(w.wk) + (size_t)l * KV_DIM * HIDDEN; q.w[2] = bf(w.wv) + (size_t)l * KV_DIM * HIDDEN;
        if (tiled) { q.q_hi = q_hi; q.q_lo = q_lo; }
        else q.qkv = e->qkv;
        const size_t row0 = (size_t)l * a->cache_capacity * KV_DIM;
        q.kc = reinterpret_cast<bf16_raw*>(a->kcache) + row0; q.vc = reinterpret_cast<bf16_raw*>(a->vcache) + row0;
        q.qn = bf(w.qn) + (size_t)l * HEAD_DIM; q.kn = bf(w.kn) + (size_t)l * HEAD_DIM; q.rope = rope;
        LAUNCH(launch_prompt_gemm(q, st));

        if (tiled) {
            LAUNCH(launch_prefill_attn_tc(m_qh, m_ql, m_k, m_v, l, attn, T, e->status, st));
        } else {
            AttnArgs t{};
            t.qkv = e->qkv; t.seq_k = s.seq_k; t.seq_v = s.seq_v;
            t.seq_layer_stride = reinterpret_cast<const long long*>(s.seq_layer_stride);
            t.seq_len = s.seq_len; t.part = e->part; t.layer = l; t.n_splits = ns; t.chunk_pad = chunk_pad_for(s.max_len, ns); t.len_bound = s.max_len;
            t.n_layers = L;
            if (ns == 1) {   // the blocks write the planes themselves: no merge launch (16 / 40 tokens: 1050 / 1020 -> 982 / 1007 us a prompt)
                t.planes_out = attn; t.plane_rows = T;
                LAUNCH(launch_attn_split(t, T, st));
            } else {
                LAUNCH(launch_attn_planes(t, attn, T, 1, T, st));
                ++e->launches;   // two kernels
            }
        }

        PromptGemmCall o = c;
        o.kind = PR_RESID; o.K = Q_DIM; o.in = &m_attn; o.x = e->x; o.xn = xn; o.gain = bf(w.ln2) + (size_t)l * HIDDEN;
        o.w[0] = bf(w.wo) + (size_t)l * HIDDEN * Q_DIM;
        LAUNCH(launch_prompt_gemm(o, st));
        PromptGemmCall g = c;
        g.kind = PR_SILU; g.K = HIDDEN; g.in = &m_xn; g.hid = hid;
        g.w[0] = bf(w.wg) + (size_t)l * INTER * HIDDEN; g.w[1] = bf(w.wu) + (size_t)l * INTER * HIDDEN;
        LAUNCH(launch_prompt_gemm(g, st));
        PromptGemmCall d = c;
        d.kind = PR_RESID; d.K = INTER; d.in = &m_hid; d.x = e->x; d.xn = xn;
        d.gain = l + 1 < L ? bf(w.ln1) + (size_t)(l + 1) * HIDDEN : bf(w.fnorm);
        d.w[0] = bf(w.wd) + (size_t)l * HIDDEN * INTER;
        LAUNCH(launch_prompt_gemm(d, st));
    }
    // the last token's logits
    GemvArgs g{};
    g.seg[0] = {bf(w.embed), V};
    g.x = e->x + (size_t)(T - 1) * HIDDEN; g.ldx = HIDDEN; g.gain = bf(w.fnorm);
    g.out = s.logits; g.ldo = V; g.n_rows = V; g.batch = 1; g.pval = e->pval; g.pidx = e->pidx;
    int lm_grid = (V + 15) / 16;
    if (lm_grid > e->lm_grid) lm_grid = e->lm_grid;
    LAUNCH(launch_gemv(1024, EPI_LOGITS, g, lm_grid, st));
    LAUNCH(launch_argmax_final(e->pval, e->pidx, lm_grid, reinterpret_cast<long long*>(s.next_token), nullptr, 0, 1, st));
#undef LAUNCH
    return Q3_OK;
}

// A prompt of fewer than Q3_TC_MIN_BATCH tokens runs through the layered path as T one-token "sequences" of the same cache, token t at
// position t, in fp32.  head_prep writes every K/V row into the cache before the attention kernels run, so token t attends rows [0, t)
// from the cache (rounded to bf16, as a later decode step will see them) and its own row in fp32.
static int prefill_any(q3_engine* e, const q3_prefill_args* a, cudaStream_t st) {
    const int T = a->n_tokens;
    char* d = reinterpret_cast<char*>(e->pf_desc);
    uint64_t* seq_k = reinterpret_cast<uint64_t*>(d + 64);
    uint64_t* seq_v = seq_k + e->cap;
    long long* stride = reinterpret_cast<long long*>(seq_v + e->cap);
    int* len = reinterpret_cast<int*>(stride + e->cap);
    q3_decode_args s{};
    s.batch = T; s.max_len = T - 1; s.flags = Q3_F_APPEND_KV | Q3_F_PATH_LAYERED;
    s.token = a->ids;
    s.seq_k = seq_k; s.seq_v = seq_v; s.seq_layer_stride = reinterpret_cast<const int64_t*>(stride); s.seq_len = len;
    s.logits = a->last_logits;
    s.next_token = a->next_token ? a->next_token : reinterpret_cast<int64_t*>(d + 32);
    if (T < 64) {   // the split attention takes a prompt's tokens as sequences of the same cache
        cudaError_t err = launch_prefill_desc(seq_k, seq_v, stride, len, reinterpret_cast<uint64_t>(a->kcache), reinterpret_cast<uint64_t>(a->vcache),
                                              (long long)a->cache_capacity * KV_DIM, T, st);
        ++e->launches;
        if (err != cudaSuccess) return fail(e, Q3_ERR_CUDA, "prefill descriptors: %s", cudaGetErrorString(err));
    }
    return T < Q3_TC_MIN_BATCH ? decode_layered(e, &s, st, true) : prefill_chain(e, a, s, st);
}

extern "C" int q3_linear_tc(const void* w, const float* x, float* out, const float* resid, int32_t n_rows, int32_t n_tok, int32_t K,
                            int32_t nsplit, void* planes, int64_t planes_bytes, void* stream) {
    if (!w || !x || !out || !planes) return fail(nullptr, Q3_ERR_INVALID, "q3_linear_tc: null argument");
    if (n_rows < 128 || n_rows % 128 || K < 128 || K % 64 || n_tok < 1 || nsplit < 1 || nsplit > 3)
        return fail(nullptr, Q3_ERR_INVALID, "q3_linear_tc: n_rows=%d (multiple of 128) n_tok=%d K=%d (multiple of 64) nsplit=%d (1..3)", n_rows, n_tok, K, nsplit);
    const int tile = n_tok <= 32 ? 32 : (n_tok <= 64 ? 64 : 128);
    const int plane_rows = (n_tok + tile - 1) / tile * tile;
    const int64_t need = (int64_t)nsplit * plane_rows * K * 2;
    if (planes_bytes < need) return fail(nullptr, Q3_ERR_INVALID, "q3_linear_tc: planes buffer holds %lld bytes, %lld needed", (long long)planes_bytes, (long long)need);
    cudaStream_t st = (cudaStream_t)stream;
    CU(nullptr, launch_act_split(x, K, K, nullptr, reinterpret_cast<bf16_raw*>(planes), plane_rows, nsplit, n_tok, st));
    GemmTcCall c{w, planes, out, resid, n_rows, n_rows, n_rows, n_tok, K, nsplit, plane_rows, nullptr};
    cudaError_t err = launch_gemm_tc(c, st);
    if (err != cudaSuccess) return fail(nullptr, Q3_ERR_CUDA, "q3_linear_tc: %s", cudaGetErrorString(err));
    return Q3_OK;
}

extern "C" int q3_prefill(q3_engine* e, const q3_prefill_args* a, void* stream) {
    if (!e || !a) return fail(e, Q3_ERR_INVALID, "q3_prefill: null argument");
    if (!e->have_weights) return fail(e, Q3_ERR_INVALID, "q3_prefill: call q3_set_weights first");
    if (!e->rope) return fail(e, Q3_ERR_INVALID, "q3_prefill: call q3_set_rope first");
    if (a->n_tokens < 1 || a->n_tokens > e->cfg.max_tokens)
        return fail(e, Q3_ERR_INVALID, "q3_prefill: n_tokens %d outside 1..max_tokens (%d)", a->n_tokens, e->cfg.max_tokens);
    if (a->cache_capacity < a->n_tokens) return fail(e, Q3_ERR_INVALID, "q3_prefill: cache_capacity %d < n_tokens %d", a->cache_capacity, a->n_tokens);
    if (a->n_tokens > e->rope_n) return fail(e, Q3_ERR_INVALID, "q3_prefill: RoPE table has %d rows, need %d", e->rope_n, a->n_tokens);
    if (!a->ids || !a->kcache || !a->vcache) return fail(e, Q3_ERR_INVALID, "q3_prefill: ids, kcache and vcache are required");
    CU(e, cudaSetDevice(e->device));
    return prefill_any(e, a, (cudaStream_t)stream);
}
