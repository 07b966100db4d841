// Host side of the C ABI declared in include/pagoda_sampler.h: handle lifecycle, grammar table
// uploads, staging of host-resident batches and kernel launches.  No CPU fallback: every entry
// point either runs the CUDA kernels or returns an error.
#include "../../include/pagoda_sampler.h"

#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <new>
#include <vector>

#include "pgs_args.cuh"
#include "pgs_kinds.cuh"
#include "pgs_stream.cuh"
#include "pgs_tp.cuh"
#include "pgs_wide.cuh"

namespace pgs {
cudaError_t configure_general();
cudaError_t launch_general(const RowArgs& a, uint32_t grid, cudaStream_t stream);
size_t general_smem_bytes();

size_t stream_smem_bytes();
cudaError_t configure_stream();
cudaError_t stream_ctas_per_sm(int* out);
cudaError_t launch_stream(const RowArgs& a, const StreamLaunch& sl, uint32_t grid, uint32_t csize, cudaStream_t stream);
cudaError_t stream_max_clusters(int csize, int* out);
cudaError_t configure_wide();
cudaError_t launch_wide(const RowArgs& a, const WideLaunch& l, uint32_t slots, uint32_t grid, cudaStream_t stream);
struct ScoreArgs {
    const float* logits;
    unsigned long long row_stride;
    uint32_t rows, vocab;
    const uint32_t* ids;
    float* out_gather;
    float* out_full;
    int32_t* status;
};
cudaError_t configure_score();
cudaError_t launch_log_softmax(const ScoreArgs& a, uint32_t grid, cudaStream_t stream);
cudaError_t configure_tp();
cudaError_t launch_tp_push(const TpArgs& a, cudaStream_t stream);
cudaError_t launch_tp_merge(const TpArgs& a, const TpOut& o, uint32_t sms, cudaStream_t stream);
cudaError_t launch_draft_accept(const uint32_t* row_argmax, const uint32_t* draft, uint32_t sequences,
                                uint32_t positions, uint32_t* accepted, uint32_t* next, cudaStream_t stream);
}  // namespace pgs

static thread_local char g_create_error[256] = "";

struct pgs_handle {
    int device = 0;
    int sm_count = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t last_stream = nullptr;   // stream of the step before: steps of one handle share its scratch and must not overlap
    cudaEvent_t ev_step = nullptr;
    uint32_t max_rows = 0, max_vocab = 0, max_history = 0;
    uint32_t slots = 0, vocab_pad = 0, sort_pad = 0, hash_cap = 0;
    // scratch slots
    float* sx = nullptr;
    uint32_t* sl_id = nullptr;
    float* sl_p = nullptr;
    unsigned long long* sl_key = nullptr;
    uint32_t* sh_key = nullptr;
    uint32_t* sh_cnt = nullptr;
    // grammar tables
    pgs::TableDir tables_host[pgs::MAX_TABLES];
    pgs::TableDir* tables_dev = nullptr;
    // staging for host-resident batches
    void* logits_stage = nullptr;
    size_t logits_stage_bytes = 0;
    unsigned char* aux_host = nullptr;   // pinned
    unsigned char* aux_dev = nullptr;
    size_t aux_bytes = 0;
    // rows that the row kernel hands on (work list)
    uint32_t* work_rows = nullptr;
    uint32_t* work_count = nullptr;   // [2]
    uint32_t* tp_done = nullptr;      // CTAs finished in the current peer-store push
    int exact = 0;
    // wide kernel: its workspaces (one block of device memory)
    unsigned char* wide_ws = nullptr;
    pgs::WideLaunch wide = {};
    pgs::WideLaunch score_wide = {};  // scoring: its own workspace
    uint32_t* score_done = nullptr;   // pinned: the last of the calls that used it to have ended
    uint32_t score_calls = 0;         // how many there were
    unsigned long long score_stream = 0;   // id of the last one's stream
    uint32_t wide_vocab = 0;          // longest row the workspace holds
    int wide_route = 0;               // tests: 1 always the grid, 2 always the general kernel, 3 always the wide kernel's CTA per row
    // streaming row kernel: id -> count slots, shared memory and CTAs per SM, the gate's counter
    uint32_t stream_hash = 0, stream_cohort = 0;
    int max_clusters[4] = {0, 0, 0, 0};   // resident clusters of 1 (unused), 2, 4, 8 CTAs of the row kernel
    int cluster_mode = 1;                 // PGS_CLUSTER=0 turns row sharing off
    size_t stream_smem = 0;
    int stream_ctas = 0;
    uint32_t* p1_done = nullptr;      // device counter: rows that finished their first pass, over all launches
    uint32_t done_total = 0;          // the value that counter has when every launch so far has completed
    unsigned long long* faulted = nullptr;   // device counters: [0] ROW_NONFINITE rows, [1] rows whose exchange wait ran out
    unsigned long long* tp_timeouts = nullptr;   // = faulted + 1
    unsigned long long timeouts_seen = 0;    // value of the second counter at the last pgs_tp_exchange_status
    uint32_t wait_polls = 1u << 21;          // bound of the merge's flag wait (about a second)
    cudaStream_t tp_stream = nullptr;        // stream of the last pgs_tp_merge_wait
    long long* prof = nullptr;        // phase timers of the row kernel (PGS_PROFILE=1)
    pgs_counters counters = {};
    char err[256] = "";
};

static int fail(pgs_handle* h, int code, const char* fmt, ...) {
    char* dst = h ? h->err : g_create_error;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(dst, 256, fmt, ap);
    va_end(ap);
    return code;
}

#define PGS_CUDA(h, call)                                                                  \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            cudaGetLastError(); /* a reported error must not resurface at the next launch */ \
            return fail(h, e_ == cudaErrorMemoryAllocation ? PGS_ERR_NOMEM : PGS_ERR_CUDA, \
                        "%s: %s", #call, cudaGetErrorString(e_));                          \
        }                                                                                  \
    } while (0)

namespace {
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && prev != cur) cudaSetDevice(prev);
    }
};

uint32_t pow2_at_least(uint32_t v, uint32_t lo) {
    uint32_t p = lo;
    while (p < v) p <<= 1;
    return p;
}
}  // namespace

namespace {
// The wide kernel's workspaces in one block of device memory.  Steps: as many rows of the handle's vocabulary as there are SMs, or
// as the handle has (the grid takes W_CHUNK of them at a time).  Scoring has its own, of as many rows as SMs: it has no row
// limit, and is not ordered with the handle's steps.
int wide_workspace(pgs_handle* h) {
    using namespace pgs;
    const uint32_t vocab = h->max_vocab < (uint32_t)W_MAX_VOCAB ? h->max_vocab : (uint32_t)W_MAX_VOCAB;
    const uint32_t regions = (vocab + W_REGION - 1) / W_REGION;
    size_t used = 0, zeroed = 0;
    unsigned char* base = nullptr;
    auto take = [&](size_t bytes) { unsigned char* const p = (unsigned char*)((uintptr_t)base + used); used += (bytes + 255) & ~size_t(255); return p; };
    auto plan = [&]() {
        used = 0;
        WideLaunch* const both[2] = {&h->wide, &h->score_wide};
        for (WideLaunch* l : both) { l->sync = (uint32_t*)take(64); l->left_count = (uint32_t*)take(4); }
        h->wide.own = (uint32_t*)take((size_t)h->slots * W_OWN * 4); h->score_wide.own = (uint32_t*)take((size_t)h->sm_count * W_OWN * 4);
        zeroed = used;
        for (WideLaunch* l : both) {
            const size_t rows = l == &h->score_wide ? (uint32_t)h->sm_count : h->slots;   // (one CTA per row: as many as there are SMs)
            l->chunk = rows < W_CHUNK ? (uint32_t)rows : W_CHUNK; l->reg_stride = regions; l->rs_stride = regions + 1u;
            l->row = (WideRow*)take(rows * sizeof(WideRow)); l->reg = (float2*)take(rows * regions * sizeof(float2));
            l->cell = (float4*)take(rows * regions * sizeof(float4)); l->seg = (uint2*)take(rows * regions * sizeof(uint2));
            l->pre = (float*)take(rows * regions * 4); l->terms = (float*)take(rows * (size_t)W_TERMS * W_REGION * 4);
        }
        // steps only
        WideLaunch& l = h->wide;
        const size_t rows = h->slots;
        l.left_rows = (uint32_t*)take((size_t)h->max_rows * 4); l.rs = (uint32_t*)take(rows * (regions + 1u) * 4);
        l.ent_id = (uint32_t*)take(rows * (W_MAX_HIST + 32) * 4); l.ent_xn = (float*)take(rows * (W_MAX_HIST + 32) * 4);
        l.hist = (uint32_t*)take(rows * W_BUCKETS * 4);
    };
    plan();
    PGS_CUDA(nullptr, cudaMalloc(&h->wide_ws, used));
    PGS_CUDA(nullptr, cudaMemsetAsync(h->wide_ws, 0, zeroed, h->stream));
    base = h->wide_ws;
    plan();
    h->wide.list = h->sl_key; h->wide.list_stride = h->sort_pad;   // (free until the launch's own leftovers go to general_rows)
    h->wide.polls = 1u << 23;
    if (const char* ev = getenv("PGS_GRID_POLLS")) h->wide.polls = (uint32_t)strtoul(ev, nullptr, 10);
    if (const char* ev = getenv("PGS_WIDE_ROUTE")) h->wide_route = atoi(ev);
    h->wide.gave_up = h->tp_timeouts;
    h->score_wide.polls = h->wide.polls; h->score_wide.gave_up = h->wide.gave_up;
    h->score_wide.score = 1u;
    h->wide_vocab = vocab;
    return PGS_OK;
}

// Every step of a handle uses the same scratch, lists and counters: a step on another stream than the one before waits for
// that one to finish on the device.
int order_steps(pgs_handle* h, cudaStream_t stream) {
    if (stream != h->last_stream) {
        PGS_CUDA(h, cudaEventRecord(h->ev_step, h->last_stream));
        PGS_CUDA(h, cudaStreamWaitEvent(stream, h->ev_step, 0));
        h->last_stream = stream;
    }
    return PGS_OK;
}

// Whether a scoring call on `stream` may use the scoring workspace.  Scoring is not ordered with anything but its own stream:
// while a call on another stream may still be running, or where the call is being captured (a graph may be replayed at any
// time), it takes the kernel that needs no workspace.  Streams are compared by their ids, which are never used again, and the
// kernel says in a word of host memory that it is done.  (An event behind every call and a wait for it: 64 rows of 151936 86 us
// in place of 83.)
bool score_workspace_free(const pgs_handle* h, cudaStream_t stream, unsigned long long* id) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone ||
        cudaStreamGetId(stream, id) != cudaSuccess) { cudaGetLastError(); return false; }
    const bool done = *(volatile uint32_t*)h->score_done == h->score_calls;
    std::atomic_thread_fence(std::memory_order_acquire);
    return done || *id == h->score_stream;
}

// How a batch is scored: by the kernel that needs no workspace, by the wide kernel's grid, or by its CTA per row.  Lines through
// (us, without workspace / grid / CTA per row): 1 x 1000 21 / 38 / 41, 64 x 1000 25 / 42 / 33, 64 x 4096 37 / 44 / 36, 64 x 16384
// 53 / 47 / 42, 148 x 16384 54 / 115 / 41, 16 x 50256 94 / 47 / 56, 64 x 50256 97 / 54 / 55, 256 x 50256 186 / 194 / 106, 64 x 151936
// 201 / 80 / 86, 256 x 151936 407 / 274 / 174; whole vectors 64 x 1000 26 / 51 / 41, 64 x 16384 64 / 58 / 54, 64 x 50256 128 / 76 / 95,
// 256 x 50256 256 / 285 / 196, 64 x 151936 305 / 149 / 201.
enum ScoreRoute { SCORE_PLAIN, SCORE_GRID, SCORE_ROWS };
ScoreRoute score_route(const pgs_handle* h, uint32_t rows, uint32_t vocab, bool full) {
    if (h->wide_route) return h->wide_route == 1 ? SCORE_GRID : h->wide_route == 2 ? SCORE_PLAIN : SCORE_ROWS;
    const uint32_t sms = (uint32_t)h->sm_count, chunk = h->score_wide.chunk;
    const double v = 1e-6 * vocab, waves = (rows - 1u) / sms + 1u, chunks = (rows - 1u) / chunk + 1u, in_chunk = rows < chunk ? rows : chunk;
    const double plain = waves * (25.0 + v * (full ? 2000.0 : 1176.0));
    const double grid = chunks * (full ? 53.0 + 10.0 * v * in_chunk : 43.0 + 3.8 * v * in_chunk);
    const double by_rows = waves * ((full ? 40.0 + 960.0 * v : 34.0 + 330.0 * v) + 0.9 * v * (rows < sms ? rows : sms));
    return plain <= grid && plain <= by_rows ? SCORE_PLAIN : grid <= by_rows ? SCORE_GRID : SCORE_ROWS;
}

// The combinations of kinds that one CTA per row does quicker (*row), and those that the grid does (returned), among those
// that the handle's rows can have.
uint32_t kinds_for(const pgs_handle* h, uint32_t rows, uint32_t vocab, uint32_t* row, pgs::KindsWay way = pgs::WAY_GRID) {
    using namespace pgs;
    const uint32_t possible = h->max_history > (uint32_t)W_MAX_HIST ? WK_POSSIBLE : WK_SHORT;
    *row = h->wide_route == 1 || h->wide_route == 3 ? 0u : h->wide_route == 2 ? possible : kinds_one_cta_each(possible, rows, h->wide.chunk, h->slots, vocab, way);
    return possible & ~*row;
}

// Whether the wide kernel takes an exact or unaligned batch one CTA per row, as many at a time as there are SMs, and not with the
// whole grid on 64 rows at a time: without grid barriers, but with a row's regions on one SM.  Lines through what sampled rows take
// (us, CTA per row / grid): 1 x 16384 41 / 46, 16 x 50256 53 / 47, 64 x 16384 40 / 48, 64 x 50256 56 / 58, 64 x 100000 70 / 64,
// 64 x 151936 96 / 88, 48 x 50257 with histories 63 / 59, 148 x 4096 56 / 240, 148 x 50256 59 / 153, 148 x 151936 118 / 226, 256 x 50256 111 / 225, 256 x 151936
// 187 / 316; without top-k and with top-p 0.9 16 x 16384 65 / 105, 64 x 16384 70 / 126, 256 x 50256 191 / 619; greedy 64 x 50256 21 / 28.
bool wide_row_by_row(const pgs_handle* h, uint32_t rows, uint32_t vocab) {
    if (h->wide_route) return h->wide_route == 3;
    const uint32_t chunk = h->wide.chunk, slots = h->slots;
    const double v = 1e-6 * vocab;
    const double by_rows = ((rows - 1u) / slots + 1u) * (36.0 + 400.0 * v + 1.2 * v * (rows < slots ? rows : slots));
    const double grid = ((rows - 1u) / chunk + 1u) * (44.0 + 4.4 * v * (rows < chunk ? rows : chunk));
    return by_rows < grid;
}

// CTAs of the wide kernel for `rows` rows: one per SM, fewer where a CTA would get less than a handful of regions (its grid
// barriers cost more with more CTAs).
uint32_t wide_grid(const pgs_handle* h, uint32_t rows, uint32_t vocab) {
    const uint64_t share = ((uint64_t)rows * ((vocab + pgs::W_REGION - 1) / pgs::W_REGION) + 7u) / 8u;
    const uint64_t want = share > rows ? share : rows;
    return want < (uint64_t)h->sm_count ? (uint32_t)want : (uint32_t)h->sm_count;
}
}  // namespace

extern "C" const char* pgs_last_error(const pgs_handle* h) { return h ? h->err : g_create_error; }

static int destroy_impl(pgs_handle* h) {
    DeviceGuard g(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->score_done && *(volatile uint32_t*)h->score_done != h->score_calls) cudaDeviceSynchronize();
    for (int t = 0; t < pgs::MAX_TABLES; t++) {
        if (h->tables_host[t].live) {
            cudaFree((void*)h->tables_host[t].words);
            cudaFree((void*)h->tables_host[t].flags);
        }
    }
    cudaFree(h->sx); cudaFree(h->sl_id); cudaFree(h->sl_p); cudaFree(h->sl_key);
    cudaFree(h->sh_key); cudaFree(h->sh_cnt); cudaFree(h->tables_dev);
    cudaFree(h->logits_stage); cudaFree(h->aux_dev); cudaFree(h->work_rows); cudaFree(h->work_count); cudaFree(h->tp_done); cudaFree(h->prof);
    cudaFree(h->p1_done); cudaFree(h->faulted); cudaFree(h->wide_ws);
    if (h->aux_host) cudaFreeHost(h->aux_host);
    if (h->ev_step) cudaEventDestroy(h->ev_step);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return PGS_OK;
}

extern "C" int pgs_create(int device, uint32_t max_rows, uint32_t max_vocab, uint32_t max_history,
                          pgs_handle** out) {
    if (!out) return fail(nullptr, PGS_ERR_INVALID, "pgs_create: out is NULL");
    *out = nullptr;
    if (max_rows == 0 || max_vocab == 0 || max_vocab > (1u << 24) || max_history > (1u << 22))
        return fail(nullptr, PGS_ERR_INVALID,
                    "pgs_create: need 1 <= max_rows, 1 <= max_vocab <= 2^24, max_history <= 2^22");
    int n_dev = 0;
    cudaError_t e = cudaGetDeviceCount(&n_dev);
    if (e != cudaSuccess || n_dev == 0)
        return fail(nullptr, PGS_ERR_CUDA, "pgs_create: no CUDA device (%s); this library has no CPU path",
                    cudaGetErrorString(e));
    if (device < 0 || device >= n_dev)
        return fail(nullptr, PGS_ERR_INVALID, "pgs_create: device %d out of range (0..%d)", device, n_dev - 1);
    pgs_handle* h = new (std::nothrow) pgs_handle();
    if (!h) return fail(nullptr, PGS_ERR_NOMEM, "pgs_create: out of host memory");
    h->device = device;
    memset(h->tables_host, 0, sizeof h->tables_host);
    DeviceGuard g(device);
    int rc = [&]() -> int {
        cudaDeviceProp prop;
        PGS_CUDA(nullptr, cudaGetDeviceProperties(&prop, device));
        if (prop.major < 10)
            return fail(nullptr, PGS_ERR_CUDA, "pgs_create: device %d is sm_%d%d; this library is built for sm_100a",
                        device, prop.major, prop.minor);
        h->sm_count = prop.multiProcessorCount;
        PGS_CUDA(nullptr, cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
        PGS_CUDA(nullptr, cudaEventCreateWithFlags(&h->ev_step, cudaEventDisableTiming));
        h->last_stream = h->stream;
        PGS_CUDA(nullptr, pgs::configure_general());
        PGS_CUDA(nullptr, pgs::configure_tp());
        PGS_CUDA(nullptr, pgs::configure_score());
        PGS_CUDA(nullptr, pgs::configure_wide());
        PGS_CUDA(nullptr, cudaMalloc(&h->work_rows, (size_t)max_rows * sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMalloc(&h->work_count, 2 * sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMemsetAsync(h->work_count, 0, 2 * sizeof(uint32_t), h->stream));
        PGS_CUDA(nullptr, cudaMalloc(&h->tp_done, sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMemsetAsync(h->tp_done, 0, sizeof(uint32_t), h->stream));
        PGS_CUDA(nullptr, cudaMalloc(&h->p1_done, sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMemsetAsync(h->p1_done, 0, sizeof(uint32_t), h->stream));
        PGS_CUDA(nullptr, cudaMalloc(&h->faulted, 2 * sizeof(unsigned long long)));
        PGS_CUDA(nullptr, cudaMemsetAsync(h->faulted, 0, 2 * sizeof(unsigned long long), h->stream));
        h->tp_timeouts = h->faulted + 1;
        h->stream_hash = pow2_at_least(2 * (max_history ? max_history : 1), 64);
        if (h->stream_hash > (uint32_t)pgs::S_MAX_HASH) h->stream_hash = pgs::S_MAX_HASH;   // longer histories go on the work list
        h->stream_smem = pgs::stream_smem_bytes();
        PGS_CUDA(nullptr, pgs::configure_stream());
        PGS_CUDA(nullptr, pgs::stream_ctas_per_sm(&h->stream_ctas));
        if (h->stream_ctas < 1) return fail(nullptr, PGS_ERR_CUDA, "pgs_create: the row kernel does not fit an SM (%zu bytes of shared memory)", h->stream_smem);
        // rows that may be in their first pass at once: no limit by default (measured on 256 x 151936: a limit of
        // about an SM count keeps pass 2 in L2 but leaves half the threads of every SM waiting at the gate)
        h->stream_cohort = 0xffffffffu;
        if (const char* ev = getenv("PGS_COHORT")) { if (atoi(ev) > 0) h->stream_cohort = (uint32_t)atoi(ev); }
        if (const char* ev = getenv("PGS_CLUSTER")) h->cluster_mode = atoi(ev);
        for (int i = 1; i < 4; i++) {
            if (pgs::stream_max_clusters(1 << i, &h->max_clusters[i]) != cudaSuccess) { cudaGetLastError(); h->max_clusters[i] = 0; }
        }
        if (const char* ev = getenv("PGS_EXACT")) h->exact = atoi(ev);
        if (const char* ev = getenv("PGS_PROFILE")) {
            if (atoi(ev)) {
                PGS_CUDA(nullptr, cudaMalloc(&h->prof, 1024 * 16 * sizeof(long long)));
                PGS_CUDA(nullptr, cudaMemsetAsync(h->prof, 0, 1024 * 16 * sizeof(long long), h->stream));
            }
        }
        h->max_rows = max_rows; h->max_vocab = max_vocab; h->max_history = max_history;
        h->slots = max_rows < (uint32_t)h->sm_count ? max_rows : (uint32_t)h->sm_count;
        h->vocab_pad = (max_vocab + 31u) & ~31u;
        h->sort_pad = pow2_at_least(max_vocab, 2);
        h->hash_cap = pow2_at_least(2 * (max_history ? max_history : 1), 64);
        const size_t s = h->slots;
        PGS_CUDA(nullptr, cudaMalloc(&h->sx, s * h->vocab_pad * sizeof(float)));
        PGS_CUDA(nullptr, cudaMalloc(&h->sl_id, s * h->vocab_pad * sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMalloc(&h->sl_p, s * h->vocab_pad * sizeof(float)));
        PGS_CUDA(nullptr, cudaMalloc(&h->sl_key, s * h->sort_pad * sizeof(unsigned long long)));
        PGS_CUDA(nullptr, cudaMalloc(&h->sh_key, s * h->hash_cap * sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMalloc(&h->sh_cnt, s * h->hash_cap * sizeof(uint32_t)));
        PGS_CUDA(nullptr, cudaMalloc(&h->tables_dev, sizeof h->tables_host));
        PGS_CUDA(nullptr, cudaMemsetAsync(h->tables_dev, 0, sizeof h->tables_host, h->stream));
        const int rc_wide = wide_workspace(h);
        if (rc_wide != PGS_OK) return rc_wide;
        // aux staging: per-row parameter and output arrays of a host-resident batch
        h->aux_bytes = (size_t)max_rows * 128 + (size_t)max_rows * max_history * 4 + 4096;
        PGS_CUDA(nullptr, cudaMalloc(&h->aux_dev, h->aux_bytes));
        const size_t staged = (h->aux_bytes + 63) & ~size_t(63);
        PGS_CUDA(nullptr, cudaMallocHost(&h->aux_host, staged + 64));
        h->score_done = (uint32_t*)(h->aux_host + staged);
        *h->score_done = 0u;
        PGS_CUDA(nullptr, cudaStreamSynchronize(h->stream));
        return PGS_OK;
    }();
    if (rc != PGS_OK) {
        destroy_impl(h);
        return rc;
    }
    *out = h;
    return PGS_OK;
}

extern "C" int pgs_destroy(pgs_handle* h) {
    if (!h) return PGS_OK;
    return destroy_impl(h);
}

extern "C" void* pgs_stream(pgs_handle* h) { return h ? (void*)h->stream : nullptr; }

extern "C" int pgs_get_counters(const pgs_handle* h, pgs_counters* out) {
    if (!h || !out) return PGS_ERR_INVALID;
    *out = h->counters;
    // faulted rows are counted on the device by the kernels that find them
    DeviceGuard g(h->device);
    unsigned long long f = 0;
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e == cudaSuccess && h->last_stream != h->stream) e = cudaStreamSynchronize(h->last_stream);
    if (e == cudaSuccess) e = cudaMemcpy(&f, h->faulted, sizeof f, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { cudaGetLastError(); return PGS_ERR_CUDA; }
    out->rows_faulted = f;
    return PGS_OK;
}

extern "C" int pgs_mask_table_upload(pgs_handle* h, uint32_t n_states, uint32_t words_per_state,
                                     const uint32_t* host_words, const uint8_t* state_flags,
                                     int32_t* table_id) {
    if (!h) return PGS_ERR_INVALID;
    if (!host_words || !table_id || n_states == 0 || words_per_state == 0)
        return fail(h, PGS_ERR_INVALID, "pgs_mask_table_upload: empty table or NULL argument");
    int t = -1;
    for (int i = 0; i < pgs::MAX_TABLES; i++)
        if (!h->tables_host[i].live) { t = i; break; }
    if (t < 0) return fail(h, PGS_ERR_LIMIT, "pgs_mask_table_upload: all %d table slots in use", pgs::MAX_TABLES);
    DeviceGuard g(h->device);
    uint32_t* words = nullptr;
    uint8_t* flags = nullptr;
    const size_t wbytes = (size_t)n_states * words_per_state * sizeof(uint32_t);
    PGS_CUDA(h, cudaMalloc(&words, wbytes));
    cudaError_t e = cudaMalloc(&flags, n_states);
    if (e != cudaSuccess) { cudaFree(words); return fail(h, PGS_ERR_NOMEM, "cudaMalloc(flags): %s", cudaGetErrorString(e)); }
    std::vector<uint8_t> zero;
    if (!state_flags) { zero.assign(n_states, 0); state_flags = zero.data(); }
    pgs::TableDir d;
    d.words = words; d.flags = flags; d.words_per_state = words_per_state; d.n_states = n_states;
    d.live = 1; d.pad = 0;
    e = cudaMemcpyAsync(words, host_words, wbytes, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(flags, state_flags, n_states, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h->tables_dev + t, &d, sizeof d, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) {
        cudaFree(words); cudaFree(flags);
        return fail(h, PGS_ERR_CUDA, "pgs_mask_table_upload: %s", cudaGetErrorString(e));
    }
    h->tables_host[t] = d;
    *table_id = t;
    return PGS_OK;
}

extern "C" int pgs_mask_table_free(pgs_handle* h, int32_t table_id) {
    if (!h) return PGS_ERR_INVALID;
    if (table_id < 0 || table_id >= pgs::MAX_TABLES || !h->tables_host[table_id].live)
        return fail(h, PGS_ERR_INVALID, "pgs_mask_table_free: table %d is not live", table_id);
    DeviceGuard g(h->device);
    pgs::TableDir d = h->tables_host[table_id];
    pgs::TableDir dead;
    memset(&dead, 0, sizeof dead);
    PGS_CUDA(h, cudaMemcpyAsync(h->tables_dev + table_id, &dead, sizeof dead, cudaMemcpyHostToDevice, h->stream));
    PGS_CUDA(h, cudaStreamSynchronize(h->stream));
    cudaFree((void*)d.words);
    cudaFree((void*)d.flags);
    h->tables_host[table_id] = dead;
    return PGS_OK;
}

// ------------------------------------------------------------------------------ batches

namespace {

// One step: the streaming row kernel serves every row it can and lists the others, which the wide kernel then processes.
// In exact mode, and where no row is 16-byte aligned, every row goes to the wide kernel at once.
int launch_step(pgs_handle* h, pgs::RowArgs& a, cudaStream_t stream) {
    const uint32_t rows = a.rows;
    const uint32_t grid = rows < h->slots ? rows : h->slots;
    a.faulted = h->faulted;
    const int rc = order_steps(h, stream);
    if (rc != PGS_OK) return rc;
    const bool wide = !a.tp_records && a.vocab <= h->wide_vocab;   // (shard records and longer rows: the general kernel)
    const uint32_t per = a.dtype == 0 ? 4u : 8u;
    const bool aligned = ((uintptr_t)a.logits & 15u) == 0u && a.row_stride % per == 0u && a.vocab % per == 0u;
    if (h->exact || a.vocab > (uint32_t)pgs::S_MAX_VOCAB || (wide && !aligned)) {
        // What the rows ask for is known on the device only: where both ways are in question, both kernels are launched, and
        // the one whose batch it is not returns at once.  Many short rows (the two kernels share no SM then) are all done by the wide
        // kernel, which runs the general kernel's code itself.  General kernel alone / both / wide kernel alone, us: 148 x 4096 greedy
        // 6.2 / 10.3 / 9.4, top-k 5 61 / 42 / 38; 200 x 12000 greedy 14 / 18 / 20, top-k 50 160 / 79 / 73; 16 x 4096 greedy 6.2 / 8.2 / 9.1.
        // (That code has little L1 there, and long histories want it.)
        pgs::WideLaunch wl = h->wide;
        uint32_t grid_kinds = 0u, row_kinds = 0u;
        wl.local = wide && wide_row_by_row(h, rows, a.vocab);
        const bool alone = wl.local && rows > (uint32_t)h->sm_count / 2u && a.vocab < 16384u && h->max_history <= (uint32_t)pgs::W_MAX_HIST;
        if (wide) grid_kinds = kinds_for(h, rows, a.vocab, &row_kinds, alone ? pgs::WAY_ROWS_ALONE : wl.local ? pgs::WAY_ROWS : pgs::WAY_GRID);
        if (alone) wl.kinds_row[0] = wl.kinds_row[1] = row_kinds;
        else wl.kinds_front = row_kinds;
        wl.look = row_kinds != 0u;
        if (!wide || !grid_kinds || wl.kinds_front) {
            pgs::RowArgs front = a;
            if (wide && grid_kinds) front.kinds_here = wl.kinds_front;
            PGS_CUDA(h, pgs::launch_general(front, grid, stream));
            h->counters.kernel_launches += 1;
        }
        if (grid_kinds) {
            // (both fit on no SM together)
            const uint32_t want = wide_grid(h, rows, a.vocab), sms = (uint32_t)h->sm_count, room = wl.kinds_front && rows <= sms / 2u ? sms - rows : sms;
            PGS_CUDA(h, pgs::launch_wide(a, wl, h->slots, wl.local ? grid : want < room ? want : room, stream));
            h->counters.kernel_launches += 1;
        }
        return PGS_OK;
    }
    pgs::StreamLaunch sl;
    sl.hash_slots = h->stream_hash; sl.cohort = h->stream_cohort;
    sl.done_base = h->done_total; sl.gate_polls = 1u << 16;   // x 200 ns: gives up after about 13 ms
    sl.p1_done = h->p1_done;
    sl.work_rows = h->work_rows; sl.work_count = h->work_count;
    sl.prof = h->prof;
    const uint32_t resident = (uint32_t)h->stream_ctas * (uint32_t)h->sm_count;
    // Small batches: the CTAs of a cluster share every row, with the largest cluster size that still has all rows
    // resident at once (a row alone on one CTA is bound by latency, not by bandwidth).
    uint32_t csize = 1;
    if (h->cluster_mode && !a.tp_records)
        for (int i = 3; i >= 2; i--)   // (pairs do not pay: two CTAs per row with half the rows' CTAs measured slower)
            if (h->max_clusters[i] > 0 && rows <= (uint32_t)h->max_clusters[i]) { csize = 1u << i; break; }
    PGS_CUDA(h, pgs::launch_stream(a, sl, csize > 1 ? rows : (rows < resident ? rows : resident), csize, stream));
    h->done_total += rows;
    // The list is usually empty.  The pass over it is set up while the row kernel still runs (programmatic stream
    // serialization) and returns at once when it finds nothing listed.
    pgs::RowArgs wl = a;
    wl.work_rows = h->work_rows;
    wl.work_count = h->work_count;
    if (wide) {
        // A CTA of the wide kernel fits on no SM that still runs the row kernel.  Where a small batch leaves most SMs free,
        // the pass takes only those, and is in place before the rows are done.
        const uint32_t busy = rows * csize, want = wide_grid(h, rows, a.vocab), sms = (uint32_t)h->sm_count;
        const uint32_t room = csize > 1u && busy <= sms / 2u ? sms - busy : sms;
        pgs::WideLaunch l = h->wide;   // (how many rows are listed is known on the device only)
        kinds_for(h, rows < l.chunk ? rows : l.chunk, a.vocab, &l.kinds_row[0]);
        if (rows > l.chunk) kinds_for(h, rows, a.vocab, &l.kinds_row[1]);
        // (one or two short rows without top-k: see listed_one_cta_each)
        if (a.vocab < 1800u) { kinds_for(h, 1u, a.vocab, &l.kinds_row[2], pgs::WAY_ROWS); kinds_for(h, 2u, a.vocab, &l.kinds_row[3], pgs::WAY_ROWS); }
        l.look = (l.kinds_row[0] | l.kinds_row[1] ? 1u : 0u) | (l.kinds_row[2] | l.kinds_row[3] ? 2u : 0u);
        l.local = h->wide_route == 0 ? 2u : h->wide_route == 3 ? 1u : 0u;
        PGS_CUDA(h, pgs::launch_wide(wl, l, h->slots, want < room ? want : room, stream));
    }
    else PGS_CUDA(h, pgs::launch_general(wl, grid < 32u ? grid : 32u, stream));
    h->counters.kernel_launches += 2;
    return PGS_OK;
}

struct AuxPlan {
    pgs_handle* h;
    size_t used = 0;
    bool overflow = false;
    // (host destination, offset, bytes) of every output to copy back
    struct Out { void* dst; size_t off, bytes; };
    std::vector<Out> outs;
    size_t out_lo = 0, out_hi = 0;

    size_t reserve(size_t bytes) {
        size_t off = (used + 15) & ~size_t(15);
        if (off + bytes > h->aux_bytes) { overflow = true; return 0; }
        used = off + bytes;
        return off;
    }
    template <class T> const T* in(const T* host, size_t n) {
        if (!host) return nullptr;
        size_t off = reserve(n * sizeof(T));
        if (overflow) return nullptr;
        memcpy(h->aux_host + off, host, n * sizeof(T));
        return (const T*)(h->aux_dev + off);
    }
    template <class T> T* out(T* host, size_t n) {
        if (!host) return nullptr;
        size_t off = reserve(n * sizeof(T));
        if (overflow) return nullptr;
        outs.push_back({host, off, n * sizeof(T)});
        return (T*)(h->aux_dev + off);
    }
};

int validate(pgs_handle* h, const pgs_batch_desc* d) {
    if (!d) return fail(h, PGS_ERR_INVALID, "desc is NULL");
    if (d->struct_size != sizeof(pgs_batch_desc))
        return fail(h, PGS_ERR_INVALID, "desc.struct_size %u != %zu (ABI mismatch)", d->struct_size,
                    sizeof(pgs_batch_desc));
    if (d->rows == 0) return PGS_OK;
    if (d->rows > h->max_rows || d->vocab > h->max_vocab)
        return fail(h, PGS_ERR_LIMIT, "batch %u x %u exceeds the handle's %u x %u", d->rows, d->vocab,
                    h->max_rows, h->max_vocab);
    if (d->vocab == 0 || !d->logits || !d->token || !d->status)
        return fail(h, PGS_ERR_INVALID, "vocab, logits, token and status are required");
    if (d->row_stride < d->vocab) return fail(h, PGS_ERR_INVALID, "row_stride < vocab");
    if (d->logits_dtype > PGS_BF16 || d->logits_mem > PGS_MEM_HOST || d->aux_mem > PGS_MEM_HOST)
        return fail(h, PGS_ERR_INVALID, "bad dtype / memory kind");
    if (d->hist_ids && !d->hist_offsets)
        return fail(h, PGS_ERR_INVALID, "hist_ids given without hist_offsets");
    // Offsets without ids: only host arrays can be checked for "every row is empty"; device offsets
    // cannot be read here, so there the pair must come together.
    if (d->hist_offsets && !d->hist_ids && (d->aux_mem != PGS_MEM_HOST || d->hist_offsets[d->rows] != 0))
        return fail(h, PGS_ERR_INVALID, "hist_offsets given without hist_ids");
    if ((d->dump_ids || d->dump_probs) && d->dump_cap == 0)
        return fail(h, PGS_ERR_INVALID, "dump arrays given with dump_cap == 0");
    return PGS_OK;
}

int run_batch(pgs_handle* h, const pgs_batch_desc* d, cudaStream_t stream, bool wait) {
    int rc = validate(h, d);
    if (rc != PGS_OK) return rc;
    if (d->rows == 0) return PGS_OK;
    DeviceGuard g(h->device);
    const uint32_t rows = d->rows;
    const size_t esz = d->logits_dtype == PGS_F32 ? 4 : 2;
    pgs::RowArgs a;
    memset(&a, 0, sizeof a);
    a.dtype = d->logits_dtype; a.rows = rows; a.vocab = d->vocab; a.eos = d->eos_token_id;
    a.tables = h->tables_dev;
    a.sx = h->sx; a.sl_id = h->sl_id; a.sl_p = h->sl_p; a.sl_key = h->sl_key;
    a.sh_key = h->sh_key; a.sh_cnt = h->sh_cnt;
    a.vocab_pad = h->vocab_pad; a.sort_pad = h->sort_pad; a.hash_cap = h->hash_cap;
    a.max_history = h->max_history;
    a.dump_cap = d->dump_cap;

    // logits
    if (d->logits_mem == PGS_MEM_HOST) {
        const size_t need = (size_t)rows * d->vocab * esz;
        if (need > h->logits_stage_bytes) {
            if (h->logits_stage) { cudaStreamSynchronize(stream); cudaFree(h->logits_stage); h->logits_stage = nullptr; }
            const size_t full = (size_t)h->max_rows * h->max_vocab * 4;
            PGS_CUDA(h, cudaMalloc(&h->logits_stage, full));
            h->logits_stage_bytes = full;
        }
        PGS_CUDA(h, cudaMemcpy2DAsync(h->logits_stage, (size_t)d->vocab * esz, d->logits,
                                      (size_t)d->row_stride * esz, (size_t)d->vocab * esz, rows,
                                      cudaMemcpyHostToDevice, stream));
        a.logits = h->logits_stage;
        a.row_stride = d->vocab;
    } else {
        a.logits = d->logits;
        a.row_stride = d->row_stride;
    }

    AuxPlan plan{h};
    uint64_t hist_total = 0, masked_rows = 0;
    if (d->aux_mem == PGS_MEM_HOST) {
        if (d->hist_offsets) {
            hist_total = d->hist_offsets[rows];
            for (uint32_t r = 0; r < rows; r++) {
                if (d->hist_offsets[r + 1] < d->hist_offsets[r])
                    return fail(h, PGS_ERR_INVALID, "hist_offsets must be non-decreasing");
                if (d->hist_offsets[r + 1] - d->hist_offsets[r] > h->max_history)
                    return fail(h, PGS_ERR_LIMIT, "row %u has %u history ids; the handle allows %u", r,
                                d->hist_offsets[r + 1] - d->hist_offsets[r], h->max_history);
            }
        }
        if (d->mask_table)
            for (uint32_t r = 0; r < rows; r++) masked_rows += d->mask_table[r] >= 0;
        a.temperature = plan.in(d->temperature, rows);
        a.top_k = plan.in(d->top_k, rows);
        a.top_p = plan.in(d->top_p, rows);
        a.freq = plan.in(d->frequency_penalty, rows);
        a.pres = plan.in(d->presence_penalty, rows);
        a.rep = plan.in(d->repetition_penalty, rows);
        a.hist_offsets = plan.in(d->hist_offsets, (size_t)rows + 1);
        a.hist_ids = hist_total ? plan.in(d->hist_ids, hist_total) : nullptr;
        a.mask_table = plan.in(d->mask_table, rows);
        a.mask_state = plan.in(d->mask_state, rows);
        a.uniform = plan.in(d->uniform, rows);
        const size_t in_bytes = plan.used;
        plan.out_lo = (plan.used + 15) & ~size_t(15);
        a.token = plan.out(d->token, rows);
        a.status = plan.out(d->status, rows);
        a.drew = plan.out(d->drew, rows);
        a.argmax = plan.out(d->argmax, rows);
        a.row_max = plan.out(d->row_max, rows);
        a.sumexp = plan.out(d->sumexp, rows);
        a.total = plan.out(d->total, rows);
        a.n_kept = plan.out(d->n_kept, rows);
        plan.out_hi = plan.used;
        if (plan.overflow)
            return fail(h, PGS_ERR_LIMIT, "per-row arrays exceed the staging buffer sized at creation");
        // the candidate dump can be large; it gets its own device buffer per call
        uint32_t* dump_ids_dev = nullptr;
        float* dump_probs_dev = nullptr;
        const size_t dump_n = (size_t)rows * d->dump_cap;
        if (d->dump_ids) PGS_CUDA(h, cudaMalloc(&dump_ids_dev, dump_n * 4));
        if (d->dump_probs) PGS_CUDA(h, cudaMalloc(&dump_probs_dev, dump_n * 4));
        a.dump_ids = dump_ids_dev; a.dump_probs = dump_probs_dev;
        PGS_CUDA(h, cudaMemcpyAsync(h->aux_dev, h->aux_host, in_bytes, cudaMemcpyHostToDevice, stream));
        rc = launch_step(h, a, stream);
        if (rc != PGS_OK) { cudaFree(dump_ids_dev); cudaFree(dump_probs_dev); return rc; }
        PGS_CUDA(h, cudaMemcpyAsync(h->aux_host + plan.out_lo, h->aux_dev + plan.out_lo,
                                    plan.out_hi - plan.out_lo, cudaMemcpyDeviceToHost, stream));
        if (dump_ids_dev) PGS_CUDA(h, cudaMemcpyAsync(d->dump_ids, dump_ids_dev, dump_n * 4, cudaMemcpyDeviceToHost, stream));
        if (dump_probs_dev) PGS_CUDA(h, cudaMemcpyAsync(d->dump_probs, dump_probs_dev, dump_n * 4, cudaMemcpyDeviceToHost, stream));
        cudaError_t e = cudaStreamSynchronize(stream);
        cudaFree(dump_ids_dev); cudaFree(dump_probs_dev);
        if (e != cudaSuccess) return fail(h, PGS_ERR_CUDA, "kernel or copy failed: %s", cudaGetErrorString(e));
        for (const auto& o : plan.outs) memcpy(o.dst, h->aux_host + o.off, o.bytes);
    } else {
        a.temperature = d->temperature; a.top_k = d->top_k; a.top_p = d->top_p;
        a.freq = d->frequency_penalty; a.pres = d->presence_penalty; a.rep = d->repetition_penalty;
        a.hist_offsets = d->hist_offsets; a.hist_ids = d->hist_ids;
        a.mask_table = d->mask_table; a.mask_state = d->mask_state; a.uniform = d->uniform;
        a.token = d->token; a.status = d->status; a.drew = d->drew; a.argmax = d->argmax;
        a.row_max = d->row_max; a.sumexp = d->sumexp; a.total = d->total; a.n_kept = d->n_kept;
        a.dump_ids = d->dump_ids; a.dump_probs = d->dump_probs;
        rc = launch_step(h, a, stream);
        if (rc != PGS_OK) return rc;
        if (wait) {
            cudaError_t e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess) return fail(h, PGS_ERR_CUDA, "kernel failed: %s", cudaGetErrorString(e));
        }
    }
    h->counters.calls += 1;
    h->counters.rows += rows;
    h->counters.bytes += (uint64_t)rows * (d->vocab * esz + 64) + hist_total * 4 + masked_rows * (d->vocab / 8);
    return PGS_OK;
}

}  // namespace

// Phase timers of the row kernel (clock ticks, [ctas x 16]); only with PGS_PROFILE=1.
extern "C" PGS_API int pgs_debug_read_profile(pgs_handle* h, long long* out, uint32_t n_ctas) {
    if (!h || !h->prof || n_ctas > 1024) return PGS_ERR_INVALID;
    DeviceGuard g(h->device);
    PGS_CUDA(h, cudaStreamSynchronize(h->stream));
    PGS_CUDA(h, cudaMemcpy(out, h->prof, (size_t)n_ctas * 16 * sizeof(long long), cudaMemcpyDeviceToHost));
    PGS_CUDA(h, cudaMemset(h->prof, 0, 1024 * 16 * sizeof(long long)));
    return PGS_OK;
}

extern "C" int pgs_set_exact(pgs_handle* h, int on) {
    if (!h) return PGS_ERR_INVALID;
    h->exact = on ? 1 : 0;
    return PGS_OK;
}

extern "C" int pgs_sample_batch(pgs_handle* h, const pgs_batch_desc* desc) {
    if (!h) return PGS_ERR_INVALID;
    return run_batch(h, desc, h->stream, true);
}

extern "C" int pgs_sample_batch_async(pgs_handle* h, const pgs_batch_desc* desc, void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    if (desc && (desc->logits_mem != PGS_MEM_DEVICE || desc->aux_mem != PGS_MEM_DEVICE))
        return fail(h, PGS_ERR_INVALID, "pgs_sample_batch_async needs every array in device memory");
    return run_batch(h, desc, cuda_stream ? (cudaStream_t)cuda_stream : h->stream, false);
}

// ------------------------------------------------------------------- vocabulary-sharded mode

extern "C" size_t pgs_tp_record_bytes(uint32_t cand) { return 16 + (size_t)cand * 8; }

static int tp_args(pgs_handle* h, const pgs_tp_desc* d, pgs::TpArgs* a) {
    if (!d || d->struct_size != sizeof(pgs_tp_desc)) return fail(h, PGS_ERR_INVALID, "bad pgs_tp_desc");
    if (d->n_shards == 0 || d->n_shards > 8 || d->shard_rank >= d->n_shards || d->vocab % d->n_shards)
        return fail(h, PGS_ERR_INVALID, "need 1 <= n_shards <= 8, rank < n_shards, vocab divisible by n_shards");
    if (d->cand == 0 || d->cand > 128) return fail(h, PGS_ERR_INVALID, "cand must be in 1..128");
    if (d->rows == 0 || d->rows > h->max_rows) return fail(h, PGS_ERR_LIMIT, "%u rows exceed the handle's %u", d->rows, h->max_rows);
    a->shard_vocab = d->vocab / d->n_shards;
    if (a->shard_vocab > h->max_vocab) return fail(h, PGS_ERR_LIMIT, "shard width %u exceeds the handle's vocab %u", a->shard_vocab, h->max_vocab);
    if (d->row_stride < a->shard_vocab) return fail(h, PGS_ERR_INVALID, "row_stride < shard width");
    a->logits = d->logits; a->row_stride = d->row_stride; a->rows = d->rows; a->vocab = d->vocab;
    a->shard_lo = d->shard_rank * a->shard_vocab; a->n_shards = d->n_shards; a->cand = d->cand;
    a->temperature = d->temperature; a->top_p = d->top_p; a->uniform = d->uniform; a->top_k = d->top_k;
    a->wait_polls = h->wait_polls; a->timeouts = h->tp_timeouts;
    a->rec_bytes = (uint32_t)pgs_tp_record_bytes(d->cand);
    memset(a->peer_records, 0, sizeof a->peer_records);
    memset(a->peer_flags, 0, sizeof a->peer_flags);
    a->flags = nullptr; a->done = nullptr; a->epoch = 0; a->shard_rank = d->shard_rank;
    return PGS_OK;
}

// The emitting half is the batch step itself over this rank's columns, with records in place of tokens: the same
// kernels, checks, penalties, mask and EOS fix; history ids and eos_token_id are global ids.
static int tp_emit(pgs_handle* h, const pgs_tp_desc* d, const pgs::TpArgs& t, unsigned char* records, cudaStream_t stream) {
    if ((d->hist_offsets == nullptr) != (d->hist_ids == nullptr))
        return fail(h, PGS_ERR_INVALID, "hist_offsets and hist_ids must be given together");
    if (((uintptr_t)records & 15u) != 0) return fail(h, PGS_ERR_INVALID, "the record buffer must be 16-byte aligned");
    pgs::RowArgs a;
    memset(&a, 0, sizeof a);
    a.logits = d->logits; a.dtype = 0; a.rows = d->rows; a.vocab = t.shard_vocab; a.row_stride = d->row_stride;
    a.temperature = d->temperature;
    a.freq = d->frequency_penalty; a.pres = d->presence_penalty; a.rep = d->repetition_penalty;
    a.hist_offsets = d->hist_offsets; a.hist_ids = d->hist_ids;
    a.mask_table = d->mask_table; a.mask_state = d->mask_state; a.tables = h->tables_dev;
    const int64_t eos_local = (int64_t)d->eos_token_id - (int64_t)t.shard_lo;
    a.eos = (d->eos_token_id >= 0 && eos_local >= 0 && eos_local < (int64_t)t.shard_vocab) ? (int32_t)eos_local : -1;
    a.sx = h->sx; a.sl_id = h->sl_id; a.sl_p = h->sl_p; a.sl_key = h->sl_key;
    a.sh_key = h->sh_key; a.sh_cnt = h->sh_cnt;
    a.vocab_pad = h->vocab_pad; a.sort_pad = h->sort_pad; a.hash_cap = h->hash_cap;
    a.max_history = h->max_history;
    a.tp_records = records; a.tp_rec_bytes = t.rec_bytes; a.tp_cand = t.cand; a.id_base = t.shard_lo;
    return launch_step(h, a, stream);
}

extern "C" int pgs_tp_partial(pgs_handle* h, const pgs_tp_desc* d, void* records_out, void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    pgs::TpArgs a;
    int rc = tp_args(h, d, &a);
    if (rc != PGS_OK) return rc;
    if (!d->logits || !records_out) return fail(h, PGS_ERR_INVALID, "logits and records_out are required");
    DeviceGuard g(h->device);
    return tp_emit(h, d, a, (unsigned char*)records_out, cuda_stream ? (cudaStream_t)cuda_stream : h->stream);
}

extern "C" int pgs_tp_merge(pgs_handle* h, const pgs_tp_desc* d, const void* records_all, const pgs_tp_out* out,
                            void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    pgs::TpArgs a;
    int rc = tp_args(h, d, &a);
    if (rc != PGS_OK) return rc;
    if (!records_all || !out || !out->token || !out->status)
        return fail(h, PGS_ERR_INVALID, "records_all, out->token and out->status are required");
    DeviceGuard g(h->device);
    a.records = (unsigned char*)records_all;
    pgs::TpOut o{out->token, out->status, out->drew, out->argmax, out->gmax, out->gsum, out->total, out->n_kept};
    PGS_CUDA(h, pgs::launch_tp_merge(a, o, (uint32_t)h->sm_count, cuda_stream ? (cudaStream_t)cuda_stream : h->stream));
    h->counters.kernel_launches += 1;
    h->counters.rows += a.rows;
    return PGS_OK;
}

extern "C" int pgs_peer_alloc(pgs_handle* h, size_t bytes, void** dev_ptr, unsigned char ipc_handle_out[64]) {
    if (!h || !dev_ptr || !ipc_handle_out || bytes == 0) return PGS_ERR_INVALID;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the IPC handle is exchanged as 64 bytes");
    DeviceGuard g(h->device);
    void* p = nullptr;
    PGS_CUDA(h, cudaMalloc(&p, bytes));
    cudaError_t e = cudaMemset(p, 0, bytes);
    cudaIpcMemHandle_t ih;
    if (e == cudaSuccess) e = cudaIpcGetMemHandle(&ih, p);
    if (e != cudaSuccess) {
        cudaFree(p);
        return fail(h, PGS_ERR_CUDA, "pgs_peer_alloc: %s", cudaGetErrorString(e));
    }
    memcpy(ipc_handle_out, &ih, sizeof ih);
    *dev_ptr = p;
    return PGS_OK;
}

extern "C" int pgs_peer_open(pgs_handle* h, const unsigned char ipc_handle[64], void** dev_ptr) {
    if (!h || !dev_ptr || !ipc_handle) return PGS_ERR_INVALID;
    DeviceGuard g(h->device);
    cudaIpcMemHandle_t ih;
    memcpy(&ih, ipc_handle, sizeof ih);
    void* p = nullptr;
    PGS_CUDA(h, cudaIpcOpenMemHandle(&p, ih, cudaIpcMemLazyEnablePeerAccess));
    // prove that this device reaches the mapping before any kernel is pointed at it
    uint32_t probe = 0;
    const cudaError_t e = cudaMemcpy(&probe, p, sizeof probe, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        cudaIpcCloseMemHandle(p);
        return fail(h, PGS_ERR_CUDA, "pgs_peer_open: the mapped buffer is not readable from device %d: %s", h->device,
                    cudaGetErrorString(e));
    }
    *dev_ptr = p;
    return PGS_OK;
}

extern "C" int pgs_peer_close(pgs_handle* h, void* dev_ptr) {
    if (!h || !dev_ptr) return PGS_ERR_INVALID;
    DeviceGuard g(h->device);
    PGS_CUDA(h, cudaIpcCloseMemHandle(dev_ptr));
    return PGS_OK;
}

extern "C" int pgs_peer_free(pgs_handle* h, void* dev_ptr) {
    if (!h || !dev_ptr) return PGS_ERR_INVALID;
    DeviceGuard g(h->device);
    PGS_CUDA(h, cudaFree(dev_ptr));
    return PGS_OK;
}

extern "C" int pgs_tp_partial_push(pgs_handle* h, const pgs_tp_desc* d, void* const* peer_records,
                                   uint32_t* const* peer_flags, uint32_t epoch, void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    pgs::TpArgs a;
    int rc = tp_args(h, d, &a);
    if (rc != PGS_OK) return rc;
    if (!d->logits || !peer_records || !peer_flags) return fail(h, PGS_ERR_INVALID, "logits, peer_records and peer_flags are required");
    for (uint32_t p = 0; p < d->n_shards; p++) {
        if (!peer_records[p] || !peer_flags[p]) return fail(h, PGS_ERR_INVALID, "peer %u: NULL gather buffer or flag array", p);
        // this shard's block inside rank p's [n_shards][rows][record] buffer
        a.peer_records[p] = (unsigned char*)peer_records[p] + (size_t)d->shard_rank * a.rows * a.rec_bytes;
        a.peer_flags[p] = peer_flags[p];
    }
    DeviceGuard g(h->device);
    // every buffer must be device memory this GPU can reach: its own, or a peer's with peer access enabled
    // (enabled here when it is not yet; an IPC mapping alone does not do that for this device)
    for (uint32_t p = 0; p < d->n_shards; p++) {
        const void* ptrs[2] = {peer_records[p], peer_flags[p]};
        for (const void* ptr : ptrs) {
            cudaPointerAttributes at;
            PGS_CUDA(h, cudaPointerGetAttributes(&at, ptr));
            if (at.type != cudaMemoryTypeDevice) return fail(h, PGS_ERR_INVALID, "peer %u: not device memory", p);
            if (at.device == h->device) continue;
            int can = 0;
            PGS_CUDA(h, cudaDeviceCanAccessPeer(&can, h->device, at.device));
            if (!can) return fail(h, PGS_ERR_INVALID, "device %d cannot access memory of device %d", h->device, at.device);
            const cudaError_t e = cudaDeviceEnablePeerAccess(at.device, 0);
            if (e == cudaErrorPeerAccessAlreadyEnabled) cudaGetLastError();
            else if (e != cudaSuccess) return fail(h, PGS_ERR_CUDA, "cudaDeviceEnablePeerAccess(%d): %s", at.device, cudaGetErrorString(e));
        }
    }
    a.records = a.peer_records[d->shard_rank];   // built in this rank's own buffer, then copied out
    a.done = h->tp_done;                         // zero between launches
    a.epoch = epoch;
    cudaStream_t stream = cuda_stream ? (cudaStream_t)cuda_stream : h->stream;
    rc = tp_emit(h, d, a, a.records, stream);
    if (rc != PGS_OK) return rc;
    PGS_CUDA(h, pgs::launch_tp_push(a, stream));
    h->counters.kernel_launches += 1;
    return PGS_OK;
}

extern "C" int pgs_tp_merge_wait(pgs_handle* h, const pgs_tp_desc* d, const void* records_all, const uint32_t* flags,
                                 uint32_t epoch, const pgs_tp_out* out, void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    pgs::TpArgs a;
    int rc = tp_args(h, d, &a);
    if (rc != PGS_OK) return rc;
    if (!records_all || !flags || !out || !out->token || !out->status)
        return fail(h, PGS_ERR_INVALID, "records_all, flags, out->token and out->status are required");
    DeviceGuard g(h->device);
    a.records = (unsigned char*)records_all;
    a.flags = (uint32_t*)flags;
    a.epoch = epoch;
    pgs::TpOut o{out->token, out->status, out->drew, out->argmax, out->gmax, out->gsum, out->total, out->n_kept};
    h->tp_stream = cuda_stream ? (cudaStream_t)cuda_stream : h->stream;
    PGS_CUDA(h, pgs::launch_tp_merge(a, o, (uint32_t)h->sm_count, h->tp_stream));
    h->counters.kernel_launches += 1;
    h->counters.rows += a.rows;
    return PGS_OK;
}

extern "C" int pgs_set_wait_limit(pgs_handle* h, uint32_t polls) {
    if (!h) return PGS_ERR_INVALID;
    if (polls == 0) return fail(h, PGS_ERR_INVALID, "pgs_set_wait_limit: at least one poll");
    h->wait_polls = polls;
    return PGS_OK;
}

extern "C" int pgs_tp_exchange_status(pgs_handle* h) {
    if (!h) return PGS_ERR_INVALID;
    DeviceGuard g(h->device);
    unsigned long long n = 0;
    cudaError_t e = cudaStreamSynchronize(h->tp_stream ? h->tp_stream : h->stream);
    if (e == cudaSuccess) e = cudaMemcpy(&n, h->tp_timeouts, sizeof n, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(h, PGS_ERR_CUDA, "pgs_tp_exchange_status: %s", cudaGetErrorString(e));
    const unsigned long long fresh = n - h->timeouts_seen;
    h->timeouts_seen = n;
    if (fresh) return fail(h, PGS_ERR_TIMEOUT, "%llu rows gave up waiting for a shard's records or for the other CTAs of the wide kernel", fresh);
    return PGS_OK;
}

extern "C" int pgs_draft_accept(pgs_handle* h, const uint32_t* row_argmax, const uint32_t* draft, uint32_t sequences,
                                uint32_t positions, uint32_t* accepted, uint32_t* next, void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    if (!row_argmax || !draft || !accepted || !next || positions == 0)
        return fail(h, PGS_ERR_INVALID, "pgs_draft_accept: NULL argument or zero positions");
    if (sequences == 0) return PGS_OK;
    DeviceGuard g(h->device);
    PGS_CUDA(h, pgs::launch_draft_accept(row_argmax, draft, sequences, positions, accepted, next,
                                         cuda_stream ? (cudaStream_t)cuda_stream : h->stream));
    h->counters.kernel_launches += 1;
    return PGS_OK;
}

// ------------------------------------------------------------------------------ scoring

extern "C" int pgs_log_softmax(pgs_handle* h, const float* logits, uint32_t rows, uint32_t vocab, uint64_t row_stride,
                               const uint32_t* ids, float* out_gather, float* out_full, int32_t* status,
                               void* cuda_stream) {
    if (!h) return PGS_ERR_INVALID;
    if (!logits || vocab == 0 || row_stride < vocab || (!out_full && !(ids && out_gather)))
        return fail(h, PGS_ERR_INVALID, "pgs_log_softmax: need logits, row_stride >= vocab and an output");
    if (rows == 0) return PGS_OK;
    DeviceGuard g(h->device);
    cudaStream_t stream = cuda_stream ? (cudaStream_t)cuda_stream : h->stream;
    unsigned long long id = 0;
    const ScoreRoute route = vocab <= h->wide_vocab ? score_route(h, rows, vocab, out_full != nullptr) : SCORE_PLAIN;
    if (route != SCORE_PLAIN && score_workspace_free(h, stream, &id)) {
        pgs::RowArgs a;
        memset(&a, 0, sizeof a);
        a.logits = logits; a.rows = rows; a.vocab = vocab; a.row_stride = row_stride; a.status = status; a.eos = -1;
        pgs::WideLaunch l = h->score_wide;
        l.ids = ids; l.out_gather = out_gather; l.out_full = out_full;
        l.done = h->score_done; l.done_value = h->score_calls + 1u;
        l.local = route == SCORE_ROWS;
        PGS_CUDA(h, pgs::launch_wide(a, l, h->slots, l.local ? (rows < (uint32_t)h->sm_count ? rows : (uint32_t)h->sm_count) : wide_grid(h, rows, vocab), stream));
        h->score_calls += 1u;
        h->score_stream = id;
    } else {   // one CTA per row, no workspace
        pgs::ScoreArgs a{logits, row_stride, rows, vocab, ids, out_gather, out_full, status};
        const uint32_t grid = rows < (uint32_t)h->sm_count ? rows : (uint32_t)h->sm_count;
        PGS_CUDA(h, pgs::launch_log_softmax(a, grid, stream));
    }
    h->counters.kernel_launches += 1;
    return PGS_OK;
}
