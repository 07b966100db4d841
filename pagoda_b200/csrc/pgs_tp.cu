// Vocabulary-sharded (tensor-parallel) sampling.  The reference has no multi-GPU code; this mode is
// an extension whose semantics are fixed by the CPU oracle (pgo_tp_sample_row):
//
//   every GPU holds columns [rank * V/n, (rank + 1) * V/n) of every row and emits, per row, one
//   fixed-size record: its max m_r, its own sequential f32 sum s_r = sum exp((x - m_r) / t) (same
//   arithmetic as pagoda/src/sampler.rs:92-114 on the shard), its argmax and its `cand` largest
//   logits by (value descending, id ascending) with their global ids;
//   the records of all shards are gathered on every GPU -- by an NCCL all-gather between the two kernels,
//   or by the emitting kernel itself, which stores its records into every peer's gather buffer over
//   NVLink and then raises a per-shard flag there that the peer's merge kernel waits for (bounded) --
//   and merged on every GPU:
//   M = max m_r, S = sum_r s_r * exp((m_r - M) / t) folded in shard order, candidate probability
//   exp((x - M) / t) / S, then the reference's top-p rule, total and inverse-CDF walk over the
//   union of the candidates; greedy rows take the best candidate, lowest id on ties, which is the
//   global argmax.
//
// Draft verification (pagoda-hf/src/qwen3_5.rs:663-755 returns per-position argmax ids; the accept
// rule itself is defined here): accept while argmax(row j) == draft[j].
#include "pgs_finish.cuh"
#include "pgs_tp.cuh"

namespace pgs {


// system-scope flag accesses: the store publishes everything this GPU wrote before it (records in peer
// memory included), the load makes it visible to the reader
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Peer-store exchange: copies this rank's finished records ([rows x rec_bytes], complete when the kernels in
// front of this one in the stream have ended) into slot [shard_rank] of every other rank's gather buffer with
// plain stores into peer memory; the last CTA then raises this shard's flag on every rank.
__global__ void __launch_bounds__(256) tp_push_kernel(const TpArgs a) {
    cudaGridDependencySynchronize();
    const size_t bytes = (size_t)a.rows * a.rec_bytes;
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
    if ((a.rec_bytes & 15u) == 0u) {   // every buffer starts on a 256-byte boundary
        const uint4* src = reinterpret_cast<const uint4*>(a.records);
        for (size_t i = i0; i < bytes / 16; i += step) {
            const uint4 v = src[i];
            for (uint32_t p = 0; p < a.n_shards; p++)
                if (p != a.shard_rank) reinterpret_cast<uint4*>(a.peer_records[p])[i] = v;
        }
    } else {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(a.records);
        for (size_t i = i0; i < bytes / 4; i += step) {
            const uint32_t v = src[i];
            for (uint32_t p = 0; p < a.n_shards; p++)
                if (p != a.shard_rank) reinterpret_cast<uint32_t*>(a.peer_records[p])[i] = v;
        }
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(a.done, 1u) == gridDim.x - 1u) {
        *a.done = 0u;
        __threadfence_system();
        for (uint32_t p = 0; p < a.n_shards; p++) st_release_sys(a.peer_flags[p] + a.shard_rank, a.epoch);
    }
}

// Most of a row's time is one warp's: few threads per row, so that an SM holds eight rows (of 256 threads it holds four, and
// 1024 rows of 8 x 64 candidates need a second wave).  Where all rows are resident either way, long lists take 256
// threads: 256 rows of 8 x 128 candidates 35 us, with 128 threads 54; of 8 x 64 19 and 27.
constexpr int TP_FEW = 128, TP_MANY = 256;
constexpr int TP_MCAP = TP_MAX_SHARDS * 128;   // candidates of all shards together (cand <= 128)

template <int CAP>
struct TpMergeSmem {
    FinishArraysT<CAP> fin;
    unsigned long long exp_tab[32];
    uint32_t cid[CAP];
    float cx[CAP];
    float M, S;
    uint32_t amax, n;
    int fault;   // the row's status when it is not ROW_OK
    uint32_t start[TP_MAX_SHARDS + 1];   // where each shard's candidates begin in cid / cx
    TpRecHead hd[TP_MAX_SHARDS];
    int unsorted;
};


// T: threads; CAP: candidates of all shards together, at most
template <int T, int CAP>
__global__ void __launch_bounds__(T, 1024 / T) tp_merge_kernel(const TpArgs a, const TpOut o) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TpMergeSmem<CAP>& sm = *reinterpret_cast<TpMergeSmem<CAP>*>(smem_raw);
    const int tid = threadIdx.x;
    const uint32_t row = blockIdx.x;
    cudaGridDependencySynchronize();
    const float temp = a.temperature ? a.temperature[row] : 0.0f;
    const float t = fmaxf(temp, 1e-9f);
    if (tid < 32) sm.exp_tab[tid] = kExp2TableDev[tid];
    if (a.flags) {   // peer-store exchange: wait (bounded, about a second) until every shard has raised its flag
        if (tid == 0) {
            int late = 0;
            for (uint32_t r = 0; r < a.n_shards && !late; r++) {
                uint32_t spin = 0;
                while ((int32_t)(ld_acquire_sys(a.flags + r) - a.epoch) < 0) {
                    if (++spin > a.wait_polls) { late = 1; break; }
                    __nanosleep(500);
                }
            }
            sm.fault = late;
        }
        __syncthreads();
        if (sm.fault) {
            if (tid == 0) {
                o.token[row] = 0; o.status[row] = ROW_LOAD_TIMEOUT; if (o.drew) o.drew[row] = 0;
                if (a.timeouts) atomicAdd(a.timeouts, 1ull);
            }
            return;
        }
    }
    __syncthreads();
    auto rec = [&](uint32_t r) {
        return reinterpret_cast<const TpRecHead*>(a.records + ((size_t)r * a.rows + row) * a.rec_bytes);
    };
    const uint32_t top_k = a.top_k ? a.top_k[row] : 0u;
    // every record slot of the row is requested at once (one trip to memory): the heads by the first threads, the
    // candidate slots one or two per thread; which of the slots are filled is known once the heads are in
    if ((uint32_t)tid < a.n_shards) sm.hd[tid] = *rec(tid);
    constexpr int SLOTS = (CAP + T - 1) / T;
    float gx[SLOTS];
    uint32_t gid[SLOTS];
#pragma unroll
    for (int u = 0; u < SLOTS; u++) {
        const uint32_t c = (uint32_t)tid + u * T;
        gx[u] = 0.0f; gid[u] = 0u;
        if (c < a.n_shards * a.cand) {
            const float* rx = reinterpret_cast<const float*>(rec(c / a.cand) + 1);
            gx[u] = rx[c % a.cand];
            gid[u] = reinterpret_cast<const uint32_t*>(rx + a.cand)[c % a.cand];
        }
    }
    __syncthreads();
    if (tid < 32) {   // one shard per lane
        static_assert(TP_MAX_SHARDS <= 32, "one lane per shard");
        const bool is = (uint32_t)tid < a.n_shards;
        const float mr = is ? sm.hd[tid].m : -INFINITY;
        const uint32_t ns = is ? sm.hd[tid].n_status : 0u, st = ns >> 24;
        int fault = (top_k > a.cand) ? ROW_BAD_PARAM : ROW_OK;   // a record holds the shard's `cand` largest, no more
        if (__any_sync(FULL, is && st == (uint32_t)ROW_BAD_PARAM)) fault = ROW_BAD_PARAM;
        const bool nonfinite = __any_sync(FULL, is && (st == (uint32_t)ROW_NONFINITE || mr != mr));
        const bool dead = __any_sync(FULL, is && st == (uint32_t)ROW_DEAD);
        // the order of engine.rs:1292-1303: parameters, then sanity, then the grammar's dead state
        if (fault == ROW_OK) fault = nonfinite ? ROW_NONFINITE : dead ? ROW_DEAD : ROW_OK;
        float M = mr == mr ? mr : -INFINITY;
#pragma unroll
        for (int o = 16; o; o >>= 1) M = fmaxf(M, __shfl_xor_sync(FULL, M, o));
        const bool counts = is && fault == ROW_OK && finite_f(mr);
        const float term = counts ? fmul(sm.hd[tid].s, pgs_expf_tab(fdiv(fsub(mr, M), t), sm.exp_tab)) : 0.0f;
        // shards are in id order: the first that holds the maximum has the lowest id
        const unsigned top = __ballot_sync(FULL, counts && mr == M);
        const uint32_t mine = min(ns & 0xffffffu, a.cand);   // a record can never hold more than `cand` entries
        float S = 0.0f;
        uint32_t before = 0u, n = 0u;
        for (uint32_t r = 0; r < a.n_shards; r++) {
            S = fadd(S, __shfl_sync(FULL, term, (int)r));
            const uint32_t nr = __shfl_sync(FULL, mine, (int)r);
            if (r < (uint32_t)tid) before += nr;
            n += nr;
        }
        if ((uint32_t)tid <= a.n_shards) sm.start[tid] = before;   // (lane n_shards: all of them)
        if (tid == 0) {
            sm.M = M; sm.S = S; sm.amax = top ? sm.hd[__ffs((int)top) - 1].argmax : 0u; sm.n = n; sm.fault = fault;
            sm.unsorted = 0; sm.fin.n_live = 0u;
        }
    }
    __syncthreads();
    if (sm.fault) {
        if (tid == 0) { o.token[row] = 0; o.status[row] = sm.fault; if (o.drew) o.drew[row] = 0; }
        return;
    }
    // the union of the candidates, shard after shard
#pragma unroll
    for (int u = 0; u < SLOTS; u++) {
        const uint32_t c = (uint32_t)tid + u * T;
        if (c < a.n_shards * a.cand) {
            const uint32_t r = c / a.cand, j = c % a.cand;
            if (j < sm.start[r + 1] - sm.start[r]) { sm.cx[sm.start[r] + j] = gx[u]; sm.cid[sm.start[r] + j] = gid[u]; }
        }
    }
    __syncthreads();
    const bool any = finite_f(sm.M);
    if (o.gmax && tid == 0) o.gmax[row] = sm.M;
    if (temp < 1e-5f || !any) {
        if (tid == 0) {
            o.token[row] = sm.amax; o.status[row] = any ? ROW_OK : ROW_EMPTY;
            if (o.drew) o.drew[row] = 0;
            if (o.argmax) o.argmax[row] = sm.amax;
            if (o.gsum) o.gsum[row] = sm.S;
            if (o.total) o.total[row] = 0.0f;
            if (o.n_kept) o.n_kept[row] = 0;
        }
        return;
    }
    RowArgs ra;
    memset(&ra, 0, sizeof ra);
    ra.token = o.token; ra.status = o.status; ra.drew = o.drew; ra.argmax = o.argmax; ra.sumexp = o.gsum;
    ra.total = o.total; ra.n_kept = o.n_kept;
    ra.row_max = nullptr;
    const float top_p = a.top_p ? a.top_p[row] : 1.0f, u01 = a.uniform ? a.uniform[row] : 0.0f;
    // Every shard's candidates arrive sorted by (logit descending, id ascending), and shards follow one another in id
    // order.  So a candidate's rank among all of them is a sum of binary searches, one per shard, and its place in id
    // order needs a count inside its own shard only: no sort.  The searches are by (probability, id); two different
    // logits can round to one probability, which may leave a shard's list out of that order: such a row (looked for
    // below) takes the general ranking instead.
    const uint32_t n = sm.n;
    const bool norm = sm.S > 1e-9f;
    for (uint32_t c = tid; c < n; c += T) {
        const float e = softmax_num(sm.cx[c], sm.M, t, sm.exp_tab);   // exact expf
        sm.fin.key[c] = ((unsigned long long)f2u(norm ? fdiv(e, sm.S) : e) << 32) | (unsigned long long)(0xffffffffu - sm.cid[c]);
    }
    __syncthreads();
    for (uint32_t c = tid; c + 1 < n; c += T) {
        uint32_t r = 0;
        while (sm.start[r + 1] <= c) r++;
        if (c + 1 < sm.start[r + 1] && !(sm.fin.key[c] > sm.fin.key[c + 1])) sm.unsorted = 1;
    }
    __syncthreads();
    if (sm.unsorted) {   // CTA-uniform
        cta_finish<T>(sm.fin, sm.exp_tab, ra, row, a.vocab, sm.cid, sm.cx, n, sm.M, t, sm.S, top_k, top_p, u01, sm.amax, ROW_OK);
        return;
    }
    for (uint32_t c = tid; c < n; c += T) {
        const unsigned long long kc = sm.fin.key[c];
        uint32_t own = 0;
        while (sm.start[own + 1] <= c) own++;
        uint32_t r_p = 0;
        for (uint32_t r = 0; r < a.n_shards; r++) {   // keys of shard r that come before kc: the list is descending
            uint32_t lo = sm.start[r], hi = sm.start[r + 1];
            const uint32_t base = lo;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (sm.fin.key[mid] > kc) lo = mid + 1; else hi = mid;
            }
            r_p += lo - base;
        }
        uint32_t r_id = sm.start[own];
        const uint32_t idc = sm.cid[c];
        for (uint32_t o2 = sm.start[own]; o2 < sm.start[own + 1]; o2++) r_id += sm.cid[o2] < idc;
        const float pc = u2f((uint32_t)(kc >> 32));
        sm.fin.sid[r_id] = idc; sm.fin.sp[r_id] = pc; sm.fin.rp[r_p] = pc; sm.fin.rpos[r_p] = r_id;
    }
    cta_finish_ranked<T>(sm.fin, ra, row, a.vocab, n, sm.M, sm.S, top_k, top_p, u01, sm.amax, ROW_OK);
}

__global__ void draft_accept_kernel(const uint32_t* row_argmax, const uint32_t* draft, uint32_t sequences,
                                    uint32_t positions, uint32_t* accepted, uint32_t* next) {
    cudaGridDependencySynchronize();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= sequences || positions == 0) return;
    uint32_t acc = 0;
    while (acc < positions && row_argmax[s * positions + acc] == draft[s * positions + acc]) acc++;
    accepted[s] = acc;
    next[s] = row_argmax[s * positions + (acc < positions ? acc : positions - 1)];
}

template <int T, int CAP>
static cudaError_t configure_merge() {
    cudaError_t e = cudaFuncSetAttribute(tp_merge_kernel<T, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TpMergeSmem<CAP>));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(tp_merge_kernel<T, CAP>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}
cudaError_t configure_tp() {
    cudaError_t e = configure_merge<TP_FEW, TP_MCAP / 2>();
    if (e == cudaSuccess) e = configure_merge<TP_FEW, TP_MCAP>();
    if (e == cudaSuccess) e = configure_merge<TP_MANY, TP_MCAP / 2>();
    if (e == cudaSuccess) e = configure_merge<TP_MANY, TP_MCAP>();
    return e;
}

// set up while the kernel before still runs (programmatic stream serialization)
template <class... A>
static cudaError_t launch_behind(void (*kernel)(A...), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t launch_tp_push(const TpArgs& a, cudaStream_t stream) {
    const size_t units = ((size_t)a.rows * a.rec_bytes) / 16 + 1;
    return launch_behind(tp_push_kernel, (uint32_t)((units + 255) / 256 < 64 ? (units + 255) / 256 : 64), 256u, 0, stream, a);
}

template <int T>
static cudaError_t launch_merge(const TpArgs& a, const TpOut& o, cudaStream_t stream) {
    // (half the longest list in half the shared memory: eight rows per SM instead of six)
    if (a.n_shards * a.cand <= (uint32_t)TP_MCAP / 2u) return launch_behind(tp_merge_kernel<T, TP_MCAP / 2>, a.rows, T, sizeof(TpMergeSmem<TP_MCAP / 2>), stream, a, o);
    return launch_behind(tp_merge_kernel<T, TP_MCAP>, a.rows, T, sizeof(TpMergeSmem<TP_MCAP>), stream, a, o);
}
cudaError_t launch_tp_merge(const TpArgs& a, const TpOut& o, uint32_t sms, cudaStream_t stream) {
    return a.n_shards * a.cand > 256u && a.rows <= 4u * sms ? launch_merge<TP_MANY>(a, o, stream) : launch_merge<TP_FEW>(a, o, stream);
}

cudaError_t launch_draft_accept(const uint32_t* row_argmax, const uint32_t* draft, uint32_t sequences,
                                uint32_t positions, uint32_t* accepted, uint32_t* next, cudaStream_t stream) {
    return launch_behind(draft_accept_kernel, (sequences + 127) / 128, 128u, 0, stream, row_argmax, draft, sequences, positions, accepted, next);
}

}  // namespace pgs
