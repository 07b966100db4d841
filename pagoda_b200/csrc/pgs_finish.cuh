// The reference's rule applied to a row's candidate list by one CTA of any size: exact probabilities
// exp((x - max) / t) / sum (sampler.rs:92-114), top-k threshold with every tie kept
// (sampler.rs:116-128), top-p walk by probability descending / id ascending (sampler.rs:130-150),
// then the total and the inverse-CDF walk in id order (sampler.rs:40-55).  Used by the streaming row
// kernel for its own rows and by the merge kernel of the vocabulary-sharded path.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>

#include "pgs_args.cuh"
#include "pgs_block.cuh"

namespace pgs {

constexpr int F_MCAP = 2048;       // longest candidate list (a power of two)
constexpr int F_QUAD = 256;        // lists up to this length are ranked by counting, longer ones by sorting

// Working arrays of the finish, in shared memory: each holds CAP entries (CAP a power of two, at least the CTA's threads:
// the longest list the owner hands in).
template <int CAP>
struct alignas(16) FinishArraysT {
    static constexpr int CAPACITY = CAP;
    unsigned long long key[CAP];   // sort keys
    uint32_t sid[CAP];             // ids ascending
    float sp[CAP];                 // probabilities in id order (zeroed when dropped)
    float rp[CAP];                 // probabilities descending (ties: id ascending)
    uint32_t rpos[CAP];            // position in the id-ordered list of the entry at each rank
    float fp[CAP];                 // running sums of the serial folds
    uint32_t n_live;
};
using FinishArrays = FinishArraysT<F_MCAP>;

// Exact left fold of n shared-memory floats, called by one warp: returns the total and leaves every
// running value in pre[0..n).  One lane does the additions: the loads do not depend on the running value, so
// they are requested eight at a time (two 128-bit loads) and the dependent chain is the additions alone
// (warp shuffles would put tens of cycles between two of them).  v and pre: 16-byte aligned arrays whose
// length is a multiple of 8 and at least n (entries past n are read and written, not used).
__device__ __forceinline__ float warp_prefix(const float* v, int n, float* pre) {
    const int lane = threadIdx.x & 31;
    float acc = 0.0f;
    if (lane == 0 && n > 0) {
        float4 lo4 = *reinterpret_cast<const float4*>(v), hi4 = *reinterpret_cast<const float4*>(v + 4);
#pragma unroll 1
        for (int j0 = 0; j0 < n; j0 += 8) {
            float x[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
            if (j0 + 8 < n) {   // the next eight are on their way while these are added
                lo4 = *reinterpret_cast<const float4*>(v + j0 + 8);
                hi4 = *reinterpret_cast<const float4*>(v + j0 + 12);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                acc = fadd(acc, j0 + u < n ? x[u] : 0.0f);
                x[u] = acc;
            }
            *reinterpret_cast<float4*>(pre + j0) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4*>(pre + j0 + 4) = make_float4(x[4], x[5], x[6], x[7]);
        }
    }
    __syncwarp();
    return __shfl_sync(FULL, acc, 0);
}

// First index whose running value satisfies the predicate (mode/target as in seq_scan), or -1; one warp.
__device__ __forceinline__ int warp_find(const float* pre, int n, int mode, float target) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int base = 0; base < n; base += 32) {
        const int j = base + lane;
        const unsigned hit = __ballot_sync(FULL, j < n && seq_pred(mode, pre[j], target));
        if (hit) return base + __ffs(hit) - 1;
    }
    return -1;
}

constexpr int RUN = 16;   // consecutive terms of a lane
// What this lane's run adds to a running value in the binade whose lower end has the bits k, in ulps, from an even (c0) and from
// an odd (c1) value; SEQ_SAT: leaves the binade.
__device__ __forceinline__ void run_increments(const float (&v)[RUN], uint32_t k, uint32_t& c0, uint32_t& c1) {
    float2 s = make_float2(u2f(k), u2f(k + 1u));
#pragma unroll
    for (int j = 0; j < RUN; j++) s = __fadd2_rn(s, make_float2(v[j], v[j]));
    c0 = (f2u(s.x) & 0x7f800000u) == k ? f2u(s.x) - k : SEQ_SAT;
    c1 = (f2u(s.y) & 0x7f800000u) == k ? f2u(s.y) - (k + 1u) : SEQ_SAT;
}
// Of c0 and c1, what the lane's run really adds when the first lane's begins with a value of parity `odd`.  A run without a term
// that ends on half an ulp adds the same either way (tie: ballot of those that do not) and only turns the parity or keeps it;
// behind a run that ends with one parity whatever it begins with, nothing in front of it matters.  (Three ballots and a few bit
// operations: composing the pairs of increments lane by lane, five rounds of shuffles and selections, took 511 cycles.)
__device__ __forceinline__ uint32_t increment_from(uint32_t c0, uint32_t c1, unsigned tie, uint32_t odd) {
    if (tie) {   // warp-uniform
        const unsigned m0 = __ballot_sync(FULL, c0 & 1u), m1 = __ballot_sync(FULL, !(c1 & 1u));   // parity behind an even, an odd one
        const unsigned before = (1u << (threadIdx.x & 31)) - 1u, fixed = ~(m0 ^ m1) & before;
        const uint32_t from = 32u - __clz((int)fixed);   // the runs in front of this lane that matter begin here (0 .. 31)
        const uint32_t p = (fixed ? m0 >> (from - 1u) : odd) + __popc(m0 & ~m1 & before & (0xffffffffu << from));
        if (p & 1u) c0 = c1;
    }
    return min(c0, 0x00800000u);   // (2^23 leaves the binade whatever the value)
}
__device__ __forceinline__ uint32_t warp_scan_u32(uint32_t v) {   // inclusive
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, v, o);
        if (lane >= (uint32_t)o) v += t;
    }
    return v;
}

// Adds runs of terms to the exact running value R, those of the lanes pos .. 31 in this order; one warp, the same result in all
// lanes.  ends: the running value behind every run (optional).  As many runs as keep the running value in its binade at once,
// then the next one term by term, and on from what that has come to: what the lanes add is looked at anew in every binade, so
// nothing rests on an estimate.  (With the increments of estimated binades, a crossing that came a run earlier or later than
// estimated left all runs behind it to be added one by one.)
__device__ __forceinline__ float add_runs(float R, const float (&v)[RUN], float* ends = nullptr, uint32_t pos = 0u) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll 1
    while (pos < 32u) {
        const uint32_t rb = f2u(R), k = rb & 0x7f800000u, room = 0x00800000u - (rb & 0x007fffffu);
        uint32_t n, inc = 0u;
        if (k == 0u) {   // nothing yet: on to the first run with a term
            uint32_t bits = 0u;
#pragma unroll
            for (int j = 0; j < RUN; j++) bits |= f2u(v[j]);
            const unsigned real = __ballot_sync(FULL, bits != 0u) >> pos;
            n = real ? (uint32_t)__ffs((int)real) - 1u : 32u - pos;
        } else {
            uint32_t c0, c1;
            run_increments(v, k, c0, c1);
            if (lane < pos) c0 = c1 = 0u;
            inc = increment_from(c0, c1, __ballot_sync(FULL, c0 != c1), rb);
            if (!ends) {
                const uint32_t all = __reduce_add_sync(FULL, inc);
                if (all < room) return u2f(rb + all);
            }
            inc = warp_scan_u32(inc);
            const unsigned ok = __ballot_sync(FULL, inc < room) >> pos;
            n = ~ok ? min((uint32_t)__ffs((int)~ok) - 1u, 32u - pos) : 32u;
        }
        if (ends && lane >= pos && lane < pos + n) ends[lane] = u2f(rb + inc);
        const uint32_t last = __shfl_sync(FULL, inc, (int)(pos + n - 1u) & 31);
        R = n ? u2f(rb + last) : R;
        pos += n;
        if (pos < 32u) {
#pragma unroll
            for (int j = 0; j < RUN; j++) R = fadd(R, v[j]);   // (every lane its own run)
            R = __shfl_sync(FULL, R, (int)pos);
            if (ends && lane == 0) ends[pos] = R;
            pos++;
        }
    }
    return R;
}

// Exact left fold of n shared-memory floats by one warp, 512 at a time as runs of 16; ends[r]: the running value behind
// run r (exact).  Stops where the running value reaches `goal`, behind the first 512 at the earliest; returns what it has come
// to.  v: readable up to the next multiple of 4.  (512 terms: the additions one by one take 4000 cycles.)
__device__ __forceinline__ float warp_fold(const float* v, uint32_t n, float goal, float* ends) {
    const uint32_t lane = threadIdx.x & 31;
    float R = 0.0f;
#pragma unroll 1
    for (uint32_t base = 0; base < n && (base == 0u || !(R >= goal)); base += 32u * RUN) {   // (a goal of zero is reached by the first term, not in front of it)
        float x[RUN];
#pragma unroll
        for (int j = 0; j < RUN; j += 4) {
            const uint32_t i = base + lane * RUN + j;
            const float4 q = i < n ? *reinterpret_cast<const float4*>(v + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            x[j] = q.x; x[j + 1] = i + 1 < n ? q.y : 0.0f; x[j + 2] = i + 2 < n ? q.z : 0.0f; x[j + 3] = i + 3 < n ? q.w : 0.0f;
        }
        R = add_runs(R, x, ends + base / RUN);
    }
    return R;
}
// First of the n terms behind which the running value satisfies the predicate, given the running values behind the runs; -1:
// none.  One warp.
__device__ __forceinline__ int warp_fold_find(const float* v, uint32_t n, const float* ends, int mode, float target) {
    const int run = warp_find(ends, (int)((n + RUN - 1) / RUN), mode, target);
    if (run < 0) return -1;
    int at = -1;
    float acc = run ? ends[run - 1] : 0.0f;
    for (uint32_t j = run * RUN; j < min(n, (uint32_t)(run + 1) * RUN); j++) {
        acc = fadd(acc, v[j]);
        if (seq_pred(mode, acc, target)) { at = (int)j; break; }
    }
    return at;
}

// How many of the n ranked probabilities the top-p walk keeps (sampler.rs:130-150); one warp.  Short lists: one lane adds,
// and stops where top-p is reached (its loads do not wait for the additions).
constexpr uint32_t F_SERIAL = 160;   // up to here one lane's additions are as fast as the runs, whose code is seldom in the cache
__device__ __forceinline__ uint32_t warp_top_p(const float* p, uint32_t n, float top_p, float* ends) {
    uint32_t keep = n;
    if (top_p >= 1.0f) return keep;
    if (n > F_SERIAL) {
        const float R = warp_fold(p, n, top_p, ends);
        __syncwarp();
        if (R >= top_p) keep = (uint32_t)warp_fold_find(p, n, ends, SEQ_FIND_GE, top_p) + 1u;
        __syncwarp();
        return keep;
    }
    if ((threadIdx.x & 31) == 0) {
        float acc = 0.0f;
#pragma unroll 1
        for (uint32_t j0 = 0; j0 < n; j0 += 8) {
            const float4 lo4 = *reinterpret_cast<const float4*>(p + j0), hi4 = *reinterpret_cast<const float4*>(p + j0 + 4);
            const float x[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
            float pre[8];
#pragma unroll
            for (int u = 0; u < 8; u++) pre[u] = acc = fadd(acc, x[u]);
            if (acc >= top_p || j0 + 8 >= n) {   // (the running value never falls, but entries behind n are not probabilities)
#pragma unroll
                for (int u = 7; u >= 0; u--)
                    if (j0 + u < n && pre[u] >= top_p) keep = j0 + u + 1;
                if (keep < n) break;
            }
        }
    }
    return __shfl_sync(FULL, keep, 0);
}

// Ascending bitonic sort of T * E 64-bit keys by a CTA of T threads: thread t holds the elements t * E .. t * E + E - 1.
// Partners in one thread or one warp are compared in registers; only what crosses warps goes through `buf` (shared memory,
// T * E keys) and barriers: ten exchanges whatever the length up to 2048 keys of 512 threads, where a sort that keeps the
// keys in shared memory has 66 steps with a barrier each (2048 candidates, both sorts of a row: 62 us, now 9).
template <int T, int E>
__device__ __forceinline__ void cta_sort(unsigned long long (&v)[E], unsigned long long* buf) {
    const uint32_t tid = threadIdx.x;
    const auto keep = [&](unsigned long long& mine, unsigned long long other, uint32_t i, uint32_t j, uint32_t k) {
        const bool lower = (i & j) == 0u, up = (i & k) == 0u;
        if ((other < mine) == (lower == up)) mine = other;   // (keys are distinct, or equal ones are alike)
    };
#pragma unroll 1
    for (uint32_t k = 2; k <= (uint32_t)(T * E); k <<= 1) {
        uint32_t j = k >> 1;
#pragma unroll 1
        for (; j >= 32u * E; j >>= 1) {
#pragma unroll
            for (int e = 0; e < E; e++) buf[e * T + tid] = v[e];
            __syncthreads();
#pragma unroll
            for (int e = 0; e < E; e++) keep(v[e], buf[e * T + (tid ^ (j / E))], tid * E + e, j, k);
            __syncthreads();
        }
#pragma unroll 1
        for (; j >= (uint32_t)E; j >>= 1) {
#pragma unroll
            for (int e = 0; e < E; e++) keep(v[e], __shfl_xor_sync(FULL, v[e], (int)(j / E)), tid * E + e, j, k);
        }
#pragma unroll
        for (int jj = E / 2; jj >= 1; jj >>= 1) {
            if ((uint32_t)jj >= k) continue;
#pragma unroll
            for (int e = 0; e < E; e++)
                if (!(e & jj)) {
                    const bool up = ((tid * E + e) & k) == 0u;
                    const unsigned long long x = v[e], y = v[e | jj];
                    if ((x > y) == up) { v[e] = y; v[e | jj] = x; }
                }
        }
    }
}
// The same for n <= LIMIT keys in shared memory (`keys`: room for the next power of two, at least T), in place; the keys
// behind n are overwritten with ones that sort to the end.  Barriers in front and behind.
template <int T, int LIMIT, int E = 1>
__device__ __forceinline__ void cta_sort_shared(unsigned long long* keys, uint32_t n) {
    if constexpr (T * E < LIMIT)
        if (n > (uint32_t)(T * E)) { cta_sort_shared<T, LIMIT, 2 * E>(keys, n); return; }
    if (E == 1 && n <= 32u) {   // one warp
        __syncthreads();
        if (threadIdx.x < 32) {
            unsigned long long v1[1] = {threadIdx.x < n ? keys[threadIdx.x] : ~0ull};
            cta_sort<32, 1>(v1, keys);
            keys[threadIdx.x] = v1[0];
        }
        __syncthreads();
        return;
    }
    unsigned long long v[E];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = threadIdx.x * E + e < n ? keys[threadIdx.x * E + e] : ~0ull;
    __syncthreads();
    cta_sort<T, E>(v, keys);
#pragma unroll
    for (int e = 0; e < E; e++) keys[threadIdx.x * E + e] = v[e];
    __syncthreads();
}

// Total and inverse-CDF pick of the n entries in f.sid / f.sp (id order; kept_n of them above zero), and the row's outputs; one warp.
template <class FA>
__device__ __forceinline__ void warp_finish(FA& f, const RowArgs& a, uint32_t row, uint32_t V, uint32_t n, uint32_t kept_n, float m, float S, float u01,
                                            uint32_t amax, int status) {
    const int lane = threadIdx.x & 31;
    const bool runs = n > F_SERIAL;
    const float total = runs ? warp_fold(f.sp, n, INFINITY, f.fp) : warp_prefix(f.sp, (int)n, f.fp);
    __syncwarp();
    int pick = -1;
    if (total > 1e-9f) {
        const float target = fmul(u01, total);
        pick = runs ? warp_fold_find(f.sp, n, f.fp, SEQ_FIND_GT, target) : warp_find(f.fp, (int)n, SEQ_FIND_GT, target);
    }
    if (lane == 0) {
        uint32_t token = amax;
        int drew = 0;
        if (total > 1e-9f) { token = pick >= 0 ? f.sid[pick] : V - 1; drew = 1; }
        a.token[row] = token; a.status[row] = status;
        if (a.drew) a.drew[row] = (uint8_t)drew;
        if (a.argmax) a.argmax[row] = amax;
        if (a.row_max) a.row_max[row] = m;
        if (a.sumexp) a.sumexp[row] = S;
        if (a.total) a.total[row] = total;
        if (a.n_kept) a.n_kept[row] = kept_n;
    }
    if (a.dump_ids || a.dump_probs) {   // diagnostics: the kept set in id order
        uint32_t done = 0;
        for (uint32_t base = 0; base < n; base += 32) {
            const uint32_t j = base + lane;
            const bool kept = j < n && f.sp[j] > 0.0f;
            const unsigned mask = __ballot_sync(FULL, kept);
            const uint32_t at = done + __popc(mask & ((1u << lane) - 1u));
            if (kept && at < a.dump_cap) {
                if (a.dump_ids) a.dump_ids[(size_t)row * a.dump_cap + at] = f.sid[j];
                if (a.dump_probs) a.dump_probs[(size_t)row * a.dump_cap + at] = f.sp[j];
            }
            done += __popc(mask);
        }
    }
}

// Entries that survive top-k, from ranked probabilities f.rp: every tie at the k-th probability survives; entries with zero
// probability never matter.  f.n_live is zero.  Every thread; barriers in front and behind.
template <int T, class FA>
__device__ __forceinline__ uint32_t cta_top_k(FA& f, uint32_t n, uint32_t top_k) {
    const int tid = threadIdx.x;
    __syncthreads();
    const float thr = (top_k != 0u && top_k <= n) ? f.rp[top_k - 1] : 0.0f;
    for (uint32_t j = tid; j < n; j += T) {
        const bool live = f.rp[j] >= thr && f.rp[j] > 0.0f;
        const bool next_live = j + 1 < n && f.rp[j + 1] >= thr && f.rp[j + 1] > 0.0f;
        if (live && !next_live) f.n_live = j + 1;
    }
    __syncthreads();
    return f.n_live;
}

// Second half of the finish, from ranked candidates: f.sid / f.sp hold the n candidates in id order, f.rp / f.rpos
// the same by (probability descending, id ascending), f.n_live is zero.  Called by every thread; ends with the row's
// outputs written.
template <int T, class FA>
__device__ __forceinline__ void cta_finish_ranked(FA& f, const RowArgs& a, uint32_t row, uint32_t V, uint32_t n, float m,
                                                  float S, uint32_t top_k, float top_p, float u01, uint32_t amax, int status) {
    const int lane = threadIdx.x & 31;
    const uint32_t n_live = cta_top_k<T>(f, n, top_k);
    if (threadIdx.x >= 32) return;
    const uint32_t keep = warp_top_p(f.rp, n_live, top_p, f.fp);
    for (uint32_t j = keep + lane; j < n; j += 32) f.sp[f.rpos[j]] = 0.0f;
    __syncwarp();
    warp_finish(f, a, row, V, n, keep, m, S, u01, amax, status);
}

// Candidates of one row -> token.  Called by every thread of a CTA of T threads (a multiple of 32)
// with a barrier in front; cand_id: the row's n <= F_MCAP candidates in any order, prob(j) their probabilities (memory
// outside of `f`); V: the full vocabulary size (the CDF walk falls through to V - 1, sampler.rs:54).  Ends with the row's
// outputs written; the caller needs a barrier before it reuses `f` or the candidate arrays.
template <int T, class FA, class P>
__device__ __forceinline__ void cta_finish_probs(FA& f, const RowArgs& a, uint32_t row, uint32_t V, const uint32_t* cand_id, P prob, uint32_t n,
                                                 float m, float S, uint32_t top_k, float top_p, float u01, uint32_t amax, int status) {
    static_assert(T % 32 == 0 && F_QUAD % T == 0 || T > F_QUAD, "whole warps");
    const int tid = threadIdx.x;
    if (tid == 0) f.n_live = 0u;
    if (n <= (uint32_t)F_QUAD) {
        // short list: every candidate counts the candidates in front of it, by id and by (probability descending,
        // id ascending)
        constexpr int U = T >= F_QUAD ? 1 : F_QUAD / T;
        uint32_t my_id[U];
        float my_p[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t j = tid + u * T;
            if (j >= n) continue;
            my_id[u] = cand_id[j];
            my_p[u] = prob(j);
            f.key[j] = ((unsigned long long)f2u(my_p[u]) << 32) | (unsigned long long)(0xffffffffu - my_id[u]);   // p >= 0
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (tid + u * T >= n) continue;
            const unsigned long long kj = f.key[tid + u * T];
            uint32_t r_id = 0, r_p = 0;
#pragma unroll 8
            for (uint32_t o = 0; o < n; o++) {   // broadcast loads, independent of one another
                const unsigned long long ko = f.key[o];
                r_p += ko > kj;
                r_id += (uint32_t)ko > (uint32_t)kj;   // larger ~id = smaller id
            }
            f.sid[r_id] = my_id[u]; f.sp[r_id] = my_p[u]; f.rp[r_p] = my_p[u]; f.rpos[r_p] = r_id;
        }
    } else {
        // long list: sorted by (probability descending, id ascending); what top-k and top-p leave is put into id order, by
        // counting where it has become short
        for (uint32_t j = tid; j < n; j += T) f.key[j] = ((unsigned long long)~f2u(prob(j)) << 32) | cand_id[j];
        cta_sort_shared<T, FA::CAPACITY>(f.key, n);
        for (uint32_t r = tid; r < n; r += T) {
            const unsigned long long k = f.key[r];
            f.rp[r] = u2f(~(uint32_t)(k >> 32));
            f.rpos[r] = (uint32_t)k;   // (the id here)
        }
        const uint32_t n_live = cta_top_k<T>(f, n, top_k);
        if (tid < 32) {
            const uint32_t keep = warp_top_p(f.rp, n_live, top_p, f.fp);
            if (tid == 0) f.n_live = keep;
        }
        __syncthreads();
        const uint32_t keep = f.n_live;
        if (keep <= (uint32_t)F_QUAD) {
            for (uint32_t r = tid; r < keep; r += T) {
                const uint32_t id = f.rpos[r];
                uint32_t at = 0;
#pragma unroll 8
                for (uint32_t o = 0; o < keep; o++) at += f.rpos[o] < id;
                f.sid[at] = id; f.sp[at] = f.rp[r];
            }
            __syncthreads();
        } else {
            for (uint32_t r = tid; r < keep; r += T) f.key[r] = ((unsigned long long)f.rpos[r] << 32) | f2u(f.rp[r]);
            cta_sort_shared<T, FA::CAPACITY>(f.key, keep);
            for (uint32_t r = tid; r < keep; r += T) { f.sid[r] = (uint32_t)(f.key[r] >> 32); f.sp[r] = u2f((uint32_t)f.key[r]); }
            __syncthreads();
        }
        if (tid < 32) warp_finish(f, a, row, V, keep, keep, m, S, u01, amax, status);
        return;
    }
    cta_finish_ranked<T, FA>(f, a, row, V, n, m, S, top_k, top_p, u01, amax, status);
}

// The same with the candidates' logits: exact probabilities exp((x - m) / t) / S.
template <int T, class FA>
__device__ __forceinline__ void cta_finish(FA& f, const unsigned long long* exp_tab, const RowArgs& a, uint32_t row,
                                           uint32_t V, const uint32_t* cand_id, const float* cand_x, uint32_t n, float m, float t,
                                           float S, uint32_t top_k, float top_p, float u01, uint32_t amax, int status) {
    const bool norm = S > 1e-9f;
    cta_finish_probs<T>(f, a, row, V, cand_id, [&](uint32_t j) {
        const float e = softmax_num(cand_x[j], m, t, exp_tab);   // exact expf
        return norm ? fdiv(e, S) : e;
    }, n, m, S, top_k, top_p, u01, amax, status);
}

}  // namespace pgs
