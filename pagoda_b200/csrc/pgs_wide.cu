// Wide kernel: all SMs work on every listed row, bit-exact with the reference's serial folds.  It serves the exact mode, the
// rows that the streaming kernel cannot (top-k off or > 1024, rows that are not 16-byte aligned, long candidate lists) and
// log-softmax scoring, as far as one CTA per row is not quicker (pgs_kinds.cuh).
//
// A launch is a sequence of phases with a grid barrier between two of them.  In "region" phases the warps of the grid share
// all regions (512 consecutive logits) of all rows; in "row" phases a CTA does what is left of a row:
//
//   row     parameters; distinct history ids and what the penalties make of them
//   region  sanity, mask, penalties; maximum and plain sum of the softmax numerators relative to it
//   row     row maximum, argmax; estimate of the reference's running f32 sum at every region
//   region  exact numerators; their increments of the running sum, in ulps of its binade
//   row     the f32 left fold, exactly (see fold below)                                  -> S
//   region  histogram of the probabilities                                               (rows with top-k or top-p)
//   row     the bucket in which top-k and top-p end
//   region  probabilities from that bucket upwards into a list, grouped by bucket
//   row     short list: top-k, top-p, total and draw (pgs_finish.cuh).  Long list: the top-p fold over the buckets
//   region  increments of the running total over the kept probabilities                  (what has no short list)
//   row     total and inverse-CDF pick
//
// Batches of many rows, or of short ones, go through the same phases with one CTA per row and a CTA barrier where the grid has
// its own (WideLaunch::local; the host chooses, wide_row_by_row): 148 exact rows of 50257 153 -> 59 us, 256 rows of 151936 316 -> 187.
//
// What bounds it: a row's fold is one warp's (8 us on average and 20 at most of a row of 151936: 500 cycles for each change of binade,
// of which there are 8 to 16); a grid barrier is two microseconds; a region phase is the latency of one or two regions per
// warp (mask, history entries and logits are one trip to L2 or HBM each) rather than bandwidth.  Against the general kernel's CTA per
// row: 32 rows of 151936 without top-k 8312 -> 204 us, 16 rows in exact mode 377 -> 62, 48 rows of 50257 360 -> 59, scoring of 64
// rows 199 -> 74.
//
// The fold (pagoda/src/sampler.rs:42, :99-113, :136-144): while the running value stays inside one binade, adding a
// non-negative term is an integer addition in ulps which depends on the running value only where the term ends exactly on
// half an ulp.  A region (or bucket) without such a tie whose running value provably stays inside one binade is one
// integer, whatever the order; the few others are added in order, each lane of a warp a run of terms that is summarised by
// its increments from an even and from an odd start.  Every summary is checked against the exact
// running value before it is used, so the result is bit-identical to the serial fold.
#include <cuda_runtime.h>

#include "pgs_args.cuh"
#include "pgs_block.cuh"
#include "pgs_finish.cuh"
#include "pgs_general.cuh"
#include "pgs_kinds.cuh"
#include "pgs_wide.cuh"

namespace pgs {

constexpr int WNW = W_NT / 32;
constexpr int WL = W_REGION / 32;        // logits per lane and region
static_assert(WL == RUN, "a region is a warp's runs");
constexpr uint32_t W_NIL = 0xffffffffu;
static_assert(W_KMAX <= F_MCAP / 2, "room for the candidates");
constexpr uint32_t W_DUAL = 2u;          // beside a segment's binade: it may also be the next one

// the terms of a fold: softmax numerators (S <= 0), or the probabilities that are kept
struct Terms {
    float m, t, S;           // S > 0: probabilities, numerator / S when that is above the reference's epsilon
    bool filter;
    float p_thr;
    uint32_t id_thr;
};

struct alignas(16) WideSmem {
    RowArgs a;                           // the launch's arguments, for the phases, which are functions of their own
    WideLaunch l;
    alignas(16) WideRow row;
    alignas(16) WideRow rows[W_CHUNK];               // region phases: the chunk's rows
    unsigned long long exp_tab[32];
    uint32_t red_u[WNW], red_v[WNW];
    float red_f[WNW];
    uint32_t last, found, ok, gave_up;
    uint32_t rank, size, target;         // of the CTA among those that take part; arrivals at the barrier behind this one
    float R;
    Terms terms;                         // of the fold
    uint32_t n_ev, at_ev;                // its events, and how many are behind it
    alignas(16) float stage[WNW][W_REGION];   // per warp: a region in id order
    alignas(16) float spare[W_REGION], spare_too[W_REGION];
    alignas(16) uint4 runs[WNW][32];     // per warp: a segment that is added term by term (see prepare_segment)
    uint32_t run_k[WNW];
    uint32_t serial[W_MAX_REGIONS];      // segments that are added term by term
    unsigned long long red_w[WNW];
    union {
        struct {
            uint2 seg[W_MAX_REGIONS];
            float pre[W_MAX_REGIONS];
            float start[W_MAX_REGIONS];  // exact running value at the segment's start
            uint4 ev[W_MAX_REGIONS + 1];              // what the fold goes through (see resolve)
            unsigned long long ev_sum[W_MAX_REGIONS + 1];   // increments of the segments before
            float ev_R[W_MAX_REGIONS];                // exact running value there; -1: sm.start has it
        };
        uint32_t hash[4 * W_MAX_HIST];   // ids, then counts
        struct {
            uint32_t bn[W_BUCKETS];      // long list: increments per bucket
            float bs[W_BUCKETS];         // plain sums, then estimates of the running value
            unsigned long long sort[W_SORT];
        };
        struct {
            FinishArrays fin;
            uint32_t cand_id[F_MCAP];
            float cand_p[F_MCAP];
        };
        GeneralSmem general;
    };
};
static_assert(sizeof(WideSmem) <= 227 * 1024, "one CTA per SM");
// (The phases are functions of their own and name the CTA's shared memory themselves: through a reference handed to them every
// access would be a generic one.)
__device__ __forceinline__ WideSmem& wide_smem() {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    return *reinterpret_cast<WideSmem*>(smem_raw);
}

// ------------------------------------------------------------------------------------------------ grid barrier

// The CTAs that take part are those that run when the first of them closes the list (at most one per SM fits; usually all
// of the grid, but where another stream's kernel keeps SMs busy the launch does not depend on the rest, which leave at
// once).  So a barrier never waits for a CTA that has not started, and the launch needs no cooperative attribute, which
// costs 3 us and keeps the work-list pass from being set up early.  Waits have a limit all the same; when one runs out the
// CTA leaves (and the others when theirs do), and the last one to leave gives the rows without results a status of their own.
__device__ __forceinline__ bool wait_for(const uint32_t* p, uint32_t target, uint32_t limit) {
    for (uint32_t i = 0; (int32_t)(*(const volatile uint32_t*)p - target) < 0; i++) {
        if (i >= limit) return false;
        __nanosleep(40);
    }
    return true;
}
constexpr uint32_t W_CLOSED = 0x80000000u;   // in sync[5], above the number of CTAs that have joined

// Joins the launch; false: too late.
__device__ __forceinline__ bool grid_join(WideSmem& sm, const WideLaunch& l) {
    if (threadIdx.x == 0) sm.rank = atomicAdd(l.sync + 5, 1u);
    __syncthreads();
    return !(sm.rank & W_CLOSED);
}

// open: rows that have no result yet
__device__ __forceinline__ bool grid_sync(WideSmem& sm, const WideLaunch& l, uint32_t open) {
    __syncthreads();
    if (l.local) return true;   // one CTA per row: nobody else to wait for
    if (threadIdx.x == 0) {
        bool good = true;
        __threadfence();
        atomicAdd(l.sync, 1u);
        if (sm.target == 0u) {   // the first barrier: how many take part?
            if (sm.rank == 0u) {
                wait_for(l.sync + 5, gridDim.x, 64u);
                *(volatile uint32_t*)(l.sync + 6) = atomicOr(l.sync + 5, W_CLOSED);
            } else good = wait_for(l.sync + 6, 1u, l.polls);
            sm.size = *(volatile uint32_t*)(l.sync + 6);
        }
        sm.target += sm.size;
        good = good && wait_for(l.sync, sm.target, l.polls);
        if (!good) { atomicMax(l.sync + 1, open); sm.gave_up = 1u; }
        __threadfence();
        sm.ok = good;
    }
    __syncthreads();
    return sm.ok != 0u;
}

// ------------------------------------------------------------------------------------------------ a warp's region

template <bool BF16, bool VEC> struct WLay {
    static constexpr int ESZ = BF16 ? 2 : 4;
    static constexpr int GE = VEC ? 16 / ESZ : 1;   // consecutive logits of a group
    static constexpr int G = WL / GE;
    static constexpr int GS = 32 * GE;
    __device__ static __forceinline__ uint32_t off(uint32_t lane, uint32_t j) { return (j / GE) * GS + lane * GE + j % GE; }
};

// the lane's raw logits of region r (nv: logits of the region; zeros behind them)
template <bool BF16, bool VEC>
__device__ __forceinline__ void wload(float (&x)[WL], const char* rowp, uint32_t r, uint32_t nv) {
    using L = WLay<BF16, VEC>;
    const uint32_t lane = threadIdx.x & 31;
    const char* p = rowp + (size_t)r * W_REGION * L::ESZ;
#pragma unroll
    for (int h = 0; h < L::G; h++) {
        const uint32_t o = h * L::GS + lane * L::GE;
        const bool in = o < nv;
        if constexpr (VEC && !BF16) {
            const float4 v = in ? __ldcg(reinterpret_cast<const float4*>(p + o * 4)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            x[4 * h] = v.x; x[4 * h + 1] = v.y; x[4 * h + 2] = v.z; x[4 * h + 3] = v.w;
        } else if constexpr (VEC) {
            const uint4 v = in ? __ldcg(reinterpret_cast<const uint4*>(p + o * 2)) : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t u4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                x[h * 8 + 2 * u] = __uint_as_float(u4[u] << 16);
                x[h * 8 + 2 * u + 1] = __uint_as_float(u4[u] & 0xffff0000u);
            }
        } else if constexpr (BF16) x[h] = in ? __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(p) + o) << 16) : 0.0f;
        else x[h] = in ? __ldcg(reinterpret_cast<const float*>(p) + o) : 0.0f;
    }
}

// raw -> processed logits: mask, history entries (values after penalties, mask and EOS fix), end of the row
template <bool BF16, bool VEC>
__device__ __forceinline__ void wprocess(float* buf, float (&x)[WL], const WideLaunch& l, uint32_t slot, const uint32_t* mw, uint32_t entries,
                                         uint32_t r, uint32_t nv) {
    using L = WLay<BF16, VEC>;
    const uint32_t lane = threadIdx.x & 31;
    if (mw) {   // warp-uniform
        const uint32_t word = lane < 16u && lane * 32u < nv ? __ldg(mw + (size_t)r * (W_REGION / 32) + lane) : 0u;
#pragma unroll
        for (int h = 0; h < L::G; h++) {
            const uint32_t o = h * L::GS + lane * L::GE, bits = __shfl_sync(FULL, word, o >> 5) >> (o & 31u);
#pragma unroll
            for (int c = 0; c < L::GE; c++)
                if (!((bits >> c) & 1u)) x[h * L::GE + c] = -INFINITY;
        }
    }
    if (nv < (uint32_t)W_REGION) {
#pragma unroll
        for (int j = 0; j < WL; j++)
            if (L::off(lane, j) >= nv) x[j] = -INFINITY;
    }
    if (entries) {
        const uint32_t* rs = l.rs + (size_t)slot * l.rs_stride + r;
        const uint32_t e0 = __ldcg(rs), e1 = __ldcg(rs + 1);
        if (e0 < e1) {
#pragma unroll
            for (int j = 0; j < WL; j++) buf[L::off(lane, j)] = x[j];
            __syncwarp();
            for (uint32_t e = e0 + lane; e < e1; e += 32)
                buf[__ldcg(l.ent_id + (size_t)slot * (W_MAX_HIST + 32) + e) - r * W_REGION] = __ldcg(l.ent_xn + (size_t)slot * (W_MAX_HIST + 32) + e);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < WL; j++) x[j] = buf[L::off(lane, j)];
            __syncwarp();
        }
    }
}

__device__ __forceinline__ float term_of(float x, uint32_t id, const Terms& f, const unsigned long long* tab) {
    float v = softmax_num(x, f.m, f.t, tab);
    if (f.S >= 0.0f) {
        if (f.S > 1e-9f) v = fdiv(v, f.S);
        if (f.filter && !(v > f.p_thr || (v == f.p_thr && id <= f.id_thr))) v = 0.0f;
    }
    return v;
}

// the terms of region r, from memory
template <bool BF16, bool VEC>
__device__ __forceinline__ void wterms(const unsigned long long* tab, float* buf, float (&x)[WL], const WideLaunch& l, const WideRow& w, uint32_t slot,
                                       uint32_t V, uint32_t r, const Terms& f) {
    using L = WLay<BF16, VEC>;
    const uint32_t lane = threadIdx.x & 31, nv = min(V - r * W_REGION, (uint32_t)W_REGION);
    wload<BF16, VEC>(x, w.rowp, r, nv);
    wprocess<BF16, VEC>(buf, x, l, slot, w.mw, w.entries, r, nv);
#pragma unroll
    for (int j = 0; j < WL; j++) x[j] = term_of(x[j], r * W_REGION + L::off(lane, j), f, tab);
}

// ------------------------------------------------------------------------------------------------ the exact fold

// Increments of the running value over this warp's terms (each lane's share), in ulps of the binade whose lower end has
// the bits `kb`: one integer whatever the order.  W_TIE: has to be added term by term (a term too large for the binade, or
// one that ends on half an ulp).
constexpr uint32_t W_TIE = 0xffffffffu;
__device__ __forceinline__ bool increment(float x, uint32_t kb, uint32_t& n) {
    const uint32_t i0 = f2u(fadd(u2f(kb), x)) - kb, i1 = f2u(fadd(u2f(kb + 1u), x)) - (kb + 1u);
    n += i0;
    return i0 == i1 && x < u2f(kb);
}

// What the approximate terms need to know: with d = x - max (exact as the reference's), log2 of a term in ulps is
// d * c + k0 - log2(ulp).
struct Approx {
    float c, k0;
};
__device__ __forceinline__ Approx approx_of(const Terms& f) {
    Approx q;
    q.c = 1.44269504f / f.t;
    q.k0 = f.S > 1e-9f ? -(float)log2((double)f.S) : 0.0f;
    return q;
}
// The increment of a term is its value in ulps, rounded: the hardware's exp2 decides that unless it lands close to half an
// ulp.  Relative errors, with p = d * c and only terms above a quarter of an ulp (|p| <= |k| + 2) of interest: rounding of
// the argument 4.2e-8 (|k| + 2), of c 5.3e-8 |p|, of the reference's quotient 4.2e-8 |p|, of k and k0 4.2e-8 each, exp2
// 2.4e-7, the reference's exp and division 1.2e-7; less than eps together.  Nearly all terms are far below the running value, so that about one of a region's 512 is in doubt and takes the
// exact exponential, which costs ten times as much (64 rows of 151936: 25 us for all of them).
template <bool BF16, bool VEC>
__device__ __forceinline__ uint32_t increments(const float (&x)[WL], uint32_t id0, const Terms& f, const Approx& q, uint32_t kb, const unsigned long long* tab) {
    const float k = q.k0 - (float)((int)(kb >> 23) - 127 - 23), eps = 2e-7f * fabsf(k) + 1e-7f * fabsf(q.k0) + 1e-6f;
    uint32_t n = 0u, doubt = 0u;
    if (!f.filter) {   // warp-uniform
        // With v the term in ulps and d its distance from the nearest integer, |d| + v * eps >= 1/2 implies d * d + v * eps >= 1/4.
        // (-inf -> 0; beyond 2^23, where d is of no use, v * eps alone is above)
        const float2 m2 = make_float2(-f.m, -f.m), c2 = make_float2(q.c, q.c), k2 = make_float2(k, k), e2 = make_float2(eps, eps);
        const float2 one = make_float2(8388608.0f, 8388608.0f), back = make_float2(-8388608.0f, -8388608.0f), minus = make_float2(-1.0f, -1.0f), quarter = make_float2(-0.25f, -0.25f);
#pragma unroll
        for (int j = 0; j < WL; j += 2) {
            const float2 v = ex2_pair(__ffma2_rn(__fadd2_rn(make_float2(x[j], x[j + 1]), m2), c2, k2)), r = __fadd2_rn(v, one);
            const float2 d = __ffma2_rn(__fadd2_rn(r, back), minus, v), s = __ffma2_rn(d, d, __ffma2_rn(v, e2, quarter));
            n += (f2u(r.x) - 0x4b000000u) + (f2u(r.y) - 0x4b000000u);
            doubt = __funnelshift_l(f2u(s.x), doubt, 1);   // the sign bits, one after the other
            doubt = __funnelshift_l(f2u(s.y), doubt, 1);
        }
        doubt = __brev(~doubt << 16);   // bit j: x[j]
    } else {
        const float p_lim = f.p_thr / u2f(kb) * 8388608.0f, slack = (4.0f * eps + 4e-6f) * p_lim;   // the threshold in ulps
#pragma unroll
        for (int j = 0; j < WL; j++) {
            const float v = ex2_approx_ftz(__fmaf_rn(fsub(x[j], f.m), q.c, k)), r = fadd(v, 8388608.0f);
            bool open = !(__fmaf_rn(v, eps, fabsf(fsub(v, fsub(r, 8388608.0f)))) < 0.5f);
            open = open && !(v < p_lim - slack);
            open = open || fabsf(v - p_lim) <= slack;
            if (!(v < p_lim) || open) n += f2u(r) - 0x4b000000u;
            if (open) doubt |= 1u << j;
        }
    }
    bool good = true;
    while (__any_sync(FULL, doubt != 0u)) {
        if (doubt) {
            const int j = __ffs((int)doubt) - 1;
            float xj = x[0];
#pragma unroll
            for (int u = 1; u < WL; u++) if (u == j) xj = x[u];
            n -= f2u(fadd(ex2_approx_ftz(__fmaf_rn(fsub(xj, f.m), q.c, k)), 8388608.0f)) - 0x4b000000u;   // (as above)
            good &= increment(term_of(xj, id0 + WLay<BF16, VEC>::off(threadIdx.x & 31u, (uint32_t)j), f, tab), kb, n);
            doubt &= doubt - 1u;
        }
    }
    if (__any_sync(FULL, !good || n >= 0x01000000u)) return W_TIE;
    return __reduce_add_sync(FULL, n);   // (the table keeps the sum below 2^24 ulps)
}

// the warp's terms, as a region holds them, into id order: lane k gets the terms k * WL ..
template <class L>
__device__ __forceinline__ void to_runs(float* buf, float (&v)[WL], const float (&x)[WL]) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < WL; j++) buf[L::off(lane, j)] = x[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < WL; j++) v[j] = buf[lane * WL + j];
    __syncwarp();
}

// A segment that is added term by term, made ready for add_segment by one warp: v, the lanes' runs; pre, the estimate of the
// running value at its start.  Most such segments are those in which the running value changes binade once.  So per lane, each
// from an even and from an odd value: the increments up to and including its run in the binade at the start (x, y), and those of
// its run and all behind it in the next binade (z, w).
__device__ __forceinline__ void prepare_segment(WideSmem& sm, uint32_t w, const float (&v)[WL], float pre) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < WL; j += 4) *reinterpret_cast<float4*>(&sm.stage[w][lane * WL + j]) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    uint32_t k = f2u(pre * 0.9995f) & 0x7f800000u;   // (the estimate is too large, by a few 1e-4, rather than too small)
    if (k == 0u || k >= 0x7f000000u) k = W_NIL;   // none
    uint4 s = make_uint4(0u, 0u, 0u, 0u);
    if (k != W_NIL) {   // warp-uniform
        uint32_t c0, c1;
        run_increments(v, k, c0, c1);
        const unsigned tie = __ballot_sync(FULL, c0 != c1);
        s.x = warp_scan_u32(increment_from(c0, c1, tie, 0u));
        s.y = tie ? warp_scan_u32(increment_from(c0, c1, tie, 1u)) : s.x;
        run_increments(v, k + 0x00800000u, c0, c1);
        s.z = min(c0, 0x00800000u); s.w = min(c1, 0x00800000u);   // (2^23 leaves the binade whatever else is added)
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {   // (left, right)(p) = left_p + right_{(p + left_p) & 1}
            const uint32_t r0 = __shfl_down_sync(FULL, s.z, o), r1 = __shfl_down_sync(FULL, s.w, o);
            if (lane + (uint32_t)o < 32u) { s.z += (s.z & 1u) ? r1 : r0; s.w += (s.w & 1u) ? r0 : r1; }
        }
    }
    sm.runs[w][lane] = s;
    if (lane == 0) sm.run_k[w] = k;
}
// the terms of the runs pos .. n - 1, one after the other
__device__ __forceinline__ float add_run(float R, const float* terms, uint32_t pos, uint32_t n) {
    const float4* v = reinterpret_cast<const float4*>(terms + pos * WL);
    float4 a[WL / 4];
#pragma unroll
    for (int j = 0; j < WL / 4; j++) a[j] = v[j];
#pragma unroll 1
    for (;;) {
        pos++;
        v += pos < n ? WL / 4 : 0;
#pragma unroll
        for (int j = 0; j < WL / 4; j++) {   // (the next run is on its way while this one is added)
            const float4 t = a[j];
            a[j] = v[j];
            R = fadd(R, t.x); R = fadd(R, t.y); R = fadd(R, t.z); R = fadd(R, t.w);
        }
        if (pos >= n) return R;
    }
}
// Adds the segment that warp q has made ready to the exact running value R, as far as what has been made ready serves for it; one
// warp.  Returns how many of the 32 runs are done.
__device__ __forceinline__ uint32_t add_segment(const WideSmem& sm, uint32_t q, float& R) {
    const uint32_t k = sm.run_k[q], rb = f2u(R);
    const uint4 s = sm.runs[q][threadIdx.x & 31];
    if ((rb & 0x7f800000u) != k) return 0u;
    const uint32_t d = (rb & 1u) ? s.y : s.x;
    const uint32_t over = ~__ballot_sync(FULL, d < 0x00800000u - (rb & 0x007fffffu));   // (the lanes' increments only grow)
    const uint32_t n = over ? (uint32_t)__ffs((int)over) - 1u : 32u, inc = __shfl_sync(FULL, d, (int)(n - 1u) & 31);
    R = u2f(rb + (n ? inc : 0u));
    if (n == 32u) return 32u;
    R = add_run(R, sm.stage[q], n, n + 1u);   // the run in which the binade changes
    if (n == 31u) return 32u;
    const uint32_t r1 = f2u(R), all = __shfl_sync(FULL, (r1 & 1u) ? s.w : s.z, (int)n + 1);
    if ((r1 & 0x7f800000u) != k + 0x00800000u || all >= 0x00800000u - (r1 & 0x007fffffu)) return n + 1u;
    R = u2f(r1 + all);
    return 32u;
}

// The segments [pos, stop), for which the estimate was not good enough, added to the exact running value R; one warp.
template <bool BF16, bool VEC>
__device__ __noinline__ float add_slowly(uint32_t slot, float R, uint32_t pos, uint32_t stop) {
    WideSmem& sm = wide_smem();
    const WideLaunch& l = sm.l;
    const uint32_t lane = threadIdx.x & 31, V = sm.a.vocab;
    while (pos < stop) {   // whole segments up to the next one that is not
        uint2 sg = pos + lane < stop ? sm.seg[pos + lane] : make_uint2(0u, 1u);
        const uint32_t rb = f2u(R), kb = rb & 0x7f800000u;
        if ((sg.y & W_DUAL) && kb == sg.y - W_DUAL + 0x00800000u) sg = make_uint2(f2u(sm.pre[pos + lane]), kb);
        sg.y &= ~W_DUAL;
        const unsigned not_ok = ~__ballot_sync(FULL, sg.y == 1u || sg.y == kb);
        uint32_t cnt = not_ok ? __ffs((int)not_ok) - 1u : 32u;
        uint32_t inc = lane < cnt ? sg.x : 0u;
        const uint32_t own = inc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, inc, o);
            if (lane >= (uint32_t)o) inc += t;
        }
        const unsigned over = __ballot_sync(FULL, (rb & 0x007fffffu) + inc >= 0x00800000u && own != 0u);
        if (over) cnt = min(cnt, (uint32_t)__ffs((int)over) - 1u);
        if (cnt) {
            if (lane < cnt && pos + lane < stop) sm.start[pos + lane] = u2f(rb + inc - own);
            R = u2f(rb + __shfl_sync(FULL, inc, (int)cnt - 1));
            pos = min(pos + cnt, stop);
        } else {
            float x[WL], v[WL];
            wterms<BF16, VEC>(sm.exp_tab, sm.spare, x, l, sm.row, slot, V, pos, sm.terms);
            to_runs<WLay<BF16, VEC>>(sm.spare, v, x);
            if (lane == 0) sm.start[pos] = R;
            R = add_runs(R, v);
            pos++;
        }
    }
    return R;
}

// the lowest id of region r whose processed logit is m; one warp
template <bool BF16, bool VEC>
__device__ __forceinline__ uint32_t find_in_region(float* buf, const WideRow& row, const WideLaunch& l, uint32_t slot, uint32_t V, uint32_t r, float m) {
    float x[WL];
    const uint32_t nv = min(V - r * W_REGION, (uint32_t)W_REGION);
    wload<BF16, VEC>(x, row.rowp, r, nv);
    wprocess<BF16, VEC>(buf, x, l, slot, row.mw, row.entries, r, nv);
    uint32_t o = W_NIL;
#pragma unroll
    for (int j = WL - 1; j >= 0; j--)
        if (x[j] == m) o = WLay<BF16, VEC>::off(threadIdx.x & 31, j);   // (a lane's logits are in id order)
    return r * W_REGION + __reduce_min_sync(FULL, o);
}

template <bool BF16, bool VEC>
__device__ __noinline__ void argmax_row(uint32_t slot) {
    WideSmem& sm = wide_smem();
    const uint32_t id = find_in_region<BF16, VEC>(sm.spare_too, sm.row, sm.l, slot, sm.a.vocab, sm.row.max_region, sm.row.m);
    if ((threadIdx.x & 31) == 0) sm.row.amax = id;
}

// Warp 0's way through the events (see resolve) up to the first segment, of those to be added term by term, that is not among
// the `ready` ones made ready so far (the first of them by warp 0, number q0).  A function of its own, whose inner loop has the
// usual cases alone: its registers hold nothing else, and nothing is called from there.
template <bool BF16, bool VEC>
__device__ __noinline__ float walk(uint32_t slot, float R, uint32_t q0, uint32_t ready) {
    WideSmem& sm = wide_smem();
    const uint32_t lane = threadIdx.x & 31, n_ev = sm.n_ev;
    uint32_t e = sm.at_ev, q = q0;
    for (;;) {
        uint32_t done = 32u;   // runs of the segment at which the loop stops; above: not a segment
        float at_start;
#pragma unroll 1
        for (; e < n_ev; e++) {
            const uint4 x = sm.ev[e];
            at_start = R;
            if (x.y == 0u) {
                if (q == ready) break;
                done = add_segment(sm, q - q0, R);
                if (done != 32u) break;
                q++;
            } else {
                const uint32_t rb = f2u(R), kb = rb & 0x7f800000u, k = x.y & ~W_DUAL;
                const bool second = (x.y & W_DUAL) && kb == k + 0x00800000u;
                const uint32_t inc = second ? x.w : x.z;
                if (x.y != 1u && (!(kb == k || second) || inc >= 0x00800000u - (rb & 0x007fffffu))) { done = 33u; break; }
                R = u2f(rb + inc);   // (zeros: inc is zero)
            }
            if (lane == 0) sm.ev_R[e] = at_start;
        }
        if (done == 32u) break;
        if (done < 32u) {
            const float* terms = sm.stage[q - q0];
            if (at_start == 0.0f) R = add_run(R, terms, 0u, done = 32u);   // the start of the row: a new binade every few terms
            else {
                float v[WL];
#pragma unroll
                for (int j = 0; j < WL; j += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(terms + lane * WL + j);
                    v[j] = t.x; v[j + 1] = t.y; v[j + 2] = t.z; v[j + 3] = t.w;
                }
                R = add_runs(R, v, nullptr, done);
            }
            q++;
        } else {
            R = add_slowly<BF16, VEC>(slot, R, sm.ev[e].x, sm.ev[e + 1u].x);
            at_start = -1.0f;
        }
        if (lane == 0) sm.ev_R[e] = at_start;
        e++;
    }
    if (lane == 0) sm.at_ev = e;
    __syncwarp();
    return R;
}

// The exact left fold of a row's terms from the segments that the grid left in l.seg (estimates of the running value in
// l.pre); the CTA.  Leaves the running value at every region's start in sm.start.  argmax: another warp looks for the row's
// argmax beside the walk.
//
// One warp goes through the row's events, each from the exact running value: a segment that is added term by term, one that
// lies in either of two binades, or a run of segments of one binade (or of zeros), whose increments a scan has added up, so that
// the run is one addition if it stays in the binade.  That walk is the serial part; 64 scored rows of 151936, whose walks have 13
// such segments and 11 runs on average, us a row on average and at most: 15 and 34 when runs were scanned 32 segments at a time
// and the runs of terms inside a segment relied on estimated binades, now 8 and 21 (in cycles: a run of segments 70, a segment
// 300, with a change of binade 500, the first segment of a row 2500).
template <bool BF16, bool VEC>
__device__ __noinline__ float resolve(uint32_t slot, uint32_t V, const Terms f, bool argmax) {
    WideSmem& sm = wide_smem();
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, n_regions = (V + W_REGION - 1) / W_REGION;
    const WideRow& row = sm.row;
    __syncthreads();
    for (uint32_t r = tid; r < n_regions; r += W_NT) {
        sm.seg[r] = __ldcg(l.seg + (size_t)slot * l.reg_stride + r);
        sm.pre[r] = __ldcg(l.pre + (size_t)slot * l.reg_stride + r);
    }
    __syncthreads();
    // the events: two regions per thread; increments, events and segments to be added term by term in one scan
    static_assert(W_MAX_REGIONS == 2 * W_NT && W_MAX_REGIONS < 1 << 12, "packed counts");
    constexpr unsigned long long EVENT = 1ull << 12;
    unsigned long long own[2], sum;   // increments << 24 | events << 12 | segments
    uint32_t n_ev, n_serial;
    {
        uint32_t yp = tid && 2u * tid <= n_regions ? sm.seg[2u * tid - 1u].y : W_NIL;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint32_t r = 2u * tid + u;
            own[u] = 0ull;
            if (r < n_regions) {
                const uint2 sg = sm.seg[r];
                const bool single = sg.y == 0u || (sg.y & W_DUAL);
                if (!single) own[u] = (unsigned long long)min(sg.x, 0x01000000u) << 24;   // (2^23 is too much already)
                if (single || sg.y != yp) own[u] |= EVENT;
                own[u] |= sg.y == 0u;
                yp = sg.y;
            }
        }
        unsigned long long inc = own[0] + own[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(FULL, inc, o);
            if (lane >= (uint32_t)o) inc += t;
        }
        if (lane == 31) sm.red_w[w] = inc;
        __syncthreads();
        unsigned long long before = sm.red_w[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(FULL, before, o);
            if (lane >= (uint32_t)o) before += t;
        }
        const unsigned long long all = __shfl_sync(FULL, before, 31);
        before = __shfl_sync(FULL, before, (int)(w + 31u) & 31);
        sum = (w ? before : 0ull) + inc - own[0] - own[1];   // in front of this thread's regions
        n_ev = (uint32_t)(all >> 12) & 0xfffu; n_serial = (uint32_t)all & 0xfffu;
        unsigned long long s = sum;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint32_t e = (uint32_t)(s >> 12) & 0xfffu;
            if (own[u] & EVENT) { sm.ev[e].x = 2u * tid + u; sm.ev_sum[e] = s >> 24; }
            if (own[u] & 1ull) sm.serial[(uint32_t)s & 0xfffu] = 2u * tid + u;
            s += own[u];
        }
        if (tid == 0) { sm.ev[n_ev].x = n_regions; sm.ev_sum[n_ev] = all >> 24; sm.n_ev = n_ev; sm.at_ev = 0u; sm.terms = f; }
    }
    __syncthreads();
    for (uint32_t e = tid; e < n_ev; e += W_NT) {
        const uint32_t at = sm.ev[e].x;
        const uint2 sg = sm.seg[at];
        const unsigned long long run = sm.ev_sum[e + 1u] - sm.ev_sum[e];
        sm.ev[e].y = sg.y;
        sm.ev[e].z = sg.y & W_DUAL ? sg.x : (uint32_t)min(run, 0xffffffffull);
        sm.ev[e].w = f2u(sm.pre[at]);   // (of a segment in either of two binades: the increments in the second)
    }
    float R = 0.0f;        // warp 0
    for (uint32_t b = 0; b < n_serial || b == 0u; b += WNW) {
        if (b + w < n_serial) {
            const uint32_t r = sm.serial[b + w], at = sm.seg[r].x;
            float v[WL];
            if (at) {   // the region phase has left the terms
                const float4* t = reinterpret_cast<const float4*>(l.terms + ((size_t)slot * W_TERMS + at - 1u) * W_REGION) + lane * (WL / 4);
#pragma unroll
                for (int j = 0; j < WL / 4; j++) {
                    const float4 q4 = __ldcg(t + j);
                    v[4 * j] = q4.x; v[4 * j + 1] = q4.y; v[4 * j + 2] = q4.z; v[4 * j + 3] = q4.w;
                }
            } else {
                float x[WL];
                wterms<BF16, VEC>(sm.exp_tab, sm.stage[w], x, l, row, slot, V, r, f);
                to_runs<WLay<BF16, VEC>>(sm.stage[w], v, x);
            }
            prepare_segment(sm, w, v, sm.pre[r]);
        }
        __syncthreads();
        if (w == 0) R = walk<BF16, VEC>(slot, R, b, min(n_serial, b + WNW));
        if (w == 1 && b == 0u && argmax) argmax_row<BF16, VEC>(slot);
        __syncthreads();
    }
    if (tid == 0) sm.R = R;
    {
        unsigned long long s = sum;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint32_t r = 2u * tid + u;
            if (r >= n_regions) break;
            const uint32_t i = ((uint32_t)((s + own[u]) >> 12) & 0xfffu) - 1u;   // the event that the region belongs to
            const float at = sm.ev_R[i];
            if (at >= 0.0f) sm.start[r] = u2f(f2u(at) + (uint32_t)((s >> 24) - sm.ev_sum[i]));
            s += own[u];
        }
    }
    __syncthreads();
    return sm.R;
}

// Table entry of a segment whose plain sum P begins at the estimate `pre` of the running value: the binade that the running
// value stays in; that binade | W_DUAL when it may also be in the next one throughout (the estimate is close to the border);
// 0 when it is expected to change there.  The plain sums overestimate the running value by up to a few 1e-4 (the small terms
// it drops), hence the slack.
__device__ __forceinline__ uint32_t binade(float v) { return f2u(v) & 0x7f800000u; }
__device__ __forceinline__ uint32_t segment_binade(float pre, float P, float slack) {
    const float lo = pre * (1.0f - slack), hi = (pre + P) * (1.0f + slack);
    const uint32_t kb = binade(lo);
    if (kb == 0u || !(hi < INFINITY) || !(P * (1.0f + slack) < 0.999f * u2f(kb))) return 0u;
    if (kb == binade(hi)) return kb;
    return kb + 0x00800000u == binade(hi) && binade(pre) == binade(pre + P) ? kb | W_DUAL : 0u;
}
// The same for the fold towards top-p, for one binade only.  It ends before the running value is 1, so what may come to 1 or more
// stays in the binade below as far as the fold goes.  (With 1 as a border like the others, every bucket behind 0.998 was to be
// added entry by entry: 32 rows of 151936 with top-p 0.999 took 2.7 ms bucket by bucket, and 9.2 on a CTA that sorts the whole
// row, where there were too many of them for the list of events; now 0.5.)
__device__ __forceinline__ uint32_t top_p_binade(float pre, float P, float slack) {
    constexpr float BELOW_ONE = 0.99999994f;
    const float lo = fminf(pre * (1.0f - slack), BELOW_ONE), hi = fminf((pre + P) * (1.0f + slack), BELOW_ONE);
    const uint32_t kb = binade(lo);
    return kb != 0u && P * (1.0f + slack) < 0.999f * u2f(kb) && kb == binade(hi) ? kb : 0u;
}

// exclusive scan over the CTA (plain adds: estimates only); one barrier in front, one behind
__device__ __forceinline__ float wscan_f32(WideSmem& sm, float v, float* total) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(FULL, inc, o);
        if (lane >= (uint32_t)o) inc += t;
    }
    __syncthreads();
    if (lane == 31) sm.red_f[w] = inc;
    __syncthreads();
    const float x = sm.red_f[lane];
    float xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(FULL, xi, o);
        if (lane >= (uint32_t)o) xi += t;
    }
    *total = __shfl_sync(FULL, xi, 31);
    return __shfl_sync(FULL, xi - x, (int)w) + (inc - v);
}

// Table of a row's regions from their plain sums P(r): estimates and binades for the next region phase.
template <class F>
__device__ __forceinline__ void make_table(WideSmem& sm, const WideLaunch& l, uint32_t slot, uint32_t n_regions, float slack, F P) {
    float carry = 0.0f;
    for (uint32_t r0 = 0; r0 < n_regions; r0 += W_NT) {
        const uint32_t r = r0 + threadIdx.x;
        const float p = r < n_regions ? P(r) : 0.0f;
        float tot;
        const float pre = carry + wscan_f32(sm, p, &tot);
        if (r < n_regions) {
            l.pre[(size_t)slot * l.reg_stride + r] = pre;
            l.seg[(size_t)slot * l.reg_stride + r] = make_uint2(0u, segment_binade(pre, p, slack));
        }
        carry += tot;
    }
}

// ------------------------------------------------------------------------------------------------ row phases

__device__ __forceinline__ void wresult(const RowArgs& a, uint32_t row, uint32_t token, int status, int drew) {
    a.token[row] = token;
    a.status[row] = status;
    if (a.drew) a.drew[row] = (uint8_t)drew;
}
// outcome of a row that draws nothing
__device__ __forceinline__ void wresult_plain(const RowArgs& a, uint32_t row, int status, uint32_t amax, float m) {
    wresult(a, row, amax, status, 0);
    if (a.argmax) a.argmax[row] = amax;
    if (a.row_max) a.row_max[row] = m;
    if (a.sumexp) a.sumexp[row] = 0.0f;
    if (a.total) a.total[row] = 0.0f;
    if (a.n_kept) a.n_kept[row] = 0u;
}
__device__ __forceinline__ void wleave(const WideLaunch& l, uint32_t row) { l.left_rows[atomicAdd(l.left_count, 1u)] = row; }

__device__ __forceinline__ void row_in(WideSmem& sm, const WideLaunch& l, uint32_t slot) {
    __syncthreads();
    const uint32_t* from = reinterpret_cast<const uint32_t*>(l.row + slot);
    if (threadIdx.x < sizeof(WideRow) / 4) reinterpret_cast<uint32_t*>(&sm.row)[threadIdx.x] = __ldcg(from + threadIdx.x);
    __syncthreads();
}
// the chunk's rows, for a region phase; a barrier behind
__device__ __forceinline__ void rows_in(WideSmem& sm, const WideLaunch& l, uint32_t n_rows) {
    const uint32_t* from = reinterpret_cast<const uint32_t*>(l.row);
    for (uint32_t i = threadIdx.x; i < n_rows * (uint32_t)(sizeof(WideRow) / 4); i += W_NT) reinterpret_cast<uint32_t*>(sm.rows)[i] = __ldcg(from + i);
    __syncthreads();
}
__device__ __forceinline__ void row_out(WideSmem& sm, const WideLaunch& l, uint32_t slot) {
    __syncthreads();
    if (threadIdx.x < sizeof(WideRow) / 4)
        reinterpret_cast<uint32_t*>(l.row + slot)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&sm.row)[threadIdx.x];
}

// Parameters (same rules as the other kernels), and the distinct history ids of the row grouped by region with the values
// the chain sees there.
template <bool BF16>
__device__ __noinline__ void open_row(uint32_t slot, uint32_t row) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x, V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    __syncthreads();
    uint32_t param = 0u;
    if (tid < 32) {   // one parameter per lane, so that their latencies overlap
        const void* from[11] = {a.temperature, a.top_k, a.top_p, a.freq, a.pres, a.rep, a.uniform, a.mask_table, a.mask_state, a.hist_offsets, a.hist_offsets};
        const void* p = nullptr;
#pragma unroll
        for (int u = 0; u < 11; u++) if (tid == (uint32_t)u) p = from[u];
        param = tid == 2u || tid == 5u ? f2u(1.0f) : tid == 7u ? 0xffffffffu : 0u;   // top-p and repetition off, no mask
        if (p) param = static_cast<const uint32_t*>(p)[row + (tid == 10u ? 1u : 0u)];
    }
    const auto get = [&](int u) { return __shfl_sync(FULL, param, u); };
    if (tid < 32) {
        WideRow& c = sm.row;
        const float temp = l.score ? 1.0f : u2f(get(0)), top_p = u2f(get(2)), freq = u2f(get(3)), pres = u2f(get(4)), rep = u2f(get(5)), u01 = u2f(get(6));
        const uint32_t top_k = get(1), h0 = get(9), h1 = get(10);
        const int32_t mt = (int32_t)get(7), ms = (int32_t)get(8);
        if (tid == 0) {
            c.row = row;
            c.rowp = (const char*)a.logits + (size_t)row * a.row_stride * (BF16 ? 2 : 4);
            c.temp = temp; c.top_k = top_k; c.top_p = top_p; c.freq = freq; c.pres = pres; c.rep = rep; c.u01 = u01;
            c.t = fmaxf(c.temp, 1e-9f);
            bool bad = !finite_f(c.temp) || !finite_f(c.top_p) || !finite_f(c.freq) || !finite_f(c.pres) || !finite_f(c.rep) || !(c.rep > 0.0f) ||
                       !finite_f(c.u01);
            c.mw = nullptr;
            c.gflags = 0u;
            if (mt >= 0) {
                if (mt >= MAX_TABLES || !a.tables[mt].live || ms < 0 || (uint32_t)ms >= a.tables[mt].n_states ||
                    (unsigned long long)a.tables[mt].words_per_state * 32ull < V) bad = true;
                else {
                    c.mw = a.tables[mt].words + (size_t)ms * a.tables[mt].words_per_state;
                    c.gflags = a.tables[mt].flags[ms];
                }
            }
            c.h0 = h0;
            c.nh = 0u;
            if (h1 < c.h0 || h1 - c.h0 > a.max_history || (h1 > c.h0 && !a.hist_ids)) bad = true; else c.nh = h1 - c.h0;
            if ((fabsf(c.freq) < 1e-6f && fabsf(c.pres) < 1e-6f) && c.rep == 1.0f) c.nh = 0u;
            c.entries = 0u;
            c.nonfinite = 0u;
            c.n_terms = 0u;
            c.state = WS_FIRST;
            c.n_list = 0u; c.cut_x = INFINITY; c.n_kept = 0u; c.p_thr = -1.0f; c.id_thr = 0u; c.cut = 0u; c.m = -INFINITY; c.S = 0.0f; c.amax = 0u;
            if (bad) { wresult_plain(a, row, ROW_BAD_PARAM, 0u, -INFINITY); c.state = WS_DONE; }
            else if (c.nh > (uint32_t)W_MAX_HIST) { wleave(l, row); c.state = WS_DONE; }
        }
    }
    __syncthreads();
    const WideRow& c = sm.row;
    const bool fix = (c.gflags & 1u) && c.mw && a.eos >= 0 && (uint32_t)a.eos < V;   // engine.rs:1307-1312
    if (c.state == WS_FIRST && (c.nh || fix)) {
        uint32_t* rcnt = sm.serial;   // ids per region, then the scatter cursor
        uint32_t H = 64;
        while (H < 2u * (c.nh + 1u) && H < 2u * W_MAX_HIST) H <<= 1;
        uint32_t *hkey = sm.hash, *hcnt = sm.hash + H;
        for (uint32_t s = tid; s < 2u * H; s += W_NT) sm.hash[s] = s < H ? W_NIL : 0u;
        for (uint32_t r = tid; r < n_regions; r += W_NT) rcnt[r] = 0u;
        __syncthreads();
        for (uint32_t j = tid; j < c.nh + (fix ? 1u : 0u); j += W_NT) {
            const bool is_fix = j == c.nh;
            const uint32_t id = is_fix ? (uint32_t)a.eos : __ldg(a.hist_ids + c.h0 + j);
            if (id >= V) continue;   // engine.rs:1562
            uint32_t s = (id * 2654435761u) & (H - 1u);
            for (uint32_t probe = 0; probe < H; probe++) {
                const uint32_t prev = atomicCAS(&hkey[s], W_NIL, id);
                if (prev == W_NIL) atomicAdd(&rcnt[id / W_REGION], 1u);
                if (prev == W_NIL || prev == id) { if (!is_fix) atomicAdd(&hcnt[s], 1u); break; }
                s = (s + 1u) & (H - 1u);
            }
        }
        __syncthreads();
        uint32_t carry = 0u;
        for (uint32_t r0 = 0; r0 < n_regions; r0 += W_NT) {
            const uint32_t r = r0 + tid, lane = tid & 31, w = tid >> 5;
            const uint32_t v = r < n_regions ? rcnt[r] : 0u;
            uint32_t inc = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= (uint32_t)o) inc += t;
            }
            if (lane == 31) sm.red_u[w] = inc;
            __syncthreads();
            const uint32_t x = sm.red_u[lane];
            const uint32_t before = carry + __reduce_add_sync(FULL, lane < w ? x : 0u) + inc - v;
            carry += __reduce_add_sync(FULL, x);
            if (r < n_regions) { l.rs[(size_t)slot * l.rs_stride + r] = before; rcnt[r] = before; }
            __syncthreads();
        }
        if (tid == 0) { l.rs[(size_t)slot * l.rs_stride + n_regions] = carry; sm.row.entries = carry; }
        const bool do_fp = !(fabsf(c.freq) < 1e-6f && fabsf(c.pres) < 1e-6f), do_pres = fabsf(c.pres) > 1e-6f, do_rep = c.rep != 1.0f;
        for (uint32_t s = tid; s < H; s += W_NT) {
            const uint32_t id = hkey[s];
            if (id == W_NIL) continue;
            float v = BF16 ? __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(c.rowp) + id) << 16)
                           : __ldcg(reinterpret_cast<const float*>(c.rowp) + id);
            const bool allowed = !c.mw || ((__ldg(c.mw + (id >> 5)) >> (id & 31u)) & 1u);
            const uint32_t n = hcnt[s];
            if (n) {
                if (do_rep) v = v > 0.0f ? fdiv(v, c.rep) : fmul(v, c.rep);
                if (do_fp) {
                    v = fsub(v, fmul(c.freq, (float)n));
                    if (do_pres) v = fsub(v, c.pres);
                }
            }
            if (!allowed || !finite_f(v)) v = -INFINITY;   // an overflowed penalty counts as masked
            if (fix && id == (uint32_t)a.eos && !finite_f(v)) v = 0.0f;
            const uint32_t at = atomicAdd(&rcnt[id / W_REGION], 1u);
            l.ent_id[(size_t)slot * (W_MAX_HIST + 32) + at] = id;
            l.ent_xn[(size_t)slot * (W_MAX_HIST + 32) + at] = v;
        }
    }
    row_out(sm, l, slot);
}

// Row maximum, argmax, and the table for the fold of the numerators.
template <bool BF16, bool VEC>
__device__ __noinline__ void maximum_row(uint32_t slot) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    row_in(sm, l, slot);
    if (sm.row.state != WS_FIRST) return;
    uint32_t k = 0u, rr = W_NIL;
    for (uint32_t r = tid; r < n_regions; r += W_NT) {
        const float2 v = __ldcg(l.reg + (size_t)slot * l.reg_stride + r);
        sm.pre[r] = v.x; sm.start[r] = v.y;
        const uint32_t kr = order_key(v.x);
        if (kr > k) { k = kr; rr = r; }
    }
    const uint32_t wk = __reduce_max_sync(FULL, k), wr = __reduce_min_sync(FULL, k == wk ? rr : W_NIL);
    if (lane == 0) { sm.red_u[w] = wk; sm.red_v[w] = wr; }
    __syncthreads();
    const uint32_t kk = sm.red_u[lane], gkey = __reduce_max_sync(FULL, kk);
    const uint32_t rstar = __reduce_min_sync(FULL, kk == gkey ? sm.red_v[lane] : W_NIL);
    const bool any = gkey != 0u;
    const float m = any ? key_to_float(gkey) : -INFINITY;
    // (a row that goes on to be sampled looks for it beside the walk of its fold)
    const bool ends_here = !l.score && (sm.row.temp < 1e-5f || (sm.row.gflags & 2u));
    if (w == 0 && any && !sm.row.nonfinite && ends_here) {
        if (lane == 0) { sm.row.m = m; sm.row.max_region = rstar; }
        __syncwarp();
        argmax_row<BF16, VEC>(slot);
    }
    __syncthreads();
    if (tid == 0) {
        WideRow& c = sm.row;
        c.m = m;
        c.max_region = rstar;
        c.state = WS_DONE;
        if (l.score) {
            if (a.status) a.status[c.row] = c.nonfinite ? ROW_NONFINITE : ROW_OK;
            if (c.nonfinite || !any) { if (l.out_gather) l.out_gather[c.row] = NAN; }   // the reference does not define scores for such rows
            else c.state = WS_SUM;
        } else if (c.nonfinite) {
            wresult_plain(a, c.row, ROW_NONFINITE, 0u, -INFINITY);
            if (a.faulted) atomicAdd(a.faulted, 1ull);
        } else if (c.gflags & 2u) wresult_plain(a, c.row, ROW_DEAD, 0u, -INFINITY);
        else if (c.temp < 1e-5f || !any) wresult_plain(a, c.row, any ? ROW_OK : ROW_EMPTY, any ? c.amax : 0u, m);
        else c.state = WS_SUM;
    }
    __syncthreads();
    if (sm.row.state == WS_SUM && sm.row.cut_x == INFINITY && !l.score && sm.row.top_k != 0u && sm.row.top_k < V && sm.row.top_k <= (uint32_t)W_KMAX) {
        // A row with a short top-k: the k-th largest of the parts' maxima is reached by at least k logits, so everything
        // from a little below it on (for ties) is a superset of the top-k set, and nearly always a small one.  As in the
        // streaming kernel: buckets of equal width between the smallest finite maximum and the largest.
        const uint32_t k = sm.row.top_k, n_cells = 4u * n_regions;
        const float* cell = reinterpret_cast<const float*>(l.cell + (size_t)slot * l.reg_stride);
        uint32_t lo = W_NIL, fin = 0u;
        float mine[8];
        static_assert(4 * W_MAX_REGIONS == 8 * W_NT && W_NT == 1024, "eight maxima and one bucket per thread");
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint32_t i = tid + u * W_NT;
            mine[u] = i < n_cells ? __ldcg(cell + i) : -INFINITY;
            const uint32_t key = order_key(mine[u]);
            if (key) { lo = umin(lo, key); fin++; }
        }
        lo = __reduce_min_sync(FULL, lo); fin = __reduce_add_sync(FULL, fin);
        if (lane == 0) { sm.red_u[w] = lo; sm.red_v[w] = fin; }
        if (tid == 0) sm.last = 0u;
        __syncthreads();
        lo = __reduce_min_sync(FULL, sm.red_u[lane]); fin = __reduce_add_sync(FULL, sm.red_v[lane]);
        if (fin >= k) {   // CTA-uniform
            const float lo_v = key_to_float(lo), scb = m > lo_v ? 1023.0f / (m - lo_v) : 0.0f;
            uint32_t* bucket = sm.serial;   // (1024 of them)
            bucket[tid] = 0u;
            __syncthreads();
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (finite_f(mine[u])) atomicAdd(&bucket[min(1023u, (uint32_t)((mine[u] - lo_v) * scb))], 1u);
            __syncthreads();
            const uint32_t own = bucket[1023u - tid];
            uint32_t inc = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= (uint32_t)o) inc += t;
            }
            if (lane == 31) sm.red_u[w] = inc;
            __syncthreads();
            const uint32_t x = sm.red_u[lane], above = __reduce_add_sync(FULL, lane < w ? x : 0u) + inc - own;
            if (above < k && k <= above + own) sm.last = 1023u - tid;
            __syncthreads();
            const float bound = sm.last >= 1u && scb > 0.0f ? lo_v + ((float)sm.last - 1.0f) / scb : lo_v;
            // (finite also where the margin overflows: what is masked, or behind the end of the row, is never a candidate)
            if (tid == 0) sm.row.cut_x = fmaxf(bound - 4.8e-7f * (fabsf(m - bound) + 4.0f * sm.row.t) - 4.8e-7f * (fabsf(bound) + fabsf(m)), -3.402823466e38f);
        }
    }
    if (sm.row.state == WS_SUM && tid == 0 && !l.score && !(sm.row.cut_x < INFINITY))   // (known to all behind the next barrier)
        atomicAdd(l.sync + ((sm.row.top_k != 0u && sm.row.top_k < V) || !(sm.row.top_p >= 1.0f) ? 2 : 3), 1u);
    if (sm.row.state == WS_SUM) {
        const float sc = 1.44269504f / sm.row.t;
        make_table(sm, l, slot, n_regions, 0.001953125f + 1e-7f * fabsf(m * sc), [&](uint32_t r) {
            return sm.start[r] > 0.0f ? sm.start[r] * ex2_approx_ftz((sm.pre[r] - m) * sc) : 0.0f;
        });
    }
    row_out(sm, l, slot);
}

__device__ __forceinline__ uint32_t bucket_of(float p) {
    const int b = (int)(f2u(p) >> 15) - (87 << 8);
    return b < 0 ? 0u : min((uint32_t)b, (uint32_t)W_BUCKETS - 1u);
}
__device__ __forceinline__ float bucket_floor(uint32_t b) { return b ? u2f((b + (87u << 8)) << 15) : 0.0f; }

// The sum of the numerators; rows with top-k or top-p go on to the selection, others to the total.
template <bool BF16, bool VEC>
__device__ __noinline__ void sum_row(uint32_t slot) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    row_in(sm, l, slot);
    if (sm.row.state != WS_SUM) return;
    Terms f;
    f.m = sm.row.m; f.t = sm.row.t; f.S = -1.0f; f.filter = false; f.p_thr = 0.0f; f.id_thr = 0u;
    const float S = resolve<BF16, VEC>(slot, V, f, !l.score);
    if (threadIdx.x == 0) sm.row.n_terms = 0u;
    const bool use_k = sm.row.top_k != 0u && sm.row.top_k < V, use_p = !(sm.row.top_p >= 1.0f);
    __syncthreads();
    if (threadIdx.x == 0) {
        WideRow& c = sm.row;
        c.S = S;
        if (l.score) {   // sampler.rs:73-87
            c.total = fmaxf(__double2float_rn(log((double)S)), 1.17549435e-38f);
            c.state = l.out_full ? WS_TOTAL : WS_DONE;
            if (l.ids && l.out_gather) {
                const uint32_t id = l.ids[c.row];
                float v = NAN;
                if (id < V) {
                    const float e = pgs_expf_tab(fsub(reinterpret_cast<const float*>(c.rowp)[id], c.m), sm.exp_tab);
                    v = fsub(__double2float_rn(log((double)e)), c.total);
                }
                l.out_gather[c.row] = v;
            }
        } else c.state = c.cut_x < INFINITY && c.n_list <= (uint32_t)F_MCAP ? WS_DONE : use_k || use_p ? WS_SELECT : WS_TOTAL;
    }
    __syncthreads();
    if (sm.row.state == WS_DONE && !l.score) {   // the second pass has found the candidates
        const uint32_t n = sm.row.n_list;
        for (uint32_t j = threadIdx.x; j < n; j += W_NT) {
            const unsigned long long v = __ldcg(l.list + (size_t)slot * l.list_stride + j);
            sm.cand_id[j] = (uint32_t)v; sm.cand_p[j] = u2f((uint32_t)(v >> 32));
        }
        __syncthreads();
        cta_finish<W_NT>(sm.fin, sm.exp_tab, a, sm.row.row, V, sm.cand_id, sm.cand_p, n, sm.row.m, sm.row.t, S, sm.row.top_k, sm.row.top_p,
                         sm.row.u01, sm.row.amax, ROW_OK);
    }
    if (sm.row.state == WS_SELECT) {
        for (uint32_t b = threadIdx.x; b < (uint32_t)W_BUCKETS; b += W_NT) l.hist[(size_t)slot * W_BUCKETS + b] = 0u;
        if (threadIdx.x == 0) sm.row.n_list = 0u;
    }
    if (sm.row.state == WS_TOTAL && !l.score) {
        const float q = S > 1e-9f ? 1.0f / S : 1.0f;
        make_table(sm, l, slot, n_regions, 0.001953125f, [&](uint32_t r) { return ((r + 1u < n_regions ? sm.start[r + 1u] : S) - sm.start[r]) * q; });
    }
    row_out(sm, l, slot);
}

// The lowest bucket that is counted.  Top-p alone ends where what lies above amounts to top_p (by the lower ends of the buckets,
// 2^-8 below the probabilities at most, and with the margin of select_row); all V logits below the bucket together are less than
// what is then left.  A row for which that does not hold, as its sum is not that of its terms, is left to the general kernel.
// (32 rows of 151936 with top-p 0.95: a quarter of the logits are counted.)
__device__ __forceinline__ uint32_t lowest_bucket(const WideRow& c, uint32_t V) {
    if ((c.top_k != 0u && c.top_k < V) || c.top_p >= 1.0f) return 0u;
    const float left = 0.999f * (1.0f - fmaxf(c.top_p, 0.0f) * 1.002f / 0.99609375f);   // (the probabilities' own sum is 1 to within 1e-3)
    return left > 0.001f ? bucket_of((left - 0.001f) / (float)V) : 0u;
}

// The lowest bucket that can matter: the one with the k-th largest probability, or the one in which the top-p fold ends (a
// lower bound of the mass above it exceeds top-p by more than the fold can lose).  List positions for the buckets above.
__device__ __noinline__ void select_row(uint32_t slot) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    constexpr int PER = (W_BUCKETS + W_NT - 1) / W_NT;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, V = a.vocab;
    row_in(sm, l, slot);
    if (sm.row.state != WS_SELECT) return;
    uint32_t* hist = l.hist + (size_t)slot * W_BUCKETS;
    const uint32_t k = sm.row.top_k;
    const bool use_k = k != 0u && k < V, use_p = !(sm.row.top_p >= 1.0f);
    uint32_t n[PER], own = 0u;
    float mass = 0.0f;
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int b = W_BUCKETS - 1 - (int)(tid * PER) - u;
        n[u] = b >= 0 ? __ldcg(hist + b) : 0u;
    }
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int b = W_BUCKETS - 1 - (int)(tid * PER) - u;
        own += n[u];
        if (b > 0) mass += (float)n[u] * bucket_floor(b);
    }
    if (tid == 0) { sm.last = 0u; sm.found = 0u; }
    float all;
    float above_mass = wscan_f32(sm, mass, &all);
    uint32_t inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, inc, o);
        if (lane >= (uint32_t)o) inc += t;
    }
    if (lane == 31) sm.red_u[w] = inc;
    __syncthreads();
    const uint32_t x = sm.red_u[lane];
    const uint32_t before = __reduce_add_sync(FULL, lane < w ? x : 0u) + inc - own;
    const float goal = fmaxf(sm.row.top_p * 1.002f, 1.17549435e-38f);   // (top-p of zero or less: the highest bucket with an entry)
    {
        uint32_t above = before;
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int b = W_BUCKETS - 1 - (int)(tid * PER) - u;
            if (b > 0) {
                if (use_k && above < k && k <= above + n[u]) atomicMax(&sm.last, (uint32_t)b);
                const float next = above_mass + (float)n[u] * bucket_floor(b);
                if (use_p && above_mass < goal && next >= goal) atomicMax(&sm.found, (uint32_t)b);
                above_mass = next;
            }
            above += n[u];
        }
    }
    __syncthreads();
    const uint32_t cut = umax(sm.last, sm.found), low = lowest_bucket(sm.row, V);
    if (cut < low) {   // CTA-uniform: what is counted does not come to top-p (a sum far from that of its terms)
        if (tid == 0) { wleave(l, sm.row.row); sm.row.state = WS_DONE; }
        row_out(sm, l, slot);
        return;
    }
    {
        uint32_t above = before;
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int b = W_BUCKETS - 1 - (int)(tid * PER) - u;
            if (b >= (int)cut) {
                hist[b] = above;
                if (b == (int)cut) sm.row.n_list = above + n[u];
            }
            above += n[u];
        }
    }
    if (tid == 0) sm.row.cut = cut | (use_k && sm.last == cut ? 0x80000000u : 0u);   // top bit: top-k ends in the cut bucket
    row_out(sm, l, slot);
}

// bucket b of the row's list as sorted keys (probability descending, id ascending) in sm.sort; false when it is too long
__device__ __forceinline__ bool sort_bucket(WideSmem& sm, const WideLaunch& l, uint32_t slot, uint32_t at, uint32_t n) {
    if (n > (uint32_t)W_SORT) return false;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < n; j += W_NT) {
        const unsigned long long v = __ldcg(l.list + (size_t)slot * l.list_stride + at + j);
        sm.sort[j] = ((unsigned long long)(~(uint32_t)(v >> 32)) << 32) | (uint32_t)v;
    }
    cta_sort_shared<W_NT, W_SORT>(sm.sort, n);
    return true;
}

// Top-k and top-p on the list.  A short list is finished here; a long one leaves the last kept (probability, id) and the
// table for the fold of the kept probabilities.
__device__ __noinline__ void choose_row(uint32_t slot) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    row_in(sm, l, slot);
    if (sm.row.state != WS_SELECT) return;
    const uint32_t n = sm.row.n_list, k = sm.row.top_k, cut = sm.row.cut & 0x7fffffffu, row = sm.row.row;
    const bool use_k = k != 0u && k < V, use_p = !(sm.row.top_p >= 1.0f), k_ends = sm.row.cut != cut;
    const unsigned long long* list = l.list + (size_t)slot * l.list_stride;
    if (n <= (uint32_t)F_MCAP) {
        for (uint32_t j = tid; j < n; j += W_NT) {
            const unsigned long long v = __ldcg(list + j);
            sm.cand_id[j] = (uint32_t)v; sm.cand_p[j] = u2f((uint32_t)(v >> 32));
        }
        __syncthreads();
        cta_finish_probs<W_NT>(sm.fin, a, row, V, sm.cand_id, [&](uint32_t j) { return sm.cand_p[j]; }, n, sm.row.m, sm.row.S, use_k ? k : 0u,
                               sm.row.top_p, sm.row.u01, sm.row.amax, ROW_OK);
        __syncthreads();
        if (tid == 0) sm.row.state = WS_DONE;
        row_out(sm, l, slot);
        return;
    }
    // the entries of the list, four of a thread under way at once (one trip to L2 after the other took 20 us for 14000 entries)
    const auto each = [&](auto what) {
#pragma unroll 1
        for (uint32_t j0 = tid; j0 < n; j0 += 4u * W_NT) {
            unsigned long long v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = j0 + u * W_NT < n ? __ldcg(list + j0 + u * W_NT) : 0ull;
#pragma unroll
            for (int u = 0; u < 4; u++) if (j0 + u * W_NT < n) what(u2f((uint32_t)(v[u] >> 32)), (uint32_t)v[u]);
        }
    };
    const uint32_t* hist = l.hist + (size_t)slot * W_BUCKETS;   // where bucket b ends in the list; it begins where b + 1 ends
    float thr_k = 0.0f;
    bool leave = false;
    uint32_t n_live = n;
    if (k_ends && k <= n) {
        const uint32_t at = cut + 1u < (uint32_t)W_BUCKETS ? __ldcg(hist + cut + 1u) : 0u, nb = n - at;
        leave = !sort_bucket(sm, l, slot, at, nb);
        if (!leave) {
            thr_k = u2f(~(uint32_t)(sm.sort[k - at - 1u] >> 32));
            uint32_t mine = 0u;
            for (uint32_t j = tid; j < nb; j += W_NT) mine += u2f(~(uint32_t)(sm.sort[j] >> 32)) >= thr_k;
            mine = __reduce_add_sync(FULL, mine);
            if (lane == 0) sm.red_u[w] = mine;
            __syncthreads();
            n_live = at + __reduce_add_sync(FULL, sm.red_u[lane]);
        }
    }
    float p_thr = thr_k;
    uint32_t id_thr = 0xffffffffu, n_kept = n_live;
    if (use_p && !leave) {
        __syncthreads();
        for (uint32_t b = cut + tid; b < (uint32_t)W_BUCKETS; b += W_NT) { sm.bn[b] = 0u; sm.bs[b] = 0.0f; }
        __syncthreads();
        // (the entries of a bucket share their upper bits: their sum is their number and the sum of the 15 lower bits, whole numbers,
        // which shared memory adds faster than floats; three bits less, 2^-20 of the sum, so that it fits 32 bits for every row)
        static_assert((0x7fffu >> 3) <= 0xffffffffu / ((uint32_t)W_MAX_REGIONS * W_REGION), "all logits in one bucket");
        uint32_t* lower = reinterpret_cast<uint32_t*>(sm.bs);
        each([&](float p, uint32_t) {
            if (!(p >= thr_k)) return;
            const uint32_t b = bucket_of(p);
            atomicAdd(&sm.bn[b], 1u);
            atomicAdd(&lower[b], (f2u(p) & 0x7fffu) >> 3);
        });
        __syncthreads();
        {   // plain sums -> the binade of the running value at each bucket
            constexpr int PER = (W_BUCKETS + W_NT - 1) / W_NT;
            float own = 0.0f, P[PER];
#pragma unroll
            for (int u = 0; u < PER; u++) {
                const int b = W_BUCKETS - 1 - (int)(tid * PER) - u;
                P[u] = 0.0f;
                if (b >= (int)cut && sm.bn[b]) {   // (bucket 0: of no account)
                    const float floor_b = bucket_floor(b);
                    P[u] = (float)sm.bn[b] * floor_b + (float)lower[b] * (u2f(binade(floor_b)) * 9.5367431640625e-07f);
                    sm.bn[b] = 0u;
                }
                own += P[u];
            }
            float all;
            float pre = wscan_f32(sm, own, &all);
#pragma unroll
            for (int u = 0; u < PER; u++) {
                const int b = W_BUCKETS - 1 - (int)(tid * PER) - u;
                if (b >= (int)cut) sm.bs[b] = u2f(top_p_binade(pre, P[u], 0.001953125f));
                pre += P[u];
            }
        }
        __syncthreads();
        each([&](float p, uint32_t) {
            if (!(p >= thr_k)) return;
            const uint32_t b = bucket_of(p), kb = f2u(sm.bs[b]);
            if (kb == 0u) { sm.bn[b] = f2u(p); return; }   // (of use where the bucket has one entry)
            const uint32_t i0 = f2u(fadd(u2f(kb), p)) - kb, i1 = f2u(fadd(u2f(kb + 1u), p)) - (kb + 1u);
            if (i0 != i1 || !(p < u2f(kb))) { sm.bs[b] = 0.0f; sm.bn[b] = f2u(p); }   // to be added one by one
            else atomicAdd(&sm.bn[b], i0);
        });
        // The fold over the buckets, highest first, by events as in resolve: a run of buckets of one binade is one addition; a
        // bucket with several entries that the running value may change binade in, the one in which top-p is reached, and one in
        // which a run turns out not as estimated, is sorted by the CTA and its entries are added in order.  (Over the buckets 256
        // at a time the walk took 27 us a row.)
        uint32_t* ends = reinterpret_cast<uint32_t*>(&sm.stage[0][0]);   // where a bucket ends in the list
        unsigned long long* ev_sum = reinterpret_cast<unsigned long long*>(ends + W_BUCKETS);
        uint32_t* ev = sm.serial;   // the bucket an event begins with
        static_assert(sizeof(sm.stage) >= W_BUCKETS * 4 + (W_MAX_REGIONS + 1) * 8 && W_BUCKETS % 2 == 0, "one word per bucket, the events' sums");
        for (uint32_t b = cut + tid; b < (uint32_t)W_BUCKETS; b += W_NT) ends[b] = __ldcg(hist + b);
        __syncthreads();
        constexpr int PER = (W_BUCKETS + W_NT - 1) / W_NT;
        constexpr uint32_t EV_MASK = 0x3fffu;   // events in the lower bits of a sum, increments above
        static_assert(W_BUCKETS <= 0x3fff, "packed counts");
        unsigned long long all, before;
        uint32_t is_event = 0u;   // bit u: this thread's bucket u
        const auto bucket = [&](int u) { return W_BUCKETS - 1 - (int)(tid * PER) - u; };
        const auto increment_in = [&](int bb) { return f2u(sm.bs[bb]) ? (unsigned long long)min(sm.bn[bb], 0x01000000u) : 0ull; };   // (2^23 is too much already)
        const auto empty = [&](int bb) { return bb < (int)cut || ends[bb] == (bb + 1 < W_BUCKETS ? ends[bb + 1] : 0u); };
        {
            uint32_t last_y = W_NIL;   // of the thread's buckets that are not empty
            unsigned long long own = 0ull;
            for (int u = 0; u < PER; u++) if (!empty(bucket(u))) last_y = f2u(sm.bs[bucket(u)]);
            const unsigned some = __ballot_sync(FULL, last_y != W_NIL) & ((1u << lane) - 1u);
            const uint32_t from = __shfl_sync(FULL, last_y, some ? 31 - __clz((int)some) : 0);
            uint32_t yp = some ? from : W_NIL;   // (an event at the start of every warp's buckets)
            for (int u = 0; u < PER; u++) {
                const int bb = bucket(u);
                if (empty(bb)) continue;
                const uint32_t y = f2u(sm.bs[bb]);
                if (y == 0u || y != yp) { is_event |= 1u << u; own++; }
                own += increment_in(bb) << 14;
                yp = y;
            }
            unsigned long long inc = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(FULL, inc, o);
                if (lane >= (uint32_t)o) inc += t;
            }
            if (lane == 31) sm.red_w[w] = inc;
            __syncthreads();
            before = sm.red_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(FULL, before, o);
                if (lane >= (uint32_t)o) before += t;
            }
            all = __shfl_sync(FULL, before, 31);
            before = __shfl_sync(FULL, before, (int)(w + 31u) & 31);
            before = (w ? before : 0ull) + inc - own;
        }
        const uint32_t n_ev = (uint32_t)all & EV_MASK;
        leave = n_ev > (uint32_t)W_MAX_REGIONS;   // CTA-uniform
        if (!leave) {
            unsigned long long at = before;
            for (int u = 0; u < PER; u++) {
                const int bb = bucket(u);
                if (empty(bb)) continue;
                if ((is_event >> u) & 1u) { ev[(uint32_t)at & EV_MASK] = (uint32_t)bb; ev_sum[(uint32_t)at & EV_MASK] = at >> 14; at++; }
                at += increment_in(bb) << 14;
            }
            if (tid == 0) ev_sum[n_ev] = all >> 14;
        }
        float R = 0.0f;                              // warp 0
        uint32_t e = 0u;
        // A run that does not go by in one addition is cut at a bucket, which is sorted like the others; the run's buckets above
        // `limit` are behind it then, with the increments up to `from`.
        uint32_t cut_run = W_NIL, limit = 0u;        // the event that these hold for
        unsigned long long from = 0ull;
        bool found = false;
        while (!leave) {
            __syncthreads();
            if (w == 0) {
                uint32_t need = W_NIL, in_run = 0u;
#pragma unroll 1
                for (; e < n_ev; e++) {
                    const uint32_t b = ev[e], k = f2u(sm.bs[b]), rb = f2u(R);
                    if (k == 0u) {   // (a single entry that does not reach top-p needs no sort)
                        const float R1 = fadd(R, u2f(sm.bn[b]));
                        if (ends[b] - (b + 1u < (uint32_t)W_BUCKETS ? ends[b + 1u] : 0u) == 1u && R1 < sm.row.top_p) R = R1;
                        else { need = b; e++; break; }
                    } else {
                        const unsigned long long run = ev_sum[e + 1u] - (e == cut_run ? from : ev_sum[e]);
                        if ((rb & 0x7f800000u) != k || run >= 0x00800000u - (rb & 0x007fffffu) || u2f(rb + (uint32_t)run) >= sm.row.top_p) {
                            need = b; in_run = 1u;
                            break;
                        }
                        R = u2f(rb + (uint32_t)run);
                    }
                }
                if (lane == 0) { sm.last = need; sm.n_ev = in_run; sm.at_ev = e; sm.R = R; sm.found = 0u; }
            }
            __syncthreads();
            if (sm.n_ev) {   // the first bucket of the run that top-p is reached in, or that leaves the binade, or any where the estimate missed it
                const uint32_t run = sm.at_ev, rb = f2u(sm.R), room = 0x00800000u - (rb & 0x007fffffu);
                const bool other = (rb & 0x7f800000u) != f2u(sm.bs[ev[run]]);
                if (run != cut_run) { cut_run = run; limit = W_BUCKETS; from = ev_sum[run]; }
                unsigned long long at = before;
                for (int u = 0; u < PER; u++) {
                    const int bb = bucket(u);
                    if (empty(bb)) continue;
                    const uint32_t i = ((uint32_t)at & EV_MASK) + ((is_event >> u) & 1u) - 1u;   // the event that the bucket belongs to
                    at += (increment_in(bb) << 14) + ((is_event >> u) & 1u);
                    if (i != run || (uint32_t)bb >= limit) continue;
                    const unsigned long long inc = (at >> 14) - from;
                    if (other || inc >= room || u2f(rb + (uint32_t)inc) >= sm.row.top_p) atomicMax(&sm.found, (uint32_t)bb + 1u);
                }
                __syncthreads();
                if (sm.found == 0u) {   // CTA-uniform: nothing is left of the run
                    e++;
                    continue;
                }
                limit = sm.found - 1u;
                at = before;
                for (int u = 0; u < PER; u++) {   // the running value in front of it
                    const int bb = bucket(u);
                    if (empty(bb)) continue;
                    const unsigned long long in_front = at >> 14;
                    at += (increment_in(bb) << 14) + ((is_event >> u) & 1u);
                    if ((uint32_t)bb == limit) { sm.R = u2f(rb + (uint32_t)(in_front - from)); sm.red_w[0] = at >> 14; sm.last = limit; }
                }
                __syncthreads();
                R = sm.R;
                from = sm.red_w[0];
            }
            const uint32_t sb = sm.last;
            if (sb == W_NIL) break;
            const uint32_t end = ends[sb], at = sb + 1u < (uint32_t)W_BUCKETS ? ends[sb + 1u] : 0u, nb = end - at;
            if (!sort_bucket(sm, l, slot, at, nb)) { leave = true; break; }
            if (w == 0) {
                uint32_t hit = W_NIL;
                for (uint32_t j0 = 0; j0 < nb && hit == W_NIL; j0 += W_REGION) {
                    float v[WL];
#pragma unroll
                    for (int j = 0; j < WL; j++) {
                        const uint32_t q = j0 + lane * WL + j;
                        const float p = q < nb ? u2f(~(uint32_t)(sm.sort[q] >> 32)) : 0.0f;
                        v[j] = p >= thr_k ? p : 0.0f;
                    }
                    const float R1 = add_runs(R, v);
                    if (R1 >= sm.row.top_p) {   // in here: one lane looks for the entry
                        if (lane == 0) {
                            float r = R;
                            uint32_t q = j0;
                            for (; q < nb && q < j0 + W_REGION; q++) {
                                const float p = u2f(~(uint32_t)(sm.sort[q] >> 32));
                                r = fadd(r, p >= thr_k ? p : 0.0f);
                                if (r >= sm.row.top_p) break;
                            }
                            hit = q;
                        }
                        hit = __shfl_sync(FULL, hit, 0);
                    }
                    R = R1;
                }
                if (lane == 0) sm.found = hit;
            }
            __syncthreads();
            if (sm.found != W_NIL) {
                found = true;
                p_thr = u2f(~(uint32_t)(sm.sort[sm.found] >> 32));
                id_thr = (uint32_t)sm.sort[sm.found];
                n_kept = at + sm.found + 1u;
                break;
            }
        }
        // top-p was not reached although the list ends where it should have been: the list is too short for this row
        if (!found && !leave && cut != 0u && !k_ends) leave = true;
    }
    __syncthreads();
    if (leave) {
        if (tid == 0) { wleave(l, row); sm.row.state = WS_DONE; }
        row_out(sm, l, slot);
        return;
    }
    for (uint32_t r = tid; r < n_regions; r += W_NT) sm.start[r] = 0.0f;
    __syncthreads();
    each([&](float p, uint32_t id) { if (p > p_thr || (p == p_thr && id <= id_thr)) atomicAdd(&sm.start[id / W_REGION], p); });
    __syncthreads();
    make_table(sm, l, slot, n_regions, 0.001953125f, [&](uint32_t r) { return sm.start[r]; });
    if (tid == 0) {
        WideRow& c = sm.row;
        c.p_thr = p_thr; c.id_thr = id_thr; c.n_kept = n_kept;
        c.state = WS_TOTAL;
        atomicAdd(l.sync + 3, 1u);
    }
    row_out(sm, l, slot);
}

__device__ __forceinline__ Terms kept_terms(const WideRow& c, uint32_t V) {
    Terms f;
    f.m = c.m; f.t = c.t; f.S = c.S;
    f.filter = (c.top_k != 0u && c.top_k < V) || !(c.top_p >= 1.0f);
    f.p_thr = c.p_thr; f.id_thr = c.id_thr;
    return f;
}

// Total of the kept probabilities and the inverse-CDF pick.
template <bool BF16, bool VEC>
__device__ __noinline__ void total_row(uint32_t slot) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    row_in(sm, l, slot);
    if (sm.row.state != WS_TOTAL) return;
    const Terms f = kept_terms(sm.row, V);
    const float total = resolve<BF16, VEC>(slot, V, f, false);
    const float target = fmul(sm.row.u01, total);
    if (tid == 0) sm.found = W_NIL;
    __syncthreads();
    if (total > 1e-9f)
        for (uint32_t r = tid; r < n_regions; r += W_NT)
            if (target < (r + 1u < n_regions ? sm.start[r + 1u] : total)) atomicMin(&sm.found, r);
    __syncthreads();
    const uint32_t row = sm.row.row, r = sm.found;
    uint32_t token = sm.row.amax;
    if (total > 1e-9f) token = V - 1u;   // (also when no running value exceeds the target, sampler.rs:54)
    if (w == 0) {
        if (r != W_NIL) {   // the running value exceeds the target in this region: one lane looks for the id
            float x[WL], v[WL];
            wterms<BF16, VEC>(sm.exp_tab, sm.spare, x, l, sm.row, slot, V, r, f);
            to_runs<WLay<BF16, VEC>>(sm.spare, v, x);
            add_runs(sm.start[r], v, sm.red_f);
            __syncwarp();
            const unsigned over = __ballot_sync(FULL, target < sm.red_f[lane]);
            if (lane == 0 && over) {
                const uint32_t run = __ffs((int)over) - 1u;
                float acc = run ? sm.red_f[run - 1u] : sm.start[r];
                for (uint32_t j = run * WL; j < (run + 1u) * WL; j++) {
                    acc = fadd(acc, sm.spare[j]);
                    if (target < acc) { token = r * W_REGION + j; break; }
                }
            }
        }
        if (lane == 0) {
            wresult(a, row, token, ROW_OK, total > 1e-9f ? 1 : 0);
            if (a.argmax) a.argmax[row] = sm.row.amax;
            if (a.row_max) a.row_max[row] = sm.row.m;
            if (a.sumexp) a.sumexp[row] = sm.row.S;
            if (a.total) a.total[row] = total;
        }
    }
    if (tid == 0 && a.n_kept) a.n_kept[row] = sm.row.n_kept;
    if (a.dump_ids || a.dump_probs) {   // diagnostics: the kept set in id order
        uint32_t done = 0u;
        for (uint32_t r0 = 0; r0 < n_regions; r0 += WNW) {
            __syncthreads();
            float x[WL], v[WL];
            uint32_t n = 0u;
            if (r0 + w < n_regions) {
                wterms<BF16, VEC>(sm.exp_tab, sm.stage[w], x, l, sm.row, slot, V, r0 + w, f);
                to_runs<WLay<BF16, VEC>>(sm.stage[w], v, x);
#pragma unroll
                for (int j = 0; j < WL; j++) n += v[j] > 0.0f;
            }
            uint32_t inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= (uint32_t)o) inc += t;
            }
            if (lane == 31) sm.red_u[w] = inc;
            __syncthreads();
            const uint32_t c = sm.red_u[lane];
            uint32_t at = done + __reduce_add_sync(FULL, lane < w ? c : 0u) + inc - n;
            done += __reduce_add_sync(FULL, c);
            if (n) {
#pragma unroll
                for (int j = 0; j < WL; j++)
                    if (v[j] > 0.0f) {
                        if (at < a.dump_cap) {
                            if (a.dump_ids) a.dump_ids[(size_t)row * a.dump_cap + at] = (r0 + w) * W_REGION + lane * WL + j;
                            if (a.dump_probs) a.dump_probs[(size_t)row * a.dump_cap + at] = v[j];
                        }
                        at++;
                    }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ region phases

enum : int { WP_FIRST = 0, WP_SUM, WP_LIST, WP_TOTAL, WP_FULL };

// One region phase, with the barrier in front of it (open: as there): the warps of the grid take the regions of all rows of the
// chunk, which begins with row c0, in turn.  False: the barrier was given up.
template <bool BF16, bool VEC, int PHASE>
__device__ __noinline__ bool region_phase(uint32_t n_rows, uint32_t c0, uint32_t open) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    using L = WLay<BF16, VEC>;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    float* buf = sm.stage[w];
    const bool first = sm.target == 0u;   // (how many take part is known behind the first barrier)
    if (PHASE == WP_FIRST) {   // the warp's first region is on its way while the barrier is waited for
        const uint32_t i = w * (first ? gridDim.x : sm.size) + sm.rank, slot = i / n_regions, at = (i - slot * n_regions) * W_REGION + lane * (128u / L::ESZ);
        if (slot < n_rows && lane < W_REGION * L::ESZ / 128u && at < V)
            prefetch_l2((const char*)a.logits + ((size_t)(a.work_rows ? a.work_rows[c0 + slot] : c0 + slot) * a.row_stride + at) * L::ESZ);
    }
    if (!grid_sync(sm, l, open)) return false;
    if (PHASE == WP_FIRST && first && sm.size < n_rows) return true;   // rows are still to be opened
    rows_in(sm, l, n_rows);
    for (uint32_t i = w * sm.size + sm.rank; i < n_rows * n_regions; i += sm.size * WNW) {
        const uint32_t slot = i / n_regions, r = i - slot * n_regions, nv = min(V - r * W_REGION, (uint32_t)W_REGION);
        const WideRow& c = sm.rows[slot];
        const uint32_t state = c.state;
        {   // the region after this one, a 128-byte line per lane
            const uint32_t i1 = i + sm.size * WNW, slot1 = i1 / n_regions, r1 = i1 - slot1 * n_regions;
            const uint32_t at = r1 * W_REGION + lane * (128u / L::ESZ);
            if (i1 < n_rows * n_regions && lane < W_REGION * L::ESZ / 128u && at < V) prefetch_l2(sm.rows[slot1].rowp + (size_t)at * L::ESZ);
        }
        float x[WL];
        if (PHASE == WP_FIRST) {
            if (state != WS_FIRST) continue;
            wload<BF16, VEC>(x, c.rowp, r, nv);
            float am = 0.0f;   // max |raw logit|, NaN-propagating
#pragma unroll
            for (int j = 0; j < WL; j += 2) am = absmax3_nan(am, x[j], x[j + 1]);
            wprocess<BF16, VEC>(buf, x, l, slot, c.mw, c.entries, r, nv);
            float top = x[0];
#pragma unroll
            for (int j = 1; j + 1 < WL; j += 2) top = max3f(top, x[j], x[j + 1]);
            top = fmaxf(top, x[WL - 1]);
            float part = top;   // of eight lanes
#pragma unroll
            for (int o = 4; o; o >>= 1) part = fmaxf(part, __shfl_xor_sync(FULL, part, o));
            if ((lane & 7u) == 0u) reinterpret_cast<float*>(l.cell + (size_t)slot * l.reg_stride + r)[lane >> 3] = part;
            uint32_t key = f2u(top);
            key = __reduce_max_sync(FULL, key ^ (((uint32_t)((int32_t)key >> 31)) | 0x80000000u));   // monotone; -inf lowest
            const float wm = u2f((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key), sc = 1.44269504f / c.t;
            float s = 0.0f;
            if (wm > -INFINITY) {
                const float2 m2 = make_float2(-wm, -wm), sc2 = make_float2(sc, sc);
                float2 a2 = make_float2(0.0f, 0.0f), b2 = a2;
#pragma unroll
                for (int j = 0; j < WL; j += 4) {
                    a2 = __fadd2_rn(a2, ex2_pair(__fmul2_rn(__fadd2_rn(make_float2(x[j], x[j + 1]), m2), sc2)));
                    b2 = __fadd2_rn(b2, ex2_pair(__fmul2_rn(__fadd2_rn(make_float2(x[j + 2], x[j + 3]), m2), sc2)));
                }
                s = (a2.x + a2.y) + (b2.x + b2.y);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
            const uint32_t bad = __any_sync(FULL, !(am < INFINITY));
            if (lane == 0) {
                l.reg[(size_t)slot * l.reg_stride + r] = make_float2(wm, s);
                if (bad) l.row[slot].nonfinite = 1u;
            }
            continue;
        }
        if (state != (PHASE == WP_SUM ? WS_SUM : PHASE == WP_LIST ? WS_SELECT : WS_TOTAL)) continue;
        if (PHASE == WP_FULL) {   // the whole log-softmax vector
            const float log_sum = c.total;
            const uint32_t row = c.row;
            wload<BF16, VEC>(x, c.rowp, r, nv);
#pragma unroll
            for (int j = 0; j < WL; j++) {
                const uint32_t o = L::off(lane, j);
                const float e = pgs_expf_tab(fsub(x[j], c.m), sm.exp_tab);
                if (o < nv) l.out_full[(size_t)row * V + r * W_REGION + o] = fsub(__double2float_rn(log((double)e)), log_sum);
            }
            continue;
        }
        Terms f;
        f.m = c.m; f.t = c.t; f.S = PHASE == WP_SUM ? -1.0f : c.S; f.filter = false; f.p_thr = 0.0f; f.id_thr = 0u;
        if (PHASE == WP_TOTAL) f = kept_terms(c, V);
        wload<BF16, VEC>(x, c.rowp, r, nv);
        uint2* seg = l.seg + (size_t)slot * l.reg_stride + r;
        uint2 out = make_uint2(0u, PHASE == WP_LIST ? 0u : __ldcg(&seg->y));
        wprocess<BF16, VEC>(buf, x, l, slot, c.mw, c.entries, r, nv);
        if (PHASE == WP_SUM) {
            const float cut = c.cut_x;
#pragma unroll
            for (int j = 0; j < WL; j++)
                if (x[j] >= cut) {   // (rare)
                    const uint32_t at = atomicAdd(&l.row[slot].n_list, 1u);
                    if (at == (uint32_t)F_MCAP) atomicAdd(l.sync + 2, 1u);   // too many: the row selects by the histogram
                    if (at < min((uint32_t)F_MCAP, l.list_stride)) l.list[(size_t)slot * l.list_stride + at] = ((unsigned long long)f2u(x[j]) << 32) | (r * W_REGION + L::off(lane, j));
                }
        }
        if (PHASE == WP_SUM || PHASE == WP_TOTAL) {
            if (PHASE == WP_TOTAL && !f.filter && a.n_kept) {   // every probability above zero is kept
                const float c1 = 1.44269504f / f.t, c0 = f.S > 1e-9f ? -log2f(f.S) : 0.0f;
                uint32_t n = 0u;
#pragma unroll
                for (int j = 0; j < WL; j++) {
                    const float e = __fmaf_rn(fsub(x[j], f.m), c1, c0);   // (a probability below 2^-149 is zero)
                    n += e > -120.0f || (x[j] > -INFINITY && e > -160.0f && term_of(x[j], 0u, f, sm.exp_tab) > 0.0f);
                }
                n = __reduce_add_sync(FULL, n);
                if (lane == 0 && n) atomicAdd(&l.row[slot].n_kept, n);
            }
            const uint32_t kb = out.y & ~W_DUAL;
            if (kb) {
                const Approx q = approx_of(f);
                out.x = increments<BF16, VEC>(x, r * W_REGION, f, q, kb, sm.exp_tab);
                uint32_t n1 = 0u;
                if (out.x != W_TIE && (out.y & W_DUAL)) n1 = increments<BF16, VEC>(x, r * W_REGION, f, q, kb + 0x00800000u, sm.exp_tab);
                if (out.x == W_TIE || n1 == W_TIE) out.y = 0u;
                else if ((out.y & W_DUAL) && lane == 0) l.pre[(size_t)slot * l.reg_stride + r] = u2f(n1);
            }
            if (out.y == 0u) {   // to be added term by term: the terms are left in id order, as far as there is room
                // (a loop over the staged logits: sixteen copies of the exponential's code, which few regions run through, take
                // longer to fetch than to execute)
                float top = x[0];
#pragma unroll
                for (int j = 1; j < WL; j++) top = fmaxf(top, x[j]);
                bool zeros = true;
                if (__any_sync(FULL, top > -INFINITY)) {
                    uint32_t at = 0u;
                    if (lane == 0) at = atomicAdd(&l.row[slot].n_terms, 1u);
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < WL; j++) buf[L::off(lane, j)] = x[j];
                    __syncwarp();
#pragma unroll 4
                    for (uint32_t o = lane; o < (uint32_t)W_REGION; o += 32u) {
                        const float t = term_of(buf[o], r * W_REGION + o, f, sm.exp_tab);
                        zeros &= t == 0.0f;
                        buf[o] = t;
                    }
                    out.x = __shfl_sync(FULL, at, 0) + 1u;
                }
                if (__all_sync(FULL, zeros)) out = make_uint2(0u, 1u);   // nothing but zeros
                else if (out.x > (uint32_t)W_TERMS) out.x = 0u;
                else {
                    float* t = l.terms + ((size_t)slot * W_TERMS + out.x - 1u) * W_REGION;
#pragma unroll
                    for (int j = 0; j < WL; j++) t[j * 32 + lane] = buf[j * 32 + lane];   // (each lane its own)
                }
                __syncwarp();   // (the next region's entries are staged there by other lanes)
            }
            if (lane == 0) *seg = out;
        } else {   // WP_LIST
            const uint32_t cut = c.cut & 0x7fffffffu;
            // the exact probability only of those that may lie in one of the buckets
            const Approx q = approx_of(f);
            const float from = cut ? bucket_floor(cut) * (1.0f - (4.0f * fabsf(q.k0) + 200.0f) * 2.4e-7f) : 0.0f;
            uint32_t may = 0u;
#pragma unroll
            for (int j = 0; j < WL; j++)
                if (x[j] > -INFINITY && ex2_approx_ftz(__fmaf_rn(fsub(x[j], f.m), q.c, q.k0)) >= from) may |= 1u << j;
            while (may) {
                const uint32_t j = __ffs((int)may) - 1u;
                may &= may - 1u;
                float p = x[0];
#pragma unroll
                for (int u = 1; u < WL; u++) if ((uint32_t)u == j) p = x[u];
                p = term_of(p, 0u, f, sm.exp_tab);
                const uint32_t b = bucket_of(p);
                if (p > 0.0f && b >= cut) {
                    const uint32_t at = atomicAdd(l.hist + (size_t)slot * W_BUCKETS + b, 1u);
                    l.list[(size_t)slot * l.list_stride + at] = ((unsigned long long)f2u(p) << 32) | (r * W_REGION + L::off(lane, j));
                }
            }
        }
    }
    return true;
}

// Histogram of the probabilities of the rows that select by them.  Every CTA takes an equal run of the rows' regions, so
// that most counting happens in shared memory and the buckets are flushed once or twice.
template <bool BF16, bool VEC>
__device__ __noinline__ void hist_phase(uint32_t n_rows) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x, w = tid >> 5, V = a.vocab, n_regions = (V + W_REGION - 1) / W_REGION;
    rows_in(sm, l, n_rows);
    uint32_t n_sel = 0u;
    for (uint32_t s = 0; s < n_rows; s++) n_sel += sm.rows[s].state == WS_SELECT;
    const uint32_t per = (n_sel * n_regions + sm.size - 1u) / sm.size, lo = min(sm.rank * per, n_sel * n_regions), hi = min(lo + per, n_sel * n_regions);
    for (uint32_t b = tid; b < (uint32_t)W_BUCKETS; b += W_NT) sm.bn[b] = 0u;
    uint32_t first = 0u;   // of the row's regions, among all
    for (uint32_t slot = 0; slot < n_rows; slot++) {   // CTA-uniform
        const WideRow& c = sm.rows[slot];
        if (c.state != WS_SELECT) continue;
        const uint32_t r0 = max(lo, first) - first, r1 = min(hi, first + n_regions) > first ? min(hi, first + n_regions) - first : 0u;
        first += n_regions;
        if (r0 >= r1) continue;
        __syncthreads();
        Terms f;
        f.m = c.m; f.t = c.t; f.S = c.S; f.filter = false; f.p_thr = 0.0f; f.id_thr = 0u;
        const Approx q = approx_of(f);
        const float eps = (4.0f * fabsf(q.k0) + 200.0f) * 2.4e-7f;   // (probabilities from 2^-40 on count)
        const uint32_t low = lowest_bucket(c, V);
        const float low_p = low ? bucket_floor(low) * (1.0f - 2.0f * eps) : -1.0f;
        for (uint32_t r = r0 + w; r < r1; r += WNW) {
            const uint32_t nv = min(V - r * W_REGION, (uint32_t)W_REGION);
            float x[WL];
            wload<BF16, VEC>(x, c.rowp, r, nv);
            wprocess<BF16, VEC>(sm.stage[w], x, l, slot, c.mw, c.entries, r, nv);
            // the hardware's exp2 decides the bucket, unless the probability lies close to a border
#pragma unroll
            for (int j = 0; j < WL; j++) {
                float p = ex2_approx_ftz(__fmaf_rn(fsub(x[j], f.m), q.c, q.k0));
                if (p < low_p) continue;
                if (x[j] > -INFINITY && (bucket_of(p * (1.0f - eps)) != bucket_of(p * (1.0f + eps)) || p < 1e-30f)) p = term_of(x[j], 0u, f, sm.exp_tab);
                const uint32_t b = bucket_of(p);
                if (p > 0.0f && b >= low) atomicAdd(&sm.bn[b], 1u);
            }
        }
        __syncthreads();
        for (uint32_t b = tid; b < (uint32_t)W_BUCKETS; b += W_NT)
            if (sm.bn[b]) { atomicAdd(l.hist + (size_t)slot * W_BUCKETS + b, sm.bn[b]); sm.bn[b] = 0u; }
    }
}

// `n` rows (of the list, or of the batch) one CTA each, by the general kernel's code on `slots` scratch slots
__device__ __noinline__ void rows_one_cta_each(uint32_t rank, uint32_t slots, uint32_t n, const uint32_t* rows) {
    WideSmem& sm = wide_smem();
    if (n == 0u || rank >= slots) return;
    __syncthreads();
    if (threadIdx.x < 32u) sm.general.exp_tab[threadIdx.x] = kExp2TableDev[threadIdx.x];
    __syncthreads();
    general_rows(sm.a, sm.general, rank, slots, n, rows);
}

// Whether the batch is done by one CTA per row; it is when this returns true.  (A general kernel for the same rows in front is
// waited for only here: what the rows ask for stands already.  A function of its own, as the usual launch would fetch the code.)
__device__ __noinline__ bool look(uint32_t n_work, uint32_t slots) {
    WideSmem& sm = wide_smem();
    const WideLaunch& l = sm.l;
    if (threadIdx.x == 0) sm.found = 0u;
    __syncthreads();
    batch_kinds(sm.a, n_work, W_NT, &sm.found);
    __syncthreads();
    const bool front = l.kinds_front != 0u;
    const bool few = l.local && sm.a.work_rows;   // (one or two listed rows, see below)
    const bool per_row = ((front ? l.kinds_front : l.kinds_row[few ? 1u + n_work : n_work > l.chunk ? 1u : 0u]) >> sm.found) & 1u;
    if (front) cudaGridDependencySynchronize();
    else if (per_row) rows_one_cta_each(blockIdx.x, min(slots, gridDim.x), n_work, sm.a.work_rows);
    return per_row;
}

// A barrier was given up: the last rows of the launch, and those still to be done by the general kernel's code, end with a
// status that says so.  One thread.
__device__ __noinline__ void give_up(const RowArgs& a, const WideLaunch& l, uint32_t n_work) {
    uint32_t n = 0u;
    const auto end = [&](uint32_t row) {
        n++;
        if (!l.score) { wresult_plain(a, row, ROW_LOAD_TIMEOUT, 0u, -INFINITY); return; }
        if (a.status) a.status[row] = ROW_LOAD_TIMEOUT;
        if (l.out_gather) l.out_gather[row] = NAN;
    };
    for (uint32_t i = n_work - __ldcg(l.sync + 1); i < n_work; i++) end(a.work_rows ? a.work_rows[i] : i);
    const uint32_t n_left = l.score ? 0u : __ldcg(l.left_count);
    for (uint32_t i = 0; i < n_left; i++) {
        const uint32_t row = __ldcg(l.left_rows + i);
        if (__ldcg(a.status + row) != ROW_LOAD_TIMEOUT) end(row);
    }
    atomicAdd(l.gave_up, (unsigned long long)n);
    l.sync[1] = 0u;
}

template <bool BF16, bool VEC>
__global__ void __launch_bounds__(W_NT, 1) wide_kernel(const RowArgs a_, const WideLaunch l_, uint32_t slots) {
    WideSmem& sm = wide_smem();
    const RowArgs& a = sm.a;
    const WideLaunch& l = sm.l;
    const uint32_t tid = threadIdx.x;
    // Launched ahead of the end of the kernel before, which may fill the list.  (No early trigger for the kernel behind: its
    // CTAs would crowd on the SMs that this one leaves free, two on an SM while others have none, or those with two rows
    // together.  us without / with it: 128 masked rows 50 / 62, 149 rows of 151936 66.4 / 69.1, 149 mixed bf16 rows of 256000 129 / 147,
    // 300 rows of 50256 with 512 ids 58 / 70; 192 to 296 rows within 2 % either way.)
    if (!l_.kinds_front) cudaGridDependencySynchronize();
    const uint32_t n_work = a_.work_rows ? *(volatile uint32_t*)a_.work_count : a_.rows;
    if (n_work == 0u) return;   // the usual case of the work-list pass
    // (how many rows are listed is known here only)
    const bool local = l_.local == 1u || (l_.local == 2u && listed_one_cta_each(n_work, l_.chunk, slots, a_.vocab));
    if (tid == 0) { sm.a = a_; sm.target = 0u; sm.gave_up = 0u; }
    if (tid == 32u) {
        sm.l = l_;
        sm.l.local = local ? 1u : 0u;   // (what the barriers go by)
        if (local) {   // this CTA's part of the workspace
            WideLaunch& o = sm.l;
            const size_t at = blockIdx.x;
            o.row += at; o.reg += at * o.reg_stride; o.cell += at * o.reg_stride; o.seg += at * o.reg_stride; o.pre += at * o.reg_stride;
            o.terms += at * W_TERMS * W_REGION; o.ent_id += at * (W_MAX_HIST + 32); o.ent_xn += at * (W_MAX_HIST + 32); o.rs += at * o.rs_stride;
            o.hist += at * W_BUCKETS; o.list += at * o.list_stride;
            o.sync = o.own + at * W_OWN; o.left_count = o.sync + 8; o.left_rows = o.sync + 9;
        }
    }
    if (local && tid == 0) { sm.rank = 0u; sm.size = 1u; sm.target = 1u; }
    if (tid < 32u) sm.exp_tab[tid] = kExp2TableDev[tid];
    __syncthreads();
    bool ok = true;   // (false for all CTAs, or none)
    if (local && l_.local == 2u ? (l_.look & 2u) && n_work <= 2u : (l_.look & 1u)) {
        ok = !look(n_work, slots);
        if (!ok && l_.kinds_front) return;
    }
    ok = ok && (local || grid_join(sm, l));
    uint32_t n_left = 0u;   // rows left to the general kernel's code
    const auto leave_one = [&]() {   // the CTA's own list has one entry; the scratch slot is the CTA's too
        rows_one_cta_each(blockIdx.x, gridDim.x, blockIdx.x + 1u, l.left_rows - blockIdx.x);
        __syncthreads();
        if (tid == 0) *l.left_count = 0u;
    };
    for (uint32_t c0 = local ? blockIdx.x : 0u; c0 < n_work && ok; c0 += local ? gridDim.x : l.chunk) {
        const uint32_t n = local ? 1u : min(n_work - c0, l.chunk), to_do = n_work - c0;
        const auto open = [&](uint32_t s) { open_row<BF16>(s, a.work_rows ? a.work_rows[c0 + s] : c0 + s); };
        if (sm.rank == 0u && tid == 0) { l.sync[2] = 0u; l.sync[3] = 0u; }
        uint32_t s = sm.rank;
        if (c0 == 0u) { if (s < n) open(s); }   // (how many take part is not known yet)
        else for (; s < n; s += sm.size) open(s);
        if (local && sm.row.state == WS_DONE) {   // CTA-uniform: bad parameters, or left to the general kernel's code
            __syncthreads();
            if (*(volatile uint32_t*)l.left_count) leave_one();
            continue;
        }
        if (!(ok = region_phase<BF16, VEC, WP_FIRST>(n, c0, to_do))) break;
        if (c0 == 0u && sm.size < n) {   // not one CTA for every row
            for (s += sm.size; s < n; s += sm.size) open(s);
            if (!(ok = region_phase<BF16, VEC, WP_FIRST>(n, c0, to_do))) break;
        }
        if (!(ok = grid_sync(sm, l, to_do))) break;
        for (uint32_t s = sm.rank; s < n; s += sm.size) maximum_row<BF16, VEC>(s);
        if (!(ok = region_phase<BF16, VEC, WP_SUM>(n, c0, to_do))) break;
        if (!(ok = grid_sync(sm, l, to_do))) break;
        for (uint32_t s = sm.rank; s < n; s += sm.size) sum_row<BF16, VEC>(s);
        // Which phases are still to come is known to all CTAs alike (nothing has been counted since the barrier), and what follows
        // the last of them needs no barrier.
        if (l.score) {
            if (l.out_full && !(ok = region_phase<BF16, VEC, WP_FULL>(n, c0, to_do))) break;
        } else {
            uint32_t totals = *(volatile uint32_t*)(l.sync + 3);
            n_left = *(volatile uint32_t*)l.left_count;
            if (*(volatile uint32_t*)(l.sync + 2)) {
                if (!(ok = grid_sync(sm, l, to_do))) break;
                hist_phase<BF16, VEC>(n);
                if (!(ok = grid_sync(sm, l, to_do))) break;
                for (uint32_t s = sm.rank; s < n; s += sm.size) select_row(s);
                if (!(ok = region_phase<BF16, VEC, WP_LIST>(n, c0, to_do))) break;
                if (!(ok = grid_sync(sm, l, to_do))) break;
                for (uint32_t s = sm.rank; s < n; s += sm.size) choose_row(s);
                if (!(ok = grid_sync(sm, l, to_do))) break;
                totals = *(volatile uint32_t*)(l.sync + 3);
                n_left = *(volatile uint32_t*)l.left_count;
            }
            if (totals) {
                if (!(ok = region_phase<BF16, VEC, WP_TOTAL>(n, c0, to_do))) break;
                if (!(ok = grid_sync(sm, l, to_do))) break;
                for (uint32_t s = sm.rank; s < n; s += sm.size) total_row<BF16, VEC>(s);
            }
        }
        if ((to_do > n || n_left) && !(ok = grid_sync(sm, l, to_do))) break;   // the chunk's workspace is free
        if (local && n_left) { leave_one(); n_left = 0u; }
    }
    if (local && !a.work_rows && !l.done) return;
    if (ok && n_left) rows_one_cta_each(sm.rank, min(slots, sm.size), n_left, l.left_rows);
    // The last CTA of the grid to leave resets the counters and empties the lists; the upper half counts the CTAs that gave up.
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const uint32_t before = atomicAdd(l_.sync + 4, sm.gave_up ? 0x10001u : 1u);
        if ((before & 0xffffu) == gridDim.x - 1u) {
            if ((before >> 16) || sm.gave_up) { __threadfence(); give_up(a, l, n_work); }
            l_.sync[0] = 0u; l_.sync[4] = 0u; l_.sync[5] = 0u; l_.sync[6] = 0u;
            *l_.left_count = 0u;
            if (a.work_rows) *a.work_count = 0u;
            if (l.done) { __threadfence(); *(volatile uint32_t*)l.done = l.done_value; }   // (the next launch starts behind this)
        }
    }
}

template <bool BF16, bool VEC>
static cudaError_t wide_configure_one() {
    return cudaFuncSetAttribute(wide_kernel<BF16, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WideSmem));
}

cudaError_t configure_wide() {
    cudaError_t e = wide_configure_one<false, true>();
    if (e == cudaSuccess) e = wide_configure_one<true, true>();
    if (e == cudaSuccess) e = wide_configure_one<false, false>();
    if (e == cudaSuccess) e = wide_configure_one<true, false>();
    return e;
}

// `grid` CTAs, at most one per SM; set up while the kernel before still runs (programmatic stream serialization)
cudaError_t launch_wide(const RowArgs& a, const WideLaunch& l, uint32_t slots, uint32_t grid, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(W_NT, 1, 1);
    cfg.dynamicSmemBytes = sizeof(WideSmem);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const uint32_t ge = a.dtype ? 8u : 4u;
    const bool vec = ((uintptr_t)a.logits & 15u) == 0u && a.row_stride % ge == 0u && a.vocab % ge == 0u;
    if (vec) return a.dtype ? cudaLaunchKernelEx(&cfg, wide_kernel<true, true>, a, l, slots) : cudaLaunchKernelEx(&cfg, wide_kernel<false, true>, a, l, slots);
    return a.dtype ? cudaLaunchKernelEx(&cfg, wide_kernel<true, false>, a, l, slots) : cudaLaunchKernelEx(&cfg, wide_kernel<false, false>, a, l, slots);
}

}  // namespace pgs
