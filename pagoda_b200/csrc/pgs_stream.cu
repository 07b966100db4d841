// Streaming row kernel: the hot path of the sampler.
//
// One CTA of 512 threads (two per SM) owns one batch row at a time and reads it twice with plain 128-bit
// coalesced loads, sixteen logits per thread and piece.  Inside a pass nothing synchronises the warps, so the
// loads of some overlap the arithmetic of the others, and what a piece costs beyond its logits (addresses, table
// look-ups, warp reductions, loop control) is paid once per sixteen logits:
//
//   before: the row's entries (distinct history ids, the EOS fix) and one bit per logit that says whether the passes may see
//           it (the grammar mask without the entries; of rows beyond 2^18 logits the passes make them, region by region); the
//           entries' logits are copied aside during pass 1 and one thread per entry adds what the penalties make of them to
//           what the passes find;
//   pass 1, last piece first, from HBM: sanity, bits; per thread its running
//           maximum and four more (one per piece number mod 4) that bound the top-k threshold; per warp and piece the
//           plain sum of the softmax numerators relative to the warp's own maximum;
//   between: row maximum and argmax (lowest id: the threads that hold the maximum look at that piece again); a bound for the top-k threshold: the k-th largest of the 2048
//           per-thread maxima is reached by at least k logits, so "logit >= that bound" is a superset of the
//           top-k set that is only slightly larger; and, from the rescaled plain sums, the value the reference's
//           running sum has when it reaches each warp's 512 logits of each piece, to within 1e-3;
//   pass 2, first piece first, from L2 (the pieces read last in pass 1 are the freshest there): the same
//           processed logits again, candidates above the bound, softmax numerators by the hardware exp2, and
//           the reference's sequential f32 sum;
//   finish: exact probabilities of the candidates, top-k with ties, top-p walk, inverse-CDF pick.
//
// A row is 600 KB, more than one SM holds, and its maximum must be known before the first numerator: the row
// is therefore read a second time.  What the second pass finds in L2 is what the first pass read last, which is
// why the passes run in opposite directions; with a whole batch in flight that is about a third of the row.
// The loops have no registers for a second piece in flight, so every warp asks for the piece it will read two
// iterations later with an L2 prefetch.  An optional gate (a counter of rows that finished pass 1, bounded
// polling, off unless the launch asks for a cohort) can hold rows back so that fewer are in their first pass at
// once.
//
// Small batches: when all rows fit as resident clusters, a thread-block cluster of 4 or 8 CTAs shares every row
// (see stream_row_kernel below): a row alone on one CTA is bound by the latency of its own instructions.
//
// The f32 left fold (pagoda/src/sampler.rs:99-113): while the running value stays inside one binade, adding a
// non-negative term is an integer addition in units of that binade's ulp which depends on the running value only
// through its parity.  Wherever the estimate above puts the running value safely inside one binade for a warp's
// whole share of a piece, every thread adds its sixteen numerators to that binade's lower end (real f32
// additions) and the increments are summed as integers; the few shares in which the running value may change
// binade are folded 128 bits at a time from their own estimates of the running value, which reproduces the
// crossing.  Ties of round-half-even are decided by the parity of a stand-in, not of the true running value: the
// sum agrees with the reference's to about 1e-6 relative, and a decision can differ only when it sits that close
// to its boundary.
//
// Fidelity of this path: argmax, masks, penalties and candidate sets follow the reference bit for bit
// (pagoda/src/engine.rs:1286-1314, pagoda/src/sampler.rs:28-150); candidate numerators use the exact expf.
// Rows this kernel does not serve (top-k off or > 1024, more candidates than its buffers, histories beyond its
// id -> count table, rows that are not 16-byte aligned) are appended to a work list for the wide kernel.
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "pgs_args.cuh"
#include "pgs_block.cuh"
#include "pgs_finish.cuh"
#include "pgs_stream.cuh"

namespace pgs {

constexpr int SNT = 512;                 // threads per CTA
constexpr int SNW = SNT / 32;            // warps per CTA
constexpr int S_EPT = 16;                // logits per thread and piece
constexpr int S_PIECE = SNT * S_EPT;     // logits per piece
constexpr int S_REGION = 32 * S_EPT;     // consecutive logits of one warp in a piece
constexpr int S_NCELL = 4;               // running maxima per thread (piece number mod S_NCELL)
constexpr int S_CELLS = S_NCELL * SNT;   // per-thread maxima that bound the top-k threshold
constexpr int S_NB = 1024;               // buckets of their histogram
constexpr int S_BPT = S_NB / SNT;        // buckets per thread
constexpr int S_ENT = S_MAX_HASH / 2 + 1;   // distinct history ids, and the EOS fix
constexpr uint32_t S_NIL = 0xffffffffu;
constexpr uint32_t ENT_MASKED = 0x80000000u, ENT_EOS = 0x40000000u;   // beside an entry's count
static_assert(SNW <= 32, "warp slots are combined by one warp");

// Everything the kernel needs to know about a row, read and validated by one thread while the CTA still works
// on the row before it.
struct SRowCtl {
    const char* rowp;       // first logit of the row
    const uint32_t* mw;     // grammar mask words of the row's state, or null
    float temp, freq, pres, rep, top_p, u01;
    float sc, sc_lo;        // log2(e) / max(temp, 1e-9) as a two-float sum
    uint32_t top_k, gflags, h0, nh;
    uint32_t kind;          // 0 serve, 1 bad parameters, 2 leave to the work list
};

// What the pass loops need to know about the row they work on.
enum : uint32_t { PF_REP = 1u, PF_FP = 2u, PF_PRES = 4u };
struct PassArgs {
    const char* rowp;
    const uint32_t* mw;     // rows beyond S_SHORT_VOCAB: the grammar mask
    float sc, sc_lo, c_hi, c_lo, cut_f, freq, pres, rep;
    uint32_t V, n_full, n_regions, flags;
    // a row shared by the CTAs of a cluster: this CTA works on the pieces q0, q0 + qstep, ...; the candidates of all of
    // them are collected by the first CTA (pointers into its shared memory)
    uint32_t q0, qstep;
    uint32_t* cand_n_p;
    uint32_t* cand_id_p;
    float* cand_x_p;
    uint32_t few;           // pass 2 meets few candidates (see few_candidates)
};

// LONG: rows beyond S_SHORT_VOCAB, whose bits do not fit beside two CTAs' tables.
template <bool LONG>
struct StreamSmem {
    static constexpr bool IS_LONG = LONG;
    static constexpr int MAX_REGIONS = (LONG ? S_MAX_VOCAB : S_SHORT_VOCAB) / S_REGION;
    SRowCtl ctl[2];
    PassArgs pa;
    unsigned long long exp_tab[32];
    uint32_t red_key[SNW], red_lo[SNW], red_fin[SNW], red_flag[SNW];
    uint32_t scan_u[SNW];
    float scan_f[SNW];
    double wacc[SNW];               // per-warp share of the fold
    uint32_t cand_n, sel_bucket, amax;
    // cluster mode: one slot per CTA of the cluster, written by that CTA into every CTA's copy (xk .. xflag) or into
    // the first CTA's copy (xs, xam)
    uint32_t xk[8], xlo[8], xfin[8], xflag[8], xam[8];
    float xb[8];
    double xs[8];
    long long prof_acc[16];
    alignas(16) float4 bit_tab[16];     // bf16 rows: what four bits add to the logits they belong to, 0 or -inf
    // Three lives of one area: the id -> count table while the entries are set up, the tables of a row while it streams, and
    // the arrays of the finish once its candidates are known (nothing of the tables is needed by then).
    union alignas(16) {
        struct {
            uint32_t cand_id[F_MCAP];
            float cand_x[F_MCAP];
            union {
                struct {
                    uint32_t hist[S_NB];
                    float cell[S_CELLS];             // [S_NCELL][SNT]
                    float t_am[SNT], t_max[SNT];   // per-thread results of pass 1 over the whole pieces
                    uint32_t t_q[SNT];
                    // per warp region of the row (512 consecutive logits): pass 1 leaves the warp's maximum and the plain
                    // sum of its numerators relative to it; then the binade's lower end the fold has there (0 = fold this
                    // region the careful way) and the estimate of the running value at its start
                    float reg_a[MAX_REGIONS], reg_b[MAX_REGIONS];
                    // a logit below this adds exactly nothing to the fold in this region; before, the plain sum of the
                    // region's entries relative to the CTA's maximum
                    float reg_t[MAX_REGIONS];
                    // The row's entries: the distinct history ids and the EOS fix, those of region r at rs[r] .. rs[r + 1].
                    // The passes leave their logits out (the bits are clear); pass 1 copies them to ent_raw, and one thread
                    // per entry adds what the chain sees there to what the passes find.
                    uint16_t rs[MAX_REGIONS + 2];
                    uint32_t ent_id[S_ENT];
                    float ent_x[S_ENT];              // before pass 1 is over: the count; ENT_MASKED, ENT_EOS
                    uint32_t ent_raw[S_ENT];         // the word that holds the raw logit (before pass 1: entries per region)
                    uint32_t bits[LONG ? 1 : S_SHORT_VOCAB / 32];   // one bit per logit: allowed, and no entry
                };
                FinishArrays fin;
                unsigned long long tpkey[SNT];   // vocabulary-sharded mode: one candidate per thread while a record is ranked
            };
        };
        uint32_t hash[2 * S_MAX_HASH];           // hkey[H], hcnt[H]: ends before reg_a
    };
};

static_assert(sizeof(StreamSmem<false>) <= 113 * 1024 && sizeof(StreamSmem<true>) <= 113 * 1024, "two CTAs per SM");
static_assert(offsetof(StreamSmem<false>, hash) + sizeof(StreamSmem<false>::hash) <= offsetof(StreamSmem<false>, reg_a) &&
              offsetof(StreamSmem<true>, hash) + sizeof(StreamSmem<true>::hash) <= offsetof(StreamSmem<true>, reg_a), "entries are set up while the table stands");

#define PGS_STICK(slot)                                             \
    do {                                                            \
        if (sl.prof && tid == 0) {                                  \
            const long long now_ = clock64();                       \
            sm.prof_acc[slot] += now_ - tick_;                      \
            tick_ = now_;                                           \
        }                                                           \
    } while (0)

__device__ __forceinline__ float max_ept(const float (&x)[S_EPT]) {
    static_assert(S_EPT % 8 == 0, "eight logits per round");
    float m[S_EPT / 8];
#pragma unroll
    for (int j = 0; j < S_EPT; j += 8)
        m[j / 8] = max3f(max3f(x[j], x[j + 1], x[j + 2]), max3f(x[j + 3], x[j + 4], x[j + 5]), fmaxf(x[j + 6], x[j + 7]));
    float r = m[0];
#pragma unroll
    for (int j = 1; j + 1 < S_EPT / 8; j += 2) r = max3f(r, m[j], m[j + 1]);
    if ((S_EPT / 8) % 2 == 0) r = fmaxf(r, m[S_EPT / 8 - 1]);
    return r;
}
__device__ __forceinline__ float absmax_ept_nan(float am, const float (&x)[S_EPT]) {
    float m[S_EPT / 8];
#pragma unroll
    for (int j = 0; j < S_EPT; j += 8)
        m[j / 8] = absmax3_nan(absmax3_nan(x[j], x[j + 1], x[j + 2]), absmax3_nan(x[j + 3], x[j + 4], x[j + 5]), absmax3_nan(x[j + 6], x[j + 7], x[j + 7]));
#pragma unroll
    for (int j = 0; j + 1 < S_EPT / 8; j += 2) am = absmax3_nan(am, m[j], m[j + 1]);
    if ((S_EPT / 8) % 2 == 1) am = absmax3_nan(am, m[S_EPT / 8 - 1], m[S_EPT / 8 - 1]);
    return am;
}

// One piece's share of a thread as it comes from memory: f32 rows eight 128-bit groups of four logits, bf16 rows
// four groups of eight.
template <bool BF16> struct Geo {
    static constexpr int G = BF16 ? S_EPT / 8 : S_EPT / 4;   // groups per thread and piece
    static constexpr int GE = S_EPT / G;        // logits per group
    static constexpr int GS = 32 * GE;          // logits between two groups of a thread
};

// id of the thread's j-th logit of a piece whose first group starts at e0
template <bool BF16> __device__ __forceinline__ uint32_t elem_id(uint32_t e0, int j) {
    return e0 + (uint32_t)(j / Geo<BF16>::GE) * Geo<BF16>::GS + (uint32_t)(j % Geo<BF16>::GE);
}

// ---- CTA-wide exclusive scans for SNW warps (one barrier each; `slots` may be written again after another barrier)
__device__ __forceinline__ uint32_t sblock_excl_scan_u32(uint32_t v, uint32_t* total, uint32_t* slots) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) slots[w] = inc;
    __syncthreads();
    const uint32_t x = lane < SNW ? slots[lane] : 0u;
    *total = __reduce_add_sync(FULL, x);
    return __reduce_add_sync(FULL, lane < w ? x : 0u) + inc - v;
}
__device__ __forceinline__ float sblock_excl_scan_f32(float v, float* total, float* slots) {   // plain adds: estimates only
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) slots[w] = inc;
    __syncthreads();
    const float x = lane < SNW ? slots[lane] : 0.0f;
    float xi = x;
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(FULL, xi, o);
        if (lane >= o) xi += t;
    }
    *total = __shfl_sync(FULL, xi, 31);
    return __shfl_sync(FULL, xi - x, w) + (inc - v);
}

// One thread reads and validates a row's parameters (same rules as the general kernel).
template <bool BF16>
__device__ __forceinline__ void sprepare_row(const RowArgs& a, const StreamLaunch& sl, uint32_t row, SRowCtl& c) {
    const uint32_t V = a.vocab;
    const float temp = a.temperature ? a.temperature[row] : 0.0f;
    // (vocabulary-sharded mode: the record's length takes the place of top-k; top-p and the draw belong to the merge)
    const uint32_t top_k = a.tp_records ? a.tp_cand : a.top_k ? a.top_k[row] : 0u;
    const float top_p = a.top_p ? a.top_p[row] : 1.0f;
    const float freq = a.freq ? a.freq[row] : 0.0f;
    const float pres = a.pres ? a.pres[row] : 0.0f;
    const float rep = a.rep ? a.rep[row] : 1.0f;
    const float u01 = a.uniform ? a.uniform[row] : 0.0f;
    bool bad = !finite_f(temp) || !finite_f(top_p) || !finite_f(freq) || !finite_f(pres) ||
               !finite_f(rep) || !(rep > 0.0f) || !finite_f(u01);
    const uint32_t* mw = nullptr;
    uint32_t gflags = 0;
    if (a.mask_table && a.mask_table[row] >= 0) {
        const int32_t t = a.mask_table[row];
        const int32_t st = a.mask_state ? a.mask_state[row] : 0;
        if (t >= MAX_TABLES || !a.tables[t].live || st < 0 || (uint32_t)st >= a.tables[t].n_states ||
            (unsigned long long)a.tables[t].words_per_state * 32ull < V) {
            bad = true;
        } else {
            mw = a.tables[t].words + (size_t)st * a.tables[t].words_per_state;
            gflags = a.tables[t].flags[st];
        }
    }
    uint32_t h0 = 0, nh = 0;
    if (a.hist_offsets) {
        h0 = a.hist_offsets[row];
        const uint32_t h1 = a.hist_offsets[row + 1];
        if (h1 < h0 || h1 - h0 > a.max_history || (h1 > h0 && !a.hist_ids)) bad = true; else nh = h1 - h0;
    }
    const bool greedy = temp < 1e-5f;
    const bool use_k = top_k != 0u && top_k < V;
    const char* rowp = (const char*)a.logits + (size_t)row * a.row_stride * (BF16 ? 2 : 4);
    const bool aligned = (((uintptr_t)rowp & 15) == 0) && (V % Geo<BF16>::GE) == 0;
    const bool pen = nh > 0 && (!(fabsf(freq) < 1e-6f && fabsf(pres) < 1e-6f) || rep != 1.0f);
    const bool defer = !aligned || (!greedy && (!use_k || top_k > (uint32_t)S_KMAX)) || (pen && 2u * nh > sl.hash_slots);
    c.rowp = rowp; c.mw = mw; c.temp = temp; c.freq = freq; c.pres = pres; c.rep = rep; c.top_p = top_p; c.u01 = u01;
    const double scale_d = 1.4426950408889634 / (double)fmaxf(temp, 1e-9f);
    // rounded down, so that the second float is positive and a masked entry (-inf) stays -inf through both products
    float sc_hi = (float)scale_d;
    if ((double)sc_hi >= scale_d) sc_hi = u2f(f2u(sc_hi) - 1u);
    c.sc = sc_hi;
    c.sc_lo = (float)(scale_d - (double)sc_hi);
    c.top_k = top_k; c.gflags = gflags; c.h0 = h0; c.nh = nh;
    c.kind = bad ? 1u : defer ? 2u : 0u;
}

// Vocabulary-sharded mode: the candidates of one row (n <= SNT, one per thread) -> this shard's record: the
// tp_cand largest by (logit descending, id ascending) behind the head.  Called by every thread; the caller has a
// barrier in front.
template <class SM>
__device__ __forceinline__ void semit_tp(SM& sm, const RowArgs& a, uint32_t row, uint32_t n, float m, float S,
                                         uint32_t amax) {
    const int tid = threadIdx.x;
    TpRecHead* head = reinterpret_cast<TpRecHead*>(a.tp_records + (size_t)row * a.tp_rec_bytes);
    float* rx = reinterpret_cast<float*>(head + 1);
    uint32_t* rid = reinterpret_cast<uint32_t*>(rx + a.tp_cand);
    const uint32_t want = a.tp_cand < n ? a.tp_cand : n;
    if ((uint32_t)tid < n)
        sm.tpkey[tid] = ((unsigned long long)order_key(sm.cand_x[tid]) << 32) | (unsigned long long)(0xffffffffu - sm.cand_id[tid]);
    __syncthreads();
    if ((uint32_t)tid < n) {
        const unsigned long long kj = sm.tpkey[tid];
        uint32_t r = 0;
#pragma unroll 8
        for (uint32_t o = 0; o < n; o++) r += sm.tpkey[o] > kj;
        if (r < want) { rx[r] = sm.cand_x[tid]; rid[r] = a.id_base + sm.cand_id[tid]; }
    }
    if (tid == 0) tp_write_head(a, row, m, S, want, ROW_OK, amax);
}

// ------------------------------------------------------------------------------------------------------------
// The two passes.  Their loops over the whole pieces of a row are functions of their own (not inlined), so that
// the registers of each loop are allocated for that loop alone (sixteen logits and a dozen values of state: no
// spills in the loops).  What they need to know about the row is in shared
// memory (PassArgs); the ragged last piece of a row, if any, is handled by the caller with the same piece code.

template <bool BF16> struct Raw;
template <> struct Raw<false> { float4 v[4]; };
template <> struct Raw<true> { uint4 v[2]; };

// a whole piece: no bounds checks
template <bool BF16>
__device__ __forceinline__ void raw_load(Raw<BF16>& r, const char* p) {
    constexpr int G = Geo<BF16>::G, STEP = Geo<BF16>::GS * (BF16 ? 2 : 4);
#pragma unroll
    for (int h = 0; h < G; h++) {
        if constexpr (BF16) r.v[h] = __ldcg(reinterpret_cast<const uint4*>(p + h * STEP));
        else r.v[h] = __ldcg(reinterpret_cast<const float4*>(p + h * STEP));
    }
}
// the ragged last piece: groups past the end of the row read as zeros
template <bool BF16>
__device__ __forceinline__ void raw_load_tail(Raw<BF16>& r, const char* p, uint32_t e0, uint32_t V) {
    constexpr int G = Geo<BF16>::G, GS = Geo<BF16>::GS, STEP = GS * (BF16 ? 2 : 4);
#pragma unroll
    for (int h = 0; h < G; h++) {
        if constexpr (BF16) r.v[h] = e0 + h * GS < V ? __ldcg(reinterpret_cast<const uint4*>(p + h * STEP)) : make_uint4(0u, 0u, 0u, 0u);
        else r.v[h] = e0 + h * GS < V ? __ldcg(reinterpret_cast<const float4*>(p + h * STEP)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}
template <bool BF16>
__device__ __forceinline__ void raw_unpack(float (&x)[S_EPT], const Raw<BF16>& r) {
    if constexpr (BF16) {
#pragma unroll
        for (int h = 0; h < Geo<true>::G; h++) {
            const uint32_t u4[4] = {r.v[h].x, r.v[h].y, r.v[h].z, r.v[h].w};
#pragma unroll
            for (int u = 0; u < 4; u++) {   // a 16-bit shift widens bf16 to f32 exactly
                x[h * 8 + 2 * u] = __uint_as_float(u4[u] << 16);
                x[h * 8 + 2 * u + 1] = __uint_as_float(u4[u] & 0xffff0000u);
            }
        }
    } else {
#pragma unroll
        for (int h = 0; h < Geo<false>::G; h++) { x[4 * h] = r.v[h].x; x[4 * h + 1] = r.v[h].y; x[4 * h + 2] = r.v[h].z; x[4 * h + 3] = r.v[h].w; }
    }
}

// Rows beyond S_SHORT_VOCAB keep no bits: the first 16 lanes make the region's 16 words from the mask (one 64-byte load, under
// way together with the logits) and the region's entries.  256 rows of 262208: top-k 103 us, with 512 ids 119, with a mask 112.
template <bool BITS, class SM>
__device__ __forceinline__ uint32_t region_word(const SM& sm, uint32_t region) {
    uint32_t word = 0u;
    if constexpr (BITS && SM::IS_LONG) {
        const uint32_t lane = threadIdx.x & 31u, at = region * (S_REGION / 32) + lane, whole = sm.pa.V / 32u;
        if (lane < S_REGION / 32u) {
            word = at < whole ? 0xffffffffu : at == whole ? (1u << (sm.pa.V & 31u)) - 1u : 0u;
            if (sm.pa.mw && word) word &= __ldg(sm.pa.mw + at);
        }
        const uint32_t e1 = sm.rs[region + 1];
        for (uint32_t e = sm.rs[region]; e < e1; e++) {
            const uint32_t id = sm.ent_id[e];
            if (((id >> 5) & 15u) == lane) word &= ~(1u << (id & 31u));
        }
    }
    return word;
}
// Raw logits of piece q -> the logits of the pass: -inf where the row's bits say so (BITS: grammar mask, entries, end of
// the row) or behind the end of the row.  The bits come from shared memory, four logits (bf16: eight) of a lane to the
// load.  (Read from the mask table a piece at a time, every group of the piece waited for L2: 128 masked rows of 151936
// took 100 us, with the bits 51.)  bf16 rows of one CTA each, whose passes are bound by instructions: four bits at a time pick what is
// added to their logits from a table, two packed additions and a load in place of four tests and four selects (256 mixed rows of
// 256000 158.5 -> 154.4 us; -0 becomes +0, which compares equal everywhere).  f32 rows wait for the extra load longer than that saves
// (128 masked rows of 151936 48.5 -> 50.9), and so do rows that a cluster shares (bf16, with top-k 1, without / with the
// table: 16 rows of 1000 17.4 / 18.4, 64 of 16384 19.7 / 20.5, 64 of 128000 with a mask 33.1 / 33.9).
template <bool BF16, bool BITS, bool TAIL, bool CL, class SM>
__device__ __forceinline__ void fix_x(const SM& sm, float (&x)[S_EPT], uint32_t q, uint32_t word) {
    constexpr int G = Geo<BF16>::G, GE = Geo<BF16>::GE, GS = Geo<BF16>::GS;
    if (!BITS && !TAIL) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t e0 = q * S_PIECE + (uint32_t)w * S_REGION + (uint32_t)lane * GE;
    const uint32_t shift = ((uint32_t)lane * GE) & 31u;
#pragma unroll
    for (int h = 0; h < G; h++) {
        const uint32_t idx = e0 + h * GS;
        if constexpr (BITS && BF16 && !CL) {
            const uint32_t bits = SM::IS_LONG ? __shfl_sync(FULL, word, (int)((idx >> 5) & 15u)) : sm.bits[idx >> 5];
#pragma unroll
            for (int c = 0; c < GE; c += 4) {
                const uint32_t at = __funnelshift_r(bits, bits, shift + c - 4u) & 0xf0u;   // sixteen times the four bits
                const float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(sm.bit_tab) + at);
                float* v = x + h * GE + c;
                const float2 lo = __fadd2_rn(make_float2(v[0], v[1]), make_float2(t.x, t.y)), hi = __fadd2_rn(make_float2(v[2], v[3]), make_float2(t.z, t.w));
                v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
            }
            continue;
        }
        uint32_t bits = 0xffffffffu;
        if (BITS && SM::IS_LONG) bits = __shfl_sync(FULL, word, (int)((idx >> 5) & 15u)) >> shift;
        else if (BITS) bits = sm.bits[idx >> 5] >> shift;
        else if (idx >= sm.pa.V) bits = 0u;
#pragma unroll
        for (int c = 0; c < GE; c++)
            if (!((bits >> c) & 1u)) x[h * GE + c] = -INFINITY;
    }
}

// What the chain sees at an entry: penalties, mask, EOS fix on the raw logit.
__device__ __forceinline__ float entry_value(const PassArgs& pa, float v, uint32_t c) {
    const uint32_t n = c & ~(ENT_MASKED | ENT_EOS);
    if (n) {
        if (pa.flags & PF_REP) v = v > 0.0f ? fdiv(v, pa.rep) : fmul(v, pa.rep);
        if (pa.flags & PF_FP) {
            v = fsub(v, fmul(pa.freq, (float)n));
            if (pa.flags & PF_PRES) v = fsub(v, pa.pres);
        }
    }
    if ((c & ENT_MASKED) || !finite_f(v)) v = (c & ENT_EOS) ? 0.0f : -INFINITY;   // an overflowed penalty counts as masked
    return v;
}
// The raw logits of the region's entries into ent_raw, asynchronously: the region's own loads bring the same lines, and
// nothing in the pass waits for these.  (Waited for in the pass, to be part of its maxima and sums, they made pass 1 over
// 256 rows take 30 us in place of 21; found through a staging area 33 us; gathered before the pass 21 us and 4 us more in
// front of it.)
template <bool BF16, class SM>
__device__ __forceinline__ void copy_entries(SM& sm, uint32_t region) {
    const uint32_t e1 = sm.rs[region + 1];
    for (uint32_t e = sm.rs[region] + (threadIdx.x & 31u); e < e1; e += 32u) {
        const uint32_t id = sm.ent_id[e];
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(&sm.ent_raw[e])),
                     "l"(sm.pa.rowp + (size_t)(BF16 ? id >> 1 : id) * 4u) : "memory");
    }
}

// pass 1 on one piece
template <bool BF16, bool BITS, bool TAIL, bool STOCH, bool CL, class SM>
__device__ __forceinline__ void p1_piece(SM& sm, const Raw<BF16>& raw, uint32_t q, float& am, float& tmx, uint32_t& tqx) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t region = q * SNW + (uint32_t)w;
    if (BITS) copy_entries<BF16>(sm, region);
    const uint32_t word = region_word<BITS>(sm, region);
    float x[S_EPT];
    raw_unpack<BF16>(x, raw);
    am = absmax_ept_nan(am, x);   // max |raw logit|, NaN-propagating: the sanity check
    fix_x<BF16, BITS, TAIL, CL>(sm, x, q, word);
    const float pm = max_ept(x);
    if (pm >= tmx) { tmx = pm; tqx = q; }   // pieces arrive in descending order: an equal maximum here has the lower id
    if (STOCH) {
        const float sc = sm.pa.sc;
        // one of the per-thread maxima that bound the top-k threshold
        const uint32_t ci = (q % S_NCELL) * SNT + threadIdx.x;
        if (pm > sm.cell[ci]) sm.cell[ci] = pm;
        // plain sum of the numerators of the warp's 512 logits, relative to their own maximum
        const uint32_t pb = f2u(pm);
        const uint32_t wkey = __reduce_max_sync(FULL, pb ^ (((uint32_t)((int32_t)pb >> 31)) | 0x80000000u));   // monotone; -inf lowest
        const float wm = u2f((wkey & 0x80000000u) ? (wkey & 0x7fffffffu) : ~wkey);
        const float cc = -wm * sc;
        const float2 sc2 = make_float2(sc, sc), cc2 = make_float2(cc, cc);
        float2 p01 = make_float2(0.0f, 0.0f), p23 = p01;
#pragma unroll
        for (int j = 0; j < S_EPT; j += 4) {
            p01 = __fadd2_rn(p01, ex2_pair(__ffma2_rn(make_float2(x[j], x[j + 1]), sc2, cc2)));
            p23 = __fadd2_rn(p23, ex2_pair(__ffma2_rn(make_float2(x[j + 2], x[j + 3]), sc2, cc2)));
        }
        // summed over the warp in fixed point (a lane's sum is at most 16, and an estimate is all that is needed); an
        // all-masked region has NaN here, which converts to 0
        const uint32_t ws = __reduce_add_sync(FULL, __float2uint_rn(((p01.x + p01.y) + (p23.x + p23.y)) * 1048576.0f));
        if (lane == 0) {
            sm.reg_a[region] = wm; sm.reg_b[region] = (float)ws * (1.0f / 1048576.0f);
        }
    }
}

// This warp's share of the fold (the same value in all its lanes): a count of ulps of the binade cur_bb, folded into
// accd whenever the binade changes.
struct FoldAcc {
    double accd;
    unsigned long long cur_n;
    uint32_t cur_bb;
    __device__ __forceinline__ void flush() {
        accd += (double)cur_n * ((double)u2f(cur_bb) * 1.1920928955078125e-07);   // units of that binade's ulp
        cur_n = 0ull;
    }
};

template <bool CL, class SM>
__device__ __forceinline__ void add_candidate(SM& sm, uint32_t id, float x) {
    uint32_t* n = CL ? sm.pa.cand_n_p : &sm.cand_n;
    const uint32_t at = atomicAdd(n, 1u);
    if (at >= (uint32_t)F_MCAP) return;
    (CL ? sm.pa.cand_id_p : sm.cand_id)[at] = id;
    (CL ? sm.pa.cand_x_p : sm.cand_x)[at] = x;
}

// x[j], four selections deep
__device__ __forceinline__ float pick(const float (&x)[S_EPT], uint32_t j) {
    float a[8];
#pragma unroll
    for (int u = 0; u < 8; u++) a[u] = (j & 1u) ? x[2 * u + 1] : x[2 * u];
#pragma unroll
    for (int u = 0; u < 4; u++) a[u] = (j & 2u) ? a[2 * u + 1] : a[2 * u];
#pragma unroll
    for (int u = 0; u < 2; u++) a[u] = (j & 4u) ? a[2 * u + 1] : a[2 * u];
    return (j & 8u) ? a[1] : a[0];
}

// the logarithm (base 2) of a numerator
template <bool BF16>
__device__ __forceinline__ float exponent_of(const PassArgs& pa, float x) {
    if (BF16) return __fmaf_rn(x, pa.sc, pa.c_hi) + __fmaf_rn(x, pa.sc_lo, pa.c_lo);
    return __fmaf_rn(x, pa.sc, pa.c_hi) + pa.c_lo;
}

// The entries' part of pass 2: candidates, and what they add to the fold where it stands in their region.  (In a region
// that is folded the careful way they are added at its start: a rounding there is half an ulp of the running value at most.)
template <bool BF16, bool CL, class SM>
__device__ __forceinline__ void p2_entries(SM& sm, uint32_t n_ent) {
    if (threadIdx.x / 32u * 32u >= n_ent) return;   // warp-uniform
    double td = 0.0;
    for (uint32_t e = threadIdx.x; e < n_ent; e += SNT) {
        const float x = sm.ent_x[e];
        const uint32_t id = sm.ent_id[e], region = id / S_REGION;
        if (x >= sm.pa.cut_f) add_candidate<CL>(sm, id, x);
        const float v = ex2_approx_ftz(exponent_of<BF16>(sm.pa, x)), base = sm.reg_a[region];
        if (base != 0.0f) td += (double)(f2u(fadd(base, v)) - f2u(base)) * ((double)base * 1.1920928955078125e-07);
        else { const float R0 = sm.reg_b[region]; td += (double)fsub(fadd(R0, v), R0); }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) td += __shfl_xor_sync(FULL, td, o);
    if ((threadIdx.x & 31u) == 0u) sm.wacc[threadIdx.x >> 5] += td;
}

// How pass 2 puts candidates on the list, for f32 rows that a cluster shares: in rounds over the lanes where there are few, in
// rounds over the sixteen positions of a lane's logits where there are many.  Over the lanes / over the positions, us: 8 rows of
// 151936 with top-k 40 27.0 / 28.5, 64 with 50 37.9 / 38.5, 64 with 500 49.4 / 50.3, 64 with 1024 68.7 / 68.0; 2048 to 256000
// logits, 1 to 64 rows and top-k 1 to 512 are within 3 % or quicker.  (One CTA per row, and bf16 rows: over the
// positions.  Some rows with long lists take half as long again over the lanes, 256 with top-k 500 92 / 80, and both ways in one
// kernel cost all others 1 %.)
template <bool BF16, bool CL>
__device__ __forceinline__ bool few_candidates(uint32_t top_k) { return CL && !BF16 && top_k <= 512u; }

// pass 2 on one piece
template <bool BF16, bool BITS, bool TAIL, bool CL, class SM>
__device__ __forceinline__ void p2_piece(SM& sm, const Raw<BF16>& raw, uint32_t q, FoldAcc& fa) {
    constexpr int G = Geo<BF16>::G, GE = Geo<BF16>::GE;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float sc = sm.pa.sc, c_hi = sm.pa.c_hi, c_lo = sm.pa.c_lo, cut_f = sm.pa.cut_f;
    const uint32_t word = region_word<BITS>(sm, q * SNW + (uint32_t)w);
    float x[S_EPT];
    raw_unpack<BF16>(x, raw);
    fix_x<BF16, BITS, TAIL, CL>(sm, x, q, word);
    const float pm = max_ept(x);
    if (pm >= cut_f) {
        const uint32_t e0 = q * S_PIECE + (uint32_t)w * S_REGION + (uint32_t)lane * GE;
        if (CL && !BF16 && sm.pa.few) {   // as many rounds as the lane with the most candidates has
            uint32_t which = 0u;
#pragma unroll
            for (int j = 0; j < S_EPT; j++) which |= x[j] >= cut_f ? 1u << j : 0u;
#pragma unroll 1
            for (; which; which &= which - 1u) {
                const int j = __ffs((int)which) - 1;
                add_candidate<CL>(sm, elem_id<BF16>(e0, j), pick(x, (uint32_t)j));
            }
        } else {   // one for each of the sixteen positions at which some lane has one
#pragma unroll
            for (int j = 0; j < S_EPT; j++)
                if (x[j] >= cut_f) add_candidate<CL>(sm, elem_id<BF16>(e0, j), x[j]);
        }
    }
    const uint32_t region = q * SNW + (uint32_t)w;
    if (TAIL && region >= sm.pa.n_regions) return;   // warp-uniform: past the end of the row
    // nothing here is large enough to move the running value: the usual case once the sum has grown
    if (__all_sync(FULL, pm < sm.reg_t[region])) return;
    const float2 sc2 = make_float2(sc, sc), hi2 = make_float2(c_hi, c_hi), lo2 = make_float2(c_lo, c_lo);
    if (BF16) {
        // bf16 rows hold every value thousands of times, and a numerator that is off by 1e-6 in the same direction for
        // all of them moves whole groups of additions across a rounding boundary: scale and constant as two floats
        const float2 sl2 = make_float2(sm.pa.sc_lo, sm.pa.sc_lo);
#pragma unroll
        for (int j = 0; j < S_EPT; j += 2) {   // -inf stays -inf
            const float2 v = make_float2(x[j], x[j + 1]), e = __fadd2_rn(__ffma2_rn(v, sc2, hi2), __ffma2_rn(v, sl2, lo2));
            x[j] = e.x; x[j + 1] = e.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < S_EPT; j += 2) {   // -inf stays -inf
            const float2 e = __ffma2_rn(make_float2(x[j], x[j + 1]), sc2, hi2);
            x[j] = e.x; x[j + 1] = e.y;
        }
        if (c_lo != 0.0f) {   // CTA-uniform: the constant needs its second float (cold rows, large maxima)
#pragma unroll
            for (int j = 0; j < S_EPT; j += 2) {
                const float2 e = __fadd2_rn(make_float2(x[j], x[j + 1]), lo2);
                x[j] = e.x; x[j + 1] = e.y;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < S_EPT; j++) x[j] = ex2_approx_ftz(x[j]);   // -inf -> 0
    const float base = sm.reg_a[region];
    const uint32_t bb = f2u(base);
    const bool quick = bb != 0u;
    if (quick) {
        // every thread from the lower end of the binade the fold is in (the table guarantees that nobody leaves it);
        // four chains: the increments do not depend on the order
        float2 a01 = make_float2(base, base), a23 = a01;
#pragma unroll
        for (int j = 0; j < S_EPT; j += 4) {
            a01 = __fadd2_rn(a01, make_float2(x[j], x[j + 1]));
            a23 = __fadd2_rn(a23, make_float2(x[j + 2], x[j + 3]));
        }
        const uint32_t ws = __reduce_add_sync(FULL, ((f2u(a01.x) - bb) + (f2u(a01.y) - bb)) + ((f2u(a23.x) - bb) + (f2u(a23.y) - bb)));   // < 32 * 2^25
        if (bb != fa.cur_bb) { fa.flush(); fa.cur_bb = bb; }
        fa.cur_n += ws;
    }
    if (!quick) {
        // the running value may leave its binade here (or the fold starts here): every 128-bit group from its own
        // estimate of the running value, real additions, so that a crossing is reproduced
        float stv[G], run = 0.0f;
#pragma unroll
        for (int h = 0; h < G; h++) {
            float gs = 0.0f;
#pragma unroll
            for (int c = 0; c < GE; c++) gs += x[h * GE + c];
            float inc = gs;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += up;
            }
            stv[h] = run + (inc - gs);
            run += __shfl_sync(FULL, inc, 31);
        }
        const float R0 = sm.reg_b[region];
        float tinc = 0.0f;
#pragma unroll
        for (int h = 0; h < G; h++) {
            const float R = fadd(R0, stv[h]);
            float a2 = R;
#pragma unroll
            for (int c = 0; c < GE; c++) a2 = fadd(a2, x[h * GE + c]);
            tinc = fadd(tinc, fsub(a2, R));
        }
        double td = (double)tinc;
#pragma unroll
        for (int o = 16; o; o >>= 1) td += __shfl_xor_sync(FULL, td, o);
        fa.accd += td;
    }
}

// The loops below wait for their loads with nothing else to do (there are no registers for a second piece), so the
// pieces they will need next are requested ahead of time as plain L2 prefetches: memory stays busy while the warps
// compute, and the loads that follow find their lines in L2.  One 128-byte line per lane of the lower half-warp.
#ifndef PGS_PF_DIST
#define PGS_PF_DIST 2
#endif
template <bool BF16>
__device__ __forceinline__ void prefetch_piece(const char* warp_piece) {
    constexpr int LINES = S_REGION * (BF16 ? 2 : 4) / 128;   // 16 (f32) or 8 (bf16)
    const int lane = threadIdx.x & 31;
    if (lane < LINES) prefetch_l2(warp_piece + lane * 128);
}

// pass 1 over the whole pieces n_full-1 .. 0; the thread's results go to sm.t_*[tid]
template <bool BF16, bool BITS, bool STOCH, bool CL, class SM>
__device__ __noinline__ void pass1_whole(SM& sm) {
    constexpr int PB = S_PIECE * (BF16 ? 2 : 4);
    const uint32_t lane_e0 = (threadIdx.x >> 5) * S_REGION + (threadIdx.x & 31) * Geo<BF16>::GE;
    const uint32_t n = sm.pa.n_full;   // >= 1
    if (CL) {   // the pieces q0, q0 + qstep, ... of the row, last one first
        float am = 0.0f, tmx = -INFINITY;
        uint32_t tqx = 0u;
        const int q0 = (int)sm.pa.q0, qs = (int)sm.pa.qstep;
        if (q0 < (int)n) {
            int q = q0 + (((int)n - 1 - q0) / qs) * qs;
            const size_t step = (size_t)qs * PB;
            const char* p = sm.pa.rowp + (size_t)lane_e0 * (BF16 ? 2 : 4) + (size_t)q * PB;
            const char* wp = sm.pa.rowp + (size_t)((threadIdx.x >> 5) * S_REGION) * (BF16 ? 2 : 4) + (size_t)q * PB;
            if (q - qs >= q0) prefetch_piece<BF16>(wp - step);
#pragma unroll 1
            for (; q >= q0; q -= qs, p -= step, wp -= step) {
                if (q - 2 * qs >= q0) prefetch_piece<BF16>(wp - 2 * step);
                Raw<BF16> b;
                raw_load<BF16>(b, p);
                p1_piece<BF16, BITS, false, STOCH, CL>(sm, b, (uint32_t)q, am, tmx, tqx);
            }
        }
        sm.t_am[threadIdx.x] = am; sm.t_max[threadIdx.x] = tmx; sm.t_q[threadIdx.x] = tqx;
        return;
    }
    const char* p = sm.pa.rowp + (size_t)lane_e0 * (BF16 ? 2 : 4) + (size_t)(n - 1u) * PB;
    float am = 0.0f, tmx = -INFINITY;
    uint32_t tqx = 0u;
    const char* wp = sm.pa.rowp + (size_t)((threadIdx.x >> 5) * S_REGION) * (BF16 ? 2 : 4) + (size_t)(n - 1u) * PB;   // the warp's 512 logits of a piece
#pragma unroll 1
    for (uint32_t d = 1; d < (uint32_t)PGS_PF_DIST && d < n; d++) prefetch_piece<BF16>(wp - (size_t)d * PB);
#pragma unroll 1
    for (uint32_t q = n; q-- > 0u; p -= PB, wp -= PB) {
        if (q >= (uint32_t)PGS_PF_DIST) prefetch_piece<BF16>(wp - (size_t)PGS_PF_DIST * PB);
        Raw<BF16> b;
        raw_load<BF16>(b, p);
        p1_piece<BF16, BITS, false, STOCH, CL>(sm, b, q, am, tmx, tqx);
    }
    sm.t_am[threadIdx.x] = am; sm.t_max[threadIdx.x] = tmx; sm.t_q[threadIdx.x] = tqx;
}

// pass 2 over the whole pieces 0 .. n_full-1; the warp's share of the fold is added to sm.wacc[w]
template <bool BF16, bool BITS, bool CL, class SM>
__device__ __noinline__ void pass2_whole(SM& sm) {
    constexpr int PB = S_PIECE * (BF16 ? 2 : 4);
    const uint32_t lane_e0 = (threadIdx.x >> 5) * S_REGION + (threadIdx.x & 31) * Geo<BF16>::GE;
    const uint32_t n = sm.pa.n_full;   // >= 1
    const char* p = sm.pa.rowp + (size_t)lane_e0 * (BF16 ? 2 : 4);
    FoldAcc fa;
    fa.accd = 0.0; fa.cur_n = 0ull; fa.cur_bb = 0u;
    if (CL) {   // the pieces q0, q0 + qstep, ... of the row, first one first
        const uint32_t q0 = sm.pa.q0, qs = sm.pa.qstep;
        const size_t step = (size_t)qs * PB;
        p += (size_t)q0 * PB;
        const char* wp = sm.pa.rowp + (size_t)((threadIdx.x >> 5) * S_REGION) * (BF16 ? 2 : 4) + (size_t)q0 * PB;
        if (q0 + qs < n) prefetch_piece<BF16>(wp + step);
#pragma unroll 1
        for (uint32_t q = q0; q < n; q += qs, p += step, wp += step) {
            if (q + 2u * qs < n) prefetch_piece<BF16>(wp + 2 * step);
            Raw<BF16> b;
            raw_load<BF16>(b, p);
            p2_piece<BF16, BITS, false, true>(sm, b, q, fa);
        }
        fa.flush();
        if ((threadIdx.x & 31) == 0) sm.wacc[threadIdx.x >> 5] += fa.accd;
        return;
    }
    const char* wp = sm.pa.rowp + (size_t)((threadIdx.x >> 5) * S_REGION) * (BF16 ? 2 : 4);
#pragma unroll 1
    for (uint32_t d = 1; d < (uint32_t)PGS_PF_DIST && d < n; d++) prefetch_piece<BF16>(wp + (size_t)d * PB);
#pragma unroll 1
    for (uint32_t q = 0u; q < n; q++, p += PB, wp += PB) {
        if (q + (uint32_t)PGS_PF_DIST < n) prefetch_piece<BF16>(wp + (size_t)PGS_PF_DIST * PB);
        Raw<BF16> b;
        raw_load<BF16>(b, p);
        p2_piece<BF16, BITS, false, false>(sm, b, q, fa);
    }
    fa.flush();
    if ((threadIdx.x & 31) == 0) sm.wacc[threadIdx.x >> 5] += fa.accd;
}

// CL: a thread-block cluster of 2, 4 or 8 CTAs shares every row (small batches: a row alone on one CTA is bound by
// the latency of its own loads and dependent instructions).  CTA k of the cluster takes the pieces k, k + size, ...;
// the CTAs exchange their maxima, region tables, histograms, candidates and fold shares through distributed shared
// memory around two cluster barriers, and the first CTA finishes the row (a launch has one cluster per row).  Every decision that ends a row
// early is taken from values all CTAs of the cluster hold alike, so they always meet at the same barriers.
template <bool BF16, bool CL, bool LONG>
__global__ void __launch_bounds__(SNT, 2) stream_row_kernel(const RowArgs a, const StreamLaunch sl) {
    namespace cg = cooperative_groups;
    constexpr int GE = Geo<BF16>::GE;
    constexpr int ESZ = BF16 ? 2 : 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using SM = StreamSmem<LONG>;
    SM& sm = *reinterpret_cast<SM*>(smem_raw);
    const uint32_t H = sl.hash_slots;
    uint32_t* hkey = sm.hash;
    uint32_t* hcnt = sm.hash + H;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t V = a.vocab;
    const uint32_t n_full = V / S_PIECE;                        // whole pieces
    const bool has_tail = (V % S_PIECE) != 0u;                  // plus a ragged one at the end of the row
    const uint32_t n_regions = (V + S_REGION - 1) / S_REGION;
    const uint32_t lane_e0 = (uint32_t)w * S_REGION + (uint32_t)lane * GE;   // first element of the thread inside a piece
    if (tid < 32) sm.exp_tab[tid] = kExp2TableDev[tid];
    if (BF16 && !CL && tid < 16) sm.bit_tab[tid] = make_float4(tid & 1 ? 0.0f : -INFINITY, tid & 2 ? 0.0f : -INFINITY, tid & 4 ? 0.0f : -INFINITY, tid & 8 ? 0.0f : -INFINITY);
    if (tid == 0)
#pragma unroll 1
        for (int i = 0; i < 16; i++) sm.prof_acc[i] = 0;
    constexpr int PREP_TID = SNT - 32;   // lane 0 of the last warp
    uint32_t crank = 0u, csize = 1u;
    if (CL) {
        crank = cg::this_cluster().block_rank(); csize = cg::this_cluster().num_blocks();
        cg::this_cluster().barrier_arrive();   // waited for where the first of the others' shared memory is written
    }
    const uint32_t first_row = CL ? blockIdx.x / csize : blockIdx.x, row_step = CL ? gridDim.x / csize : gridDim.x;
    const uint32_t tail_owner = n_full % csize;   // the CTA that takes the ragged piece
    // set up while the kernel before this one drains; the pass over the work list is set up in the same way behind this one
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    if (tid == PREP_TID && first_row < a.rows) sprepare_row<BF16>(a, sl, first_row, sm.ctl[0]);
    long long tick_ = clock64();
    uint32_t it = 0;
    for (uint32_t row = first_row; row < a.rows; row += row_step, it++) {
        // ---- gate: at most `cohort` rows ahead of the rows that have left their first pass
        if (!CL && tid == 0 && row >= sl.cohort) {
            const uint32_t need = row - sl.cohort + 1u;
            const volatile uint32_t* done = sl.p1_done;
#pragma unroll 1
            for (uint32_t poll = 0; poll < sl.gate_polls; poll++) {
                if (*done - sl.done_base >= need) break;
                __nanosleep(200);
            }
        }
        // this row's parameters are complete, and every warp is done with the row before
        __syncthreads();
        PGS_STICK(0);   // gate + row barrier
        const SRowCtl& ctl = sm.ctl[it & 1];
        if (tid == PREP_TID && row + row_step < a.rows) sprepare_row<BF16>(a, sl, row + row_step, sm.ctl[(it + 1) & 1]);
        const bool writer = tid == 0 && crank == 0u;   // one thread of the row's (first) CTA
        if (ctl.kind != 0u) {
            if (writer) {
                if (ctl.kind == 1u) {
                    if (a.tp_records) tp_write_head(a, row, -INFINITY, 0.0f, 0u, ROW_BAD_PARAM, 0u);
                    else { a.token[row] = 0; a.status[row] = ROW_BAD_PARAM; if (a.drew) a.drew[row] = 0; }
                } else sl.work_rows[atomicAdd(sl.work_count, 1u)] = row;
                atomicAdd(sl.p1_done, 1u);
            }
            continue;
        }
        const float temp = ctl.temp;
        const uint32_t top_k = ctl.top_k, gflags = ctl.gflags, h0 = ctl.h0, nh = ctl.nh;
        const char* rowp = ctl.rowp;
        const float sc = ctl.sc;
        const bool greedy = temp < 1e-5f;
        const bool has_mask = ctl.mw != nullptr;
        const bool do_fp = !(fabsf(ctl.freq) < 1e-6f && fabsf(ctl.pres) < 1e-6f), do_pres = fabsf(ctl.pres) > 1e-6f;
        const bool do_rep = ctl.rep != 1.0f;
        const bool pen = nh > 0 && (do_fp || do_rep);
        const bool fix = has_mask && (gflags & 1u) && a.eos >= 0 && (uint32_t)a.eos < V;   // engine.rs:1307-1312
        const bool has_bits = has_mask || pen;
        if (tid == 0) {   // what the pass loops read
            PassArgs& pa = sm.pa;
            pa.rowp = rowp; pa.mw = ctl.mw; pa.freq = ctl.freq; pa.pres = ctl.pres; pa.rep = ctl.rep; pa.sc = sc; pa.sc_lo = ctl.sc_lo; pa.c_hi = 0.0f; pa.c_lo = 0.0f; pa.cut_f = 0.0f;
            pa.V = V; pa.n_full = n_full; pa.n_regions = n_regions; if (CL && !BF16) pa.few = few_candidates<BF16, CL>(top_k);
            pa.q0 = crank; pa.qstep = csize;
            pa.cand_n_p = &sm.cand_n; pa.cand_id_p = sm.cand_id; pa.cand_x_p = sm.cand_x;
            if (CL) {
                cg::cluster_group cluster = cg::this_cluster();
                pa.cand_n_p = cluster.map_shared_rank(&sm.cand_n, 0);
                pa.cand_id_p = cluster.map_shared_rank(sm.cand_id, 0);
                pa.cand_x_p = cluster.map_shared_rank(sm.cand_x, 0);
            }
            pa.flags = (do_rep ? PF_REP : 0u) | (do_fp ? PF_FP : 0u) | (do_pres ? PF_PRES : 0u);
        }

        // the history ids of the thread
        constexpr int HPT = S_MAX_HASH / 2 / SNT;
        uint32_t hid[HPT];
#pragma unroll
        for (int u = 0; u < HPT; u++) hid[u] = pen && (uint32_t)(tid + u * SNT) < nh ? __ldg(a.hist_ids + h0 + tid + u * SNT) : S_NIL;
        // the pieces the first pass starts with are requested now, so that they arrive while the history is indexed
        if (n_full > 0u) {
            constexpr int PB = S_PIECE * ESZ;
            const uint32_t qs = CL ? csize : 1u;
            if (n_full > crank) {
                const uint32_t qlast = crank + ((n_full - 1u - crank) / qs) * qs;
                const char* wp = rowp + (size_t)(w * S_REGION) * ESZ + (size_t)qlast * PB;
                prefetch_piece<BF16>(wp);
                if (qlast >= qs + crank) prefetch_piece<BF16>(wp - (size_t)qs * PB);
            }
        }
        // ---- entries (distinct history ids with what the penalties make of them; the EOS fix) and the row's bits
        bool defer_row = false;
        uint32_t n_ent = 0u;
        if (has_bits) {
#pragma unroll
            for (int u = 0; u < HPT; u++) {
                if (hid[u] != S_NIL) hid[u] -= a.id_base;   // ids below a shard wrap around
                // engine.rs:1562; CL: another CTA's piece
                if (hid[u] >= V || (CL && (hid[u] / S_PIECE) % csize != crank)) hid[u] = S_NIL;
            }
            uint32_t* rcnt = sm.ent_raw;   // per region, until pass 1
            const uint32_t* mw = ctl.mw;
            if constexpr (!LONG) {
                const uint32_t whole = V / 32u, words = ((V + S_PIECE - 1) / S_PIECE) * (S_PIECE / 32);
#pragma unroll 4
                for (uint32_t k = tid; k < words; k += SNT) {
                    uint32_t b = k < whole ? 0xffffffffu : k == whole ? (1u << (V & 31u)) - 1u : 0u;
                    if (has_mask && b) b &= __ldg(mw + k);
                    sm.bits[k] = b;
                }
            }
            static_assert(SM::MAX_REGIONS % SNT == 0 && SM::MAX_REGIONS <= S_ENT, "whole regions per thread, their counts in the entries' space");
#pragma unroll
            for (int u = 0; u < SM::MAX_REGIONS / SNT; u++) { rcnt[tid + u * SNT] = 0u; sm.rs[tid + u * SNT] = 0; sm.reg_t[tid + u * SNT] = 0.0f; }
            if (tid < 2) sm.rs[SM::MAX_REGIONS + tid] = 0;
            if (pen || fix) {
#pragma unroll 1
                for (uint32_t s = tid; s < 2u * H; s += SNT) sm.hash[s] = s < H ? S_NIL : 0u;
                __syncthreads();
                // the thread that meets an id first owns its entry
                bool spilled = false;
                const auto insert = [&](uint32_t id, uint32_t n) {   // the id's slot | 2^31 where it is not new
                    const uint32_t mul = id * 2654435761u;
                    uint32_t s = (mul ^ (mul >> 15)) & (H - 1u);
#pragma unroll 1
                    for (int probe = 0; probe < 128; probe++) {
                        const uint32_t prev = atomicCAS(&hkey[s], S_NIL, id);
                        if (prev == S_NIL || prev == id) {
                            if (prev == S_NIL) {
                                const uint32_t bit = 1u << (id & 31u);
                                if constexpr (LONG) { if (has_mask && !(__ldg(mw + (id >> 5)) & bit)) n |= ENT_MASKED; }
                                else if (!(atomicAnd(&sm.bits[id >> 5], ~bit) & bit)) n |= ENT_MASKED;
                                if (fix && id == (uint32_t)a.eos) n |= ENT_EOS;
                                atomicAdd(&rcnt[id / S_REGION], 1u);
                            }
                            atomicAdd(&hcnt[s], n);
                            return prev == S_NIL ? s : s | 0x80000000u;
                        }
                        s = (s + 1u) & (H - 1u);
                    }
                    spilled = true;
                    return S_NIL;
                };
                uint32_t slot[HPT];
#pragma unroll
                for (int u = 0; u < HPT; u++) slot[u] = hid[u] != S_NIL ? insert(hid[u], 1u) : S_NIL;
                uint32_t eos_slot = S_NIL;
                if (tid == 0 && fix && (!CL || ((uint32_t)a.eos / S_PIECE) % csize == crank)) eos_slot = insert((uint32_t)a.eos, 0u);
                if (__syncthreads_or(spilled)) {
                    if (!CL) {   // CTA-uniform
                        if (writer) { sl.work_rows[atomicAdd(sl.work_count, 1u)] = row; atomicAdd(sl.p1_done, 1u); }
                        continue;
                    }
                    // A cluster must meet at its barriers whatever one of its CTAs finds here: the CTA goes through the
                    // first pass without entries and says so in the exchange behind it, where all CTAs give the row up
                    // together.
                    defer_row = true;
                } else {
                    constexpr int RPT = SM::MAX_REGIONS / SNT;   // regions per thread
                    uint32_t cnt[RPT], own = 0u;
#pragma unroll
                    for (int u = 0; u < RPT; u++) { cnt[u] = rcnt[tid * RPT + u]; own += cnt[u]; }
                    uint32_t before = sblock_excl_scan_u32(own, &n_ent, sm.scan_u);
#pragma unroll
                    for (int u = 0; u < RPT; u++) { sm.rs[tid * RPT + u] = (uint16_t)before; rcnt[tid * RPT + u] = before; before += cnt[u]; }
                    if (tid < 2) sm.rs[SM::MAX_REGIONS + tid] = (uint16_t)n_ent;
                    __syncthreads();
                    const auto entry = [&](uint32_t id, uint32_t s) {
                        if (s & 0x80000000u) return;
                        const uint32_t at = atomicAdd(&rcnt[id / S_REGION], 1u);
                        sm.ent_id[at] = id;
                        sm.ent_x[at] = u2f(hcnt[s]);
                    };
#pragma unroll
                    for (int u = 0; u < HPT; u++) entry(hid[u], slot[u]);
                    if (tid == 0 && fix) entry((uint32_t)a.eos, eos_slot);
                }
                __syncthreads();
            }
        }
#pragma unroll
        for (int c = 0; c < S_NCELL; c++) sm.cell[c * SNT + tid] = -INFINITY;
        __syncthreads();   // PassArgs, entries and bits are set
        PGS_STICK(1);   // history indexed

        // ================================================================ pass 1 (HBM, last piece first)
        float am = 0.0f;            // max |raw logit|
        float tmx = -INFINITY;      // the thread's running maximum without entries, and the lowest piece that holds it
        uint32_t tqx = 0u;
        const bool my_tail = has_tail && (!CL || tail_owner == crank);
        if (my_tail) {
            Raw<BF16> raw;
            raw_load_tail<BF16>(raw, rowp + ((size_t)n_full * S_PIECE + lane_e0) * ESZ, n_full * S_PIECE + lane_e0, V);
            if (has_bits) { if (greedy) p1_piece<BF16, true, true, false, CL>(sm, raw, n_full, am, tmx, tqx); else p1_piece<BF16, true, true, true, CL>(sm, raw, n_full, am, tmx, tqx); }
            else { if (greedy) p1_piece<BF16, false, true, false, CL>(sm, raw, n_full, am, tmx, tqx); else p1_piece<BF16, false, true, true, CL>(sm, raw, n_full, am, tmx, tqx); }
        }
        if (n_full > 0u) {
            if (has_bits) { if (greedy) pass1_whole<BF16, true, false, CL>(sm); else pass1_whole<BF16, true, true, CL>(sm); }
            else { if (greedy) pass1_whole<BF16, false, false, CL>(sm); else pass1_whole<BF16, false, true, CL>(sm); }
            am = absmax3_nan(am, sm.t_am[tid], 0.0f);
            if (sm.t_max[tid] >= tmx) { tmx = sm.t_max[tid]; tqx = sm.t_q[tid]; }   // the whole pieces come before the ragged one
        }
        PGS_STICK(2);   // pass 1

        // ---- row maximum, sanity, and the material for the top-k bound
        float emx = -INFINITY;      // the largest of the thread's entries
        if (n_ent) {   // CTA-uniform
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            for (uint32_t e = tid, c = 0; e < n_ent; e += SNT, c++) {
                const uint32_t raw = sm.ent_raw[e];
                const float v = entry_value(sm.pa, u2f(!BF16 ? raw : (sm.ent_id[e] & 1u) ? raw & 0xffff0000u : raw << 16), f2u(sm.ent_x[e]));
                sm.ent_x[e] = v;
                emx = fmaxf(emx, v);
                float& cell = sm.cell[c % S_NCELL * SNT + tid];   // (any cell: a logit counts in one)
                if (v > cell) cell = v;
            }
        }
        {
            uint32_t lo = 0xffffffffu, fin = 0u;
            if (!greedy) {
#pragma unroll
                for (int c = 0; c < S_NCELL; c++) {
                    const uint32_t k = order_key(sm.cell[c * SNT + tid]);
                    if (!k) continue;
                    lo = umin(lo, k);
                    fin++;
                }
            }
            const uint32_t wk = __reduce_max_sync(FULL, order_key(fmaxf(tmx, emx)));
            const uint32_t wlo = __reduce_min_sync(FULL, lo);
            const uint32_t wfin = __reduce_add_sync(FULL, fin);
            const uint32_t wbad = __any_sync(FULL, !(am < INFINITY)) ? 1u : 0u;
            if (lane == 0) { sm.red_key[w] = wk; sm.red_lo[w] = wlo; sm.red_fin[w] = wfin; sm.red_flag[w] = wbad; sm.wacc[w] = 0.0; }
#pragma unroll
            for (int u = 0; u < S_BPT; u++) sm.hist[u * SNT + tid] = 0u;
            if (tid == 0) { sm.cand_n = 0u; sm.sel_bucket = 0u; sm.amax = 0xffffffffu; }
        }
        __syncthreads();
        uint32_t gkey = __reduce_max_sync(FULL, lane < SNW ? sm.red_key[lane] : 0u);
        uint32_t lo_key = __reduce_min_sync(FULL, lane < SNW ? sm.red_lo[lane] : 0xffffffffu);
        uint32_t n_fin = __reduce_add_sync(FULL, lane < SNW ? sm.red_fin[lane] : 0u);
        bool nonfinite = __any_sync(FULL, lane < SNW && sm.red_flag[lane] != 0u);
        const float lm = key_to_float(gkey);   // (of no interest without one)
        if (!greedy && gkey)
            // (Entries are in region order: the lanes of one region add up first.  With one atomic per entry crowded regions
            // waited for one after the other: 256 rows of 4096 with 2048 ids 44 us, now 28.)
            for (uint32_t e = tid; (e & ~31u) < n_ent; e += SNT) {   // warp-uniform
                const bool is = e < n_ent;
                const uint32_t r = is ? sm.ent_id[e] / S_REGION : S_NIL;
                float v = is && sm.ent_x[e] > -INFINITY ? ex2_approx_ftz((sm.ent_x[e] - lm) * sc) : 0.0f;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float t = __shfl_up_sync(FULL, v, o);
                    const uint32_t tr = __shfl_up_sync(FULL, r, o);
                    if (lane >= o && tr == r) v += t;
                }
                const uint32_t next = __shfl_down_sync(FULL, r, 1);
                if (v > 0.0f && is && (lane == 31 || next != r)) atomicAdd(&sm.reg_t[r], v);
            }
        // The per-thread maxima are spread over S_NB equal-width buckets between `lo_v` and `top` (a monotone map); with b
        // the highest bucket such that the buckets b.. hold at least `need` maxima, every logit of bucket b - 1 or higher
        // counts: at least `need` logits reach the bound returned.  all: over the CTAs of the cluster.
        const auto kth_bound = [&](uint32_t need, float lo_v, float top, bool all) {
            const float scb = top > lo_v ? (float)(S_NB - 1) / (top - lo_v) : 0.0f;
#pragma unroll
            for (int c = 0; c < S_NCELL; c++) {
                const float cv = sm.cell[c * SNT + tid];
                if (finite_f(cv)) atomicAdd(&sm.hist[min((uint32_t)(S_NB - 1), (uint32_t)((cv - lo_v) * scb))], 1u);
            }
            __syncthreads();
            // thread j owns the S_BPT buckets S_NB-1 - j*S_BPT - u; `above` = maxima in higher buckets
            uint32_t hv[S_BPT], own = 0u;
            if (CL && all) {
                cg::cluster_group cluster = cg::this_cluster();
                cluster.sync();
#pragma unroll
                for (int u = 0; u < S_BPT; u++) {
                    hv[u] = 0u;
                    for (uint32_t k = 0; k < csize; k++) hv[u] += *cluster.map_shared_rank(&sm.hist[(S_NB - 1) - tid * S_BPT - u], k);
                    own += hv[u];
                }
            } else
#pragma unroll
            for (int u = 0; u < S_BPT; u++) { hv[u] = sm.hist[(S_NB - 1) - tid * S_BPT - u]; own += hv[u]; }
            uint32_t total;
            uint32_t above = sblock_excl_scan_u32(own, &total, sm.scan_u);
#pragma unroll
            for (int u = 0; u < S_BPT; u++) {
                if (above < need && need <= above + hv[u]) sm.sel_bucket = (uint32_t)((S_NB - 1) - tid * S_BPT - u);
                above += hv[u];
            }
            __syncthreads();
            const uint32_t bsel = sm.sel_bucket;
            return (bsel >= 1u && scb > 0.0f) ? lo_v + ((float)bsel - 1.0f) / scb : lo_v;
        };
        float bound = NAN;   // CL: at least top_k logits of the row reach it (NaN: not known yet)
        if (CL) {
            // Every CTA bounds its own share of the top-k from below, hands that, its part of the region table and its
            // numbers to all the others, and combines what it gets: one barrier.  (The share: top-k by the CTA's part of the
            // row's logits, so that the shares of all CTAs together make k.  With equal shares the CTA with the fewest pieces
            // sets the bound: top-k 1024 of 50256 on four CTAs listed more candidates than there is room for.  A bound over
            // all histograms is tighter, but takes a second barrier and a trip to every other CTA.)
            cg::cluster_group cluster = cg::this_cluster();
            if (!greedy) {
                const uint32_t mine = (n_full > crank ? ((n_full - 1u - crank) >> (__ffs((int)csize) - 1)) + 1u : 0u) * S_PIECE + (my_tail ? V - n_full * S_PIECE : 0u);
                const uint32_t share = (uint32_t)(__fdividef((float)(top_k * mine), (float)V) * 1.000001f) + 1u;   // (rounded up, whatever the quotient's error; top-k is 1024 at most)
                if (mine == 0u) bound = INFINITY;
                if (mine && n_fin >= share) bound = kth_bound(share, key_to_float(lo_key), lm, false);   // CTA-uniform
                else __syncthreads();   // (the entries' sums are complete)
            }
            cluster.barrier_wait();   // all of them run
            if (!greedy) {
#pragma unroll 1
                for (uint32_t r = tid; r < n_regions; r += SNT) {
                    const uint32_t q = r / SNW;
                    if ((q < n_full ? q % csize : tail_owner) != crank) continue;
                    float ra = sm.reg_a[r], rb = sm.reg_b[r];
                    if (has_bits && sm.reg_t[r] > 0.0f) {   // with the entries, from now on relative to this CTA's maximum
                        rb = (rb > 0.0f ? rb * ex2_approx_ftz((ra - lm) * sc) : 0.0f) + sm.reg_t[r];
                        ra = lm;
                        sm.reg_a[r] = ra; sm.reg_b[r] = rb;
                    }
                    for (uint32_t k = 0; k < csize; k++) {
                        if (k == crank) continue;
                        *cluster.map_shared_rank(&sm.reg_a[r], k) = ra;
                        *cluster.map_shared_rank(&sm.reg_b[r], k) = rb;
                    }
                }
            }
            if ((uint32_t)tid < csize) {
                *cluster.map_shared_rank(&sm.xk[crank], tid) = gkey;
                *cluster.map_shared_rank(&sm.xlo[crank], tid) = lo_key;
                *cluster.map_shared_rank(&sm.xfin[crank], tid) = n_fin;
                *cluster.map_shared_rank(&sm.xflag[crank], tid) = (nonfinite ? 1u : 0u) | (defer_row ? 2u : 0u);
                *cluster.map_shared_rank(&sm.xb[crank], tid) = bound;
            }
            cluster.sync();
            gkey = 0u; lo_key = 0xffffffffu; n_fin = 0u; nonfinite = false; defer_row = false;
            float low = INFINITY;
            bool known = true;
            for (uint32_t k = 0; k < csize; k++) {
                gkey = umax(gkey, sm.xk[k]); lo_key = umin(lo_key, sm.xlo[k]); n_fin += sm.xfin[k];
                nonfinite |= (sm.xflag[k] & 1u) != 0u; defer_row |= (sm.xflag[k] & 2u) != 0u;
                low = fminf(low, sm.xb[k]); known &= sm.xb[k] == sm.xb[k];
            }
            bound = known ? low : NAN;
        }
        const bool any = gkey != 0u;
        const float m = any ? key_to_float(gkey) : -INFINITY;
        const int status = any ? ROW_OK : ROW_EMPTY;
        if (writer) atomicAdd(sl.p1_done, 1u);
        // ---- argmax: the lowest id that holds the maximum.  Every thread whose own maximum is the row's looks at
        // the lowest of its pieces that holds it once more (the penalised values are in place by now).
        if (any && !nonfinite && !(gflags & 2u)) {
            // (the piece code is a warp-wide operation, so a warp goes through the pieces its lanes ask for one by
            // one; nearly always that is a single piece of a single warp)
            unsigned pending = __ballot_sync(FULL, order_key(tmx) == gkey);
#pragma unroll 1
            while (pending) {   // warp-uniform
                const uint32_t q = __shfl_sync(FULL, tqx, __ffs(pending) - 1);
                Raw<BF16> raw;
                raw_load_tail<BF16>(raw, rowp + ((size_t)q * S_PIECE + lane_e0) * ESZ, q * S_PIECE + lane_e0, V);
                float x[S_EPT];
                raw_unpack<BF16>(x, raw);
                if (has_bits) fix_x<BF16, true, true, CL>(sm, x, q, region_word<true>(sm, q * SNW + (uint32_t)w)); else fix_x<BF16, false, true, CL>(sm, x, q, 0u);
                const bool mine = ((pending >> lane) & 1u) && tqx == q;
                if (mine) {
                    int j0 = 0;
#pragma unroll
                    for (int j = S_EPT - 1; j >= 0; j--) if (x[j] == m) j0 = j;
                    atomicMin(&sm.amax, elem_id<BF16>(q * S_PIECE + lane_e0, j0));
                }
                pending &= ~__ballot_sync(FULL, mine);
            }
            for (uint32_t e = tid; e < n_ent; e += SNT)
                if (sm.ent_x[e] == m) atomicMin(&sm.amax, sm.ent_id[e]);
            __syncthreads();
        }
        uint32_t amax = any ? sm.amax : 0u;
        if (defer_row || nonfinite || (gflags & 2u) || greedy || !any) {
            if (CL) {   // the lowest id over all CTAs; the first CTA writes the row
                cg::cluster_group cluster = cg::this_cluster();
                if (tid == 0) *cluster.map_shared_rank(&sm.xam[crank], 0) = sm.amax;
                cluster.sync();
                if (crank != 0u) continue;
                uint32_t am_all = 0xffffffffu;
                for (uint32_t k = 0; k < csize; k++) am_all = umin(am_all, sm.xam[k]);
                amax = any ? am_all : 0u;
            }
            if (defer_row) {   // (cluster mode only) a CTA could not index the history: the work list takes the row
                if (writer) sl.work_rows[atomicAdd(sl.work_count, 1u)] = row;
                continue;
            }
            if (writer && a.tp_records) {
                if (nonfinite) {
                    tp_write_head(a, row, NAN, 0.0f, 0u, ROW_NONFINITE, 0u);
                    if (a.faulted) atomicAdd(a.faulted, 1ull);
                } else if (gflags & 2u) tp_write_head(a, row, -INFINITY, 0.0f, 0u, ROW_DEAD, 0u);
                else tp_write_head(a, row, m, 0.0f, 0u, ROW_OK, amax);   // greedy or empty: maximum + argmax alone
            } else if (writer) {
                if (nonfinite) {
                    a.token[row] = 0; a.status[row] = ROW_NONFINITE; if (a.drew) a.drew[row] = 0;
                    if (a.faulted) atomicAdd(a.faulted, 1ull);
                } else if (gflags & 2u) {
                    a.token[row] = 0; a.status[row] = ROW_DEAD; if (a.drew) a.drew[row] = 0;
                } else {
                    a.token[row] = amax; a.status[row] = status;
                    if (a.drew) a.drew[row] = 0;
                    if (a.argmax) a.argmax[row] = amax;
                    if (a.row_max) a.row_max[row] = m;
                    if (a.sumexp) a.sumexp[row] = 0.0f;
                    if (a.total) a.total[row] = 0.0f;
                    if (a.n_kept) a.n_kept[row] = 0u;
                }
            }
            PGS_STICK(3);
            continue;
        }

        PGS_STICK(6);   // reductions + argmax
        // numerators are 2^(x * sc - m * sc) here: where that overflows, the row goes to the kernels that subtract first
        if (!(fabsf(m) * sc < 1e38f)) {   // CTA-uniform; CL: the same in all CTAs
            if (writer) sl.work_rows[atomicAdd(sl.work_count, 1u)] = row;
            continue;
        }
        // ---- top-k bound
        const float t = fmaxf(temp, 1e-9f);
        float cut = -INFINITY;
        if (n_fin >= top_k) {   // CTA-uniform; CL: the same in all CTAs
            if (!(bound == bound)) {
                if (CL) {   // some CTA has too few maxima for its share (a mask that leaves its pieces empty)
                    __syncthreads();
#pragma unroll
                    for (int u = 0; u < S_BPT; u++) sm.hist[u * SNT + tid] = 0u;
                    if (tid == 0) sm.sel_bucket = 0u;
                    __syncthreads();
                }
                bound = kth_bound(top_k, key_to_float(lo_key), m, true);
            }
            // every logit whose probability could still tie with the k-th one stays above the cut
            const float delta = 4.8e-7f * (fabsf(m - bound) + 4.0f * t) + 4.8e-7f * (fabsf(bound) + fabsf(m));
            cut = bound - delta;
        }
        PGS_STICK(7);   // top-k bound
        // numerator = 2^(x * sc + c): c = -m * sc as c_hi + c_lo (c_lo only when it matters: the numerators then keep
        // the reference's scale to 1e-7, which the fold needs where many logits are equal); what is left of c scales
        // the final sum
        const double scale_d = BF16 ? (double)sc + (double)ctl.sc_lo : (double)sc;
        const double c_d = -(double)m * scale_d;
        const float c_hi = (float)c_d;
        float c_lo = (float)(c_d - (double)c_hi);
        if (!BF16 && fabsf(c_lo) < 1e-7f) c_lo = 0.0f;
        const double c_rest = c_d - (double)c_hi - (double)c_lo;
        if (tid == 0) { sm.pa.c_hi = c_hi; sm.pa.c_lo = c_lo; sm.pa.cut_f = fmaxf(cut, -3.4e38f); }   // masked entries (-inf) are never candidates

        // ---- where the fold stands at every warp region.  The plain sums overestimate the fold's running value
        // by up to a few 1e-4 (the small terms it drops), so a region takes the quick path only if the whole
        // interval [start * (1 - slack), end * (1 + slack)], slack >= 2^-9, lies inside one binade.
        {
            float carry = 0.0f;
#pragma unroll 1
            for (uint32_t r0 = 0; r0 < n_regions; r0 += SNT) {   // CTA-uniform trip count
                const uint32_t r = r0 + (uint32_t)tid;
                float P = 0.0f;
                if (r < n_regions && sm.reg_b[r] > 0.0f) P = sm.reg_b[r] * ex2_approx_ftz((sm.reg_a[r] - m) * sc);
                if (!CL && has_bits && r < n_regions) P += sm.reg_t[r];
                float tot;
                const float pre = carry + sblock_excl_scan_f32(P, &tot, sm.scan_f);
                if (r < n_regions) {
                    // (the plain sums carry the rounding of their exponents' constant: 2^-24 of |max * sc|)
                    const float slack = 0.001953125f + 1e-7f * fabsf(m * sc);
                    const float lo_e = pre * (1.0f - slack), hi_e = (pre + P) * (1.0f + slack);
                    const uint32_t kb = f2u(lo_e) & 0x7f800000u;
                    // quick: one binade for the whole region, and the region's own sum stays below that binade's
                    // lower end, so that no thread's additions from there can leave the binade either
                    const bool quick = kb != 0u && kb == (f2u(hi_e) & 0x7f800000u) && P * (1.0f + slack) < 0.999f * u2f(kb);
                    sm.reg_a[r] = quick ? u2f(kb) : 0.0f;
                    sm.reg_b[r] = pre;
                    // A numerator below half an ulp of the running value leaves it unchanged, and lo_e never exceeds the
                    // running value: a logit with x * scale + c < exponent(lo_e) - 24 (less a margin for the hardware
                    // exp2) adds exactly nothing.  In units of logits:
                    float thr = -INFINITY;
                    if (kb != 0u) {
                        const double lim = (double)((int)(kb >> 23) - 127 - 24) - 0.02;
                        thr = (float)((lim - c_d) / scale_d);
                        thr -= 4e-7f * fabsf(thr) + 1e-30f;
                    }
                    sm.reg_t[r] = thr;
                }
                carry += tot;
                __syncthreads();   // scan_f is reused by the next round; after the last one the table and PassArgs are complete
            }
        }
        PGS_STICK(3);   // fold table

        // ================================================================ pass 2 (L2, first piece first)
        p2_entries<BF16, CL>(sm, n_ent);
        if (my_tail) {
            Raw<BF16> raw;
            raw_load_tail<BF16>(raw, rowp + ((size_t)n_full * S_PIECE + lane_e0) * ESZ, n_full * S_PIECE + lane_e0, V);
            FoldAcc fa;
            fa.accd = 0.0; fa.cur_n = 0ull; fa.cur_bb = 0u;
            if (has_bits) p2_piece<BF16, true, true, CL>(sm, raw, n_full, fa); else p2_piece<BF16, false, true, CL>(sm, raw, n_full, fa);
            fa.flush();
            if (lane == 0) sm.wacc[w] += fa.accd;
        }
        if (n_full > 0u) {
            if (has_bits) pass2_whole<BF16, true, CL>(sm); else pass2_whole<BF16, false, CL>(sm);
        }
        __syncthreads();   // the candidate list and the warps' shares are complete
        PGS_STICK(4);   // pass 2
        double s_d = lane < SNW ? sm.wacc[lane] : 0.0;
#pragma unroll
        for (int o = 16; o; o >>= 1) s_d += __shfl_xor_sync(FULL, s_d, o);
        if (CL) {   // the fold shares and the argmax candidates of all CTAs meet in the first one
            cg::cluster_group cluster = cg::this_cluster();
            if (tid == 0) { *cluster.map_shared_rank(&sm.xs[crank], 0) = s_d; *cluster.map_shared_rank(&sm.xam[crank], 0) = sm.amax; }
            cluster.sync();
            if (crank != 0u) continue;
            s_d = 0.0;
            uint32_t am_all = 0xffffffffu;
            for (uint32_t k = 0; k < csize; k++) { s_d += sm.xs[k]; am_all = umin(am_all, sm.xam[k]); }
            amax = am_all;
        }
        const float S = (float)(s_d * exp2(c_rest));
        const uint32_t n_cand = sm.cand_n;
        if (n_cand > (uint32_t)F_MCAP) {   // CTA-uniform
            if (writer) { sl.work_rows[atomicAdd(sl.work_count, 1u)] = row; }
            continue;
        }
        if (a.tp_records) {   // CTA-uniform
            if (n_cand > (uint32_t)SNT) {
                if (writer) { sl.work_rows[atomicAdd(sl.work_count, 1u)] = row; }
                continue;
            }
            semit_tp(sm, a, row, n_cand, m, S, amax);
        } else {
            cta_finish<SNT>(sm.fin, sm.exp_tab, a, row, V, sm.cand_id, sm.cand_x, n_cand, m, t, S, top_k, ctl.top_p, ctl.u01, amax,
                            status);
        }
        PGS_STICK(5);   // finish
    }
    if (sl.prof && tid == 0)
#pragma unroll 1
        for (int i = 0; i < 16; i++) sl.prof[blockIdx.x * 16 + i] += sm.prof_acc[i];
}

size_t stream_smem_bytes() { return sizeof(StreamSmem<false>); }
uint32_t stream_threads() { return SNT; }

template <bool BF16, bool CL, bool LONG>
static cudaError_t configure_one() {
    cudaError_t e = cudaFuncSetAttribute(stream_row_kernel<BF16, CL, LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StreamSmem<LONG>));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(stream_row_kernel<BF16, CL, LONG>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}
template <bool BF16, bool CL>
static cudaError_t configure_both() {
    const cudaError_t e = configure_one<BF16, CL, false>();
    return e != cudaSuccess ? e : configure_one<BF16, CL, true>();
}

cudaError_t configure_stream() {
    cudaError_t e = configure_both<false, false>();
    if (e == cudaSuccess) e = configure_both<true, false>();
    if (e == cudaSuccess) e = configure_both<false, true>();
    if (e == cudaSuccess) e = configure_both<true, true>();
    return e;
}

// CTAs of this kernel that one SM holds (of either length of row)
cudaError_t stream_ctas_per_sm(int* out) {
    int longs = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, stream_row_kernel<false, false, false>, SNT, sizeof(StreamSmem<false>));
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&longs, stream_row_kernel<false, false, true>, SNT, sizeof(StreamSmem<true>));
    if (longs < *out) *out = longs;
    return e;
}

// Clusters of `csize` CTAs of this kernel that the device holds at once (csize 2, 4 or 8)
template <bool LONG>
static cudaError_t max_clusters(int csize, int* out) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)csize, 1, 1);
    cfg.blockDim = dim3(SNT, 1, 1);
    cfg.dynamicSmemBytes = sizeof(StreamSmem<LONG>);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)csize; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(out, stream_row_kernel<false, true, LONG>, &cfg);
}
cudaError_t stream_max_clusters(int csize, int* out) {
    int longs = 0;
    cudaError_t e = max_clusters<false>(csize, out);
    if (e == cudaSuccess) e = max_clusters<true>(csize, &longs);
    if (longs < *out) *out = longs;
    return e;
}

template <bool BF16, bool CL>
static cudaError_t launch_length(const RowArgs& a, const StreamLaunch& sl, cudaLaunchConfig_t& cfg) {
    const bool is_long = a.vocab > (uint32_t)S_SHORT_VOCAB;
    cfg.dynamicSmemBytes = is_long ? sizeof(StreamSmem<true>) : sizeof(StreamSmem<false>);
    return is_long ? cudaLaunchKernelEx(&cfg, stream_row_kernel<BF16, CL, true>, a, sl) : cudaLaunchKernelEx(&cfg, stream_row_kernel<BF16, CL, false>, a, sl);
}
// csize == 1: one CTA per row, `grid` CTAs.  csize > 1: `grid` clusters of csize CTAs, one cluster per row at a time.
cudaError_t launch_stream(const RowArgs& a, const StreamLaunch& sl, uint32_t grid, uint32_t csize, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid * csize, 1, 1);
    cfg.blockDim = dim3(SNT, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = csize; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = csize > 1u ? 2 : 1;
    if (csize > 1u) return a.dtype == 0 ? launch_length<false, true>(a, sl, cfg) : launch_length<true, true>(a, sl, cfg);
    return a.dtype == 0 ? launch_length<false, false>(a, sl, cfg) : launch_length<true, false>(a, sl, cfg);
}

}  // namespace pgs
