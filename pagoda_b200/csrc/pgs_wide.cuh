// Workspace and launch block of the wide kernel (pgs_wide.cu), shared with the host launcher.
#pragma once

#include <stdint.h>

#include "pgs_args.cuh"

namespace pgs {

constexpr int W_NT = 1024;              // threads per CTA, one CTA per SM
constexpr int W_REGION = 512;           // consecutive logits of one warp
constexpr int W_MAX_VOCAB = 1 << 20;
constexpr int W_MAX_REGIONS = W_MAX_VOCAB / W_REGION;
constexpr int W_MAX_HIST = 2048;
constexpr int W_CHUNK = 64;             // rows in flight together, at most
constexpr int W_BUCKETS = 41 * 256;     // probabilities by exponent (2^-40 .. 1) and eight mantissa bits
constexpr int W_TERMS = 64;             // segments of a row whose terms the region phase leaves for the fold
constexpr int W_KMAX = 1024;            // top-k up to which the second pass lists the candidates
constexpr int W_OWN = 16;               // words of WideLaunch::own
constexpr int W_SORT = 4096;            // entries of a bucket that one CTA sorts

// One row of the chunk.
struct WideRow {
    const char* rowp;
    const uint32_t* mw;
    float temp, t, freq, pres, rep, top_p, u01;
    uint32_t top_k, gflags, h0, nh, row;
    uint32_t entries;        // history entries (and EOS fix) of the row, grouped by region
    uint32_t nonfinite;      // set by the first pass
    uint32_t state;          // WS_*
    float m, S, total;
    uint32_t amax, max_region;   // max_region: the first region that holds the maximum
    uint32_t cut, n_list;    // entries in buckets >= cut
    float cut_x;             // rows with a short top-k: the second pass lists the logits from here on (n_list of them)
    uint32_t n_terms;        // segments whose terms are in WideLaunch::terms
    float p_thr;             // kept: p > p_thr, or p == p_thr and id <= id_thr
    uint32_t id_thr, n_kept;
};
enum : uint32_t { WS_FIRST = 0u, WS_SUM = 1u, WS_SELECT = 2u, WS_TOTAL = 3u, WS_DONE = 4u };

struct WideLaunch {
    // The workspace's parts: as many as scratch slots (min(rows of the handle, SMs)) for steps, as SMs for scoring.  The grid uses the
    // first `chunk` of them, one for every row in flight; with one CTA per row each CTA has the part of its number, so that
    // min(CTAs, rows) must not be more than there are.
    WideRow* row;               // [parts]
    float2* reg;                // [parts][n_regions]: a region's maximum, its plain sum
    float4* cell;               // [parts][n_regions]: the maxima of four parts of the region
    uint2* seg;                 // [parts][n_regions]: increments in ulps, binade (0: add term by term)
    float* pre;                 // [parts][n_regions]: estimate of the running value at the region's start
    float* terms;               // [parts][W_TERMS][W_REGION]: terms of segments that are added one by one
    uint32_t* ent_id;           // [parts][W_MAX_HIST + 32]
    float* ent_xn;
    uint32_t* rs;               // [parts][n_regions + 1]
    uint32_t* hist;             // [parts][W_BUCKETS]: counts, then list positions
    unsigned long long* list;   // [parts][list_stride] (the general kernel's sort buffer): probability bits and id
    uint32_t* sync;             // [0] barrier arrivals, [1] rows without results where a barrier was given up, [2] rows that select by the histogram, [3] rows in the last pass, [4] CTAs that have left, [5] CTAs that have joined, [6] how many take part
    // Combinations of kinds (pgs_kinds.cuh) that are done by the general kernel's code, one CTA per row: here ([0]: at most a chunk of
    // rows, [1]: more; [2]: one listed row that would have a CTA of its own, [3]: two), or by the general kernel in front of this one.
    uint32_t kinds_row[4], kinds_front, look;   // look: bits are set, 1: in kinds_row[0, 1] or kinds_front, 2: in kinds_row[2, 3]
    uint32_t local;             // 1: one CTA per row, with the part of the workspace that has the CTA's number; 2: by the number of listed rows
    uint32_t* own;              // [CTAs][W_OWN]: what `sync`, `left_count` and `left_rows` are for the grid
    uint32_t polls;             // limit of a barrier's wait
    unsigned long long* gave_up; // rows that ended without results because one ran out
    uint32_t chunk;             // rows that the grid takes at a time (<= W_CHUNK, and what the workspace holds)
    uint32_t reg_stride, rs_stride, list_stride;
    uint32_t* left_rows;        // rows left to the general kernel
    uint32_t* left_count;
    // log-softmax scoring in place of sampling (score != 0)
    uint32_t score;
    const uint32_t* ids;
    float* out_gather;
    float* out_full;
    uint32_t* done;             // host memory: gets done_value when the launch no longer uses its workspace
    uint32_t done_value;
};

}  // namespace pgs
