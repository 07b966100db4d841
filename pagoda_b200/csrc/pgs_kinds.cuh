// Which rows are done by the wide kernel (pgs_wide.cu) and which by one CTA each of the general one (pgs_general.cuh).  Both give the same bits; the
// choice is which is quicker for a batch, from what its rows ask for.
#pragma once

#include "pgs_args.cuh"
#include "pgs_wide.cuh"

namespace pgs {

// What rows ask for, as far as it decides that; a batch: all of its rows together.
enum : uint32_t { WK_SAMPLED = 1u, WK_HIST = 2u, WK_OPEN = 4u, WK_SORT = 8u, WK_LONG = 16u };
// the combinations that there are, one bit each: greedy; sampled, and that by the histogram, with top-k off, sort, or both
constexpr uint32_t WK_SHORT = 1u | 1u << WK_SAMPLED | 1u << (WK_SAMPLED | WK_HIST) | 1u << (WK_SAMPLED | WK_HIST | WK_OPEN) |
                              1u << (WK_SAMPLED | WK_HIST | WK_SORT) | 1u << (WK_SAMPLED | WK_HIST | WK_OPEN | WK_SORT);
constexpr uint32_t WK_POSSIBLE = WK_SHORT | WK_SHORT << WK_LONG;

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t row_kind(const RowArgs& a, uint32_t row) {
    const float temp = a.temperature ? a.temperature[row] : 0.0f, top_p = a.top_p ? a.top_p[row] : 1.0f;
    const uint32_t k = a.top_k ? a.top_k[row] : 0u, n_regions = (a.vocab + W_REGION - 1) / W_REGION;
    const uint32_t nh = a.hist_offsets ? a.hist_offsets[row + 1] - a.hist_offsets[row] : 0u;
    const uint32_t is_long = nh > (uint32_t)W_MAX_HIST ? WK_LONG : 0u;
    if (temp < 1e-5f) return is_long;
    const bool open = k == 0u || k >= a.vocab, big = open || k > (uint32_t)W_KMAX;
    return WK_SAMPLED | is_long | (big || k > 4u * n_regions ? WK_HIST : 0u) | (open ? WK_OPEN : 0u) | (big && !(top_p >= 1.0f) ? WK_SORT : 0u);
}
// the kinds of the first n rows (of the list, or of the batch); `slot`: zero, with a barrier behind it.  A barrier is needed
// before the result is in `slot`.
__device__ __forceinline__ void batch_kinds(const RowArgs& a, uint32_t n, uint32_t threads, uint32_t* slot) {
    uint32_t kinds = 0u;
    for (uint32_t i = threadIdx.x; i < n; i += threads) kinds |= row_kind(a, a.work_rows ? a.work_rows[i] : i);
    kinds = __reduce_or_sync(0xffffffffu, kinds);
    if ((threadIdx.x & 31u) == 0u && kinds) atomicOr(slot, kinds);
}
#endif

// Whether the wide kernel takes n listed rows one CTA each, `parts` at a time, and not with the whole grid on `chunk` at a time.
// Listed rows have no top-k as a rule, and often top-p.  us with a CTA per row / with the grid, top-p off and 0.9: 1 x 4096 57 / 67,
// 16 x 16384 64 / 75 and 65 / 105, 64 x 16384 69 / 81 and 70 / 126, 16 x 50256 97 / 82 and 95 / 120, 64 x 50256 96 / 99 and 112 / 167,
// 64 x 151936 149 / 147 and 223 / 244, 148 x 4096 60 / 212, 256 x 151936 333 / 574 and 464 / 954.  (The line goes by number and length
// alone and is drawn for rows without top-p; with it a few that the grid gets would be quicker on a CTA each, 16 x 50256 by 20 %.)
__host__ __device__ __forceinline__ bool listed_one_cta_each(uint32_t n, uint32_t chunk, uint32_t parts, uint32_t V) {
    const float v = 1e-6f * (float)V;
    const float by_rows = (float)((n - 1u) / parts + 1u) * (58.0f + 800.0f * v + 2.5f * v * (float)(n < parts ? n : parts));
    const float grid = (float)((n - 1u) / chunk + 1u) * (75.0f + 10.0f * v * (float)(n < chunk ? n : chunk));
    return V > 1024u && by_rows < grid;
}

// Those of the combinations `of` for which one CTA per row is the quicker way for `n` rows.  Short rows do not pay for the grid's
// barriers, and batches of many rows go through the grid in chunks of 64 where one CTA per row takes an SM count at a time.
// us of one row on one CTA: greedy 9 + 0.37 per thousand logits, sampled 47 + 2.2, without top-k 5 more per thousand, with a
// sort for top-p 60 + 18; of a chunk: greedy 27, sampled 44 (70 where the threshold needs the histogram), 4 per million
// logits.  Measured (one CTA per row / grid): top-k 50, 1 x 1000 48 / 68, 64 x 4096 64 / 83, 64 x 16384 93 / 54, 128 x 16384
// 94 / 102, 256 x 50256 338 / 240, 1024 x 16384 576 / 769; greedy 1 x 1000 9 / 27, 64 x 50256 31 / 35, 1 x 151936 64 / 27,
// 256 x 50256 64 / 126, 256 x 151936 217 / 166; no top-k 16 x 1000 59 / 68, 16 x 16384 160 / 91, with top-p 1 x 1000 76 / 71,
// 16 x 4096 161 / 78.  Rows with a history beyond the workspace end on one CTA either way (4 of 50256: 187 at once, 239
// behind the phases).
//
// WAY_ROWS: the wide kernel takes a CTA per row itself (wide_row_by_row), behind the general kernel; WAY_ROWS_ALONE: it does,
// and runs the general kernel's code where that is quicker.  us of one row, as many at a time as there are SMs, general /
// wide, v in thousands of logits: greedy 9 + 0.37 v / 14 + 0.12 v (alone 5 + 0.45 v / 13 + 0.16 v); sampled 48 + 2.9 v (one
// row 43 + 1.6 v, two 46 + 2.3 v) / 33 + 0.55 v, 57 + 0.3 v (alone 53 + 0.3 v) where the threshold needs the histogram;
// without top-k 50 + 6 v / 57 + 0.7 v, a sort for top-p 60 + 18 v / 60 + v.  Measured, each on its own: k 50 1 x 1100 43 / 55,
// 1 x 6000 51 / 57, 51 x 2040 59 / 55, 148 x 4096 64 / 56, 148 x 16385 104 / 43; k 5 1 x 1100 41 / 33, 148 x 3000 60 / 36; no
// top-k 1 x 1100 35 / 52, 1 x 3000 47 / 52, 2 x 1500 63 / 52, 148 x 3000 93 / 61; with top-p 1 x 1100 65 / 52, 148 x 4096 158
// / 53; 2100 history ids 148 x 4096 83 / 100, 200 x 50257 388 / 503; greedy 148 x 4096 6.2 / 14.3, 64 x 16385 12.3 / 16.7, 148
// x 50257 31 / 22.  (The lines for greedy rows end the look at what rows ask for, 4 us with both kernels, where sampled rows
// need it no more: 64 x 16385 with top-k 42 / 47, 200 x 16385 76 / 82.)  Up to 2048 logits and beyond a chunk of rows the look
// costs most of them more than it gives (210 x 1719 with top-k 27 100 / 103).
enum KindsWay { WAY_GRID, WAY_ROWS, WAY_ROWS_ALONE };
inline uint32_t kinds_one_cta_each(uint32_t of, uint32_t n, uint32_t chunk, uint32_t ctas, uint32_t V, KindsWay way) {
    const bool by_rows = way != WAY_GRID;
    if (V <= 1024u || (by_rows && V <= 2048u && n > chunk)) return of;   // (the slowest kind is as quick either way, and nothing has to be looked at)
    const float v = (float)V, waves = (float)((n - 1u) / ctas + 1u), chunks = (float)((n - 1u) / chunk + 1u);
    const float m = 1e-6f * v * (float)(n < chunk ? n : chunk), together = (float)(n < ctas ? n : ctas);
    uint32_t mask = 0u;
    for (uint32_t left = of; left; left &= left - 1u) {
        const uint32_t kinds = (uint32_t)__builtin_ctz(left);
        float row, grid;
        if (kinds & WK_SAMPLED) {
            row = kinds & WK_SORT ? 60.0f + 0.018f * v : 47.0f + 0.0022f * v + (kinds & WK_OPEN ? 0.005f * v : 0.0f);
            grid = (kinds & WK_HIST ? 70.0f : 44.0f) + 4.0f * m;
        } else {
            row = 9.0f + 3.7e-4f * v + 1.5e-6f * v * together;
            grid = 27.0f + 1.65f * m;
        }
        if (by_rows) {
            const float v3 = 1e-3f * v;
            if (!(kinds & WK_SAMPLED)) {
                if (way == WAY_ROWS_ALONE) row = 5.0f + 0.45f * v3;
                grid = way == WAY_ROWS_ALONE ? 13.0f + 0.16f * v3 : 14.0f + 0.12f * v3;
            } else if (kinds & WK_SORT) grid = 60.0f + v3;
            else if (kinds & WK_OPEN) {
                row = n == 1u && V <= 3100u || n == 2u && V < 1100u ? 0.0f : 50.0f + 6.0f * v3;
                grid = 57.0f + 0.7f * v3;
            } else {
                row = n == 1u ? 43.0f + 1.6f * v3 : n == 2u ? 46.0f + 2.3f * v3 : 48.0f + 2.9f * v3;
                grid = kinds & WK_HIST ? (way == WAY_ROWS_ALONE ? 53.0f : 57.0f) + 0.3f * v3 : 33.0f + 0.55f * v3;
            }
            grid *= waves;
        } else grid *= chunks;
        if (kinds & WK_LONG) grid += by_rows ? waves * row : row;   // (ends in the general kernel's code either way)
        if (waves * row < grid) mask |= 1u << kinds;
    }
    return mask;
}

}  // namespace pgs
