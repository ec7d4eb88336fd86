// Traceback kernels (host interface): one optimal path per aligned pair.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "sw_strips.h"

namespace gbsw {

struct TraceParams {
    const uint8_t* ref;
    const int64_t* ref_off;
    const uint8_t* query;
    const int64_t* query_off;
    const int32_t* score;        // the pairs' results (int32 SoA)
    const int32_t* ref_begin;
    const int32_t* ref_end;
    const int32_t* query_begin;
    const int32_t* query_end;
    int64_t first, count;        // this launch: pairs [first, first + count)
    int protein;
    int match, mismatch, open, ext;
    const int* aa_matrix;        // protein: 25x25 padded, row = first index
    const int* aa_encoding;      // protein: 91 entries
    const int64_t* dir_off;      // per pair: first direction word within `dir` (this launch)
    uint32_t* dir;
    const int64_t* bnd_off;      // per pair: first strip-boundary entry within `bnd` (this launch)
    int2* bnd;
    const int64_t* order;        // the pairs of this launch in the order its groups take them (ids), or
                                 // nullptr: first, first + 1, ...
    const int64_t* slot_off;     // per pair: first operation slot within `ops`
    uint32_t* ops;
    int32_t* nops;               // per pair: operations written
    int32_t* path_score;         // per pair: H(k, m) of the path
    int* error;
    int* queue;                  // int16 kernel: work-queue counter (0 before the launch)
    int neg, top;                // int16 kernel: Trace16Limits
};

// Error bit: a path's end value differs from the pair's score.
constexpr int kErrTrace = 8;

// Columns per lane of the traceback kernel (one 4-bit direction code each, so a
// lane's row is one 16- or 32-bit word), lanes per pair's group and columns per
// strip.  With one 32-lane warp per pair, 8 columns took 14.5 ms on the
// 100,000-pair DNA batch and 4 columns 15.0 ms: narrower strips waste fewer
// columns past a segment's end, but 8 columns amortise the per-row shuffles
// and stores over twice the cells.  Groups of 8 lanes (64-column strips, four
// pairs per warp) waste fewer still: a 150-300-column segment in 256-column
// strips, plus 31 fill steps per strip, computes 1.7 x its cells, in
// 64-column strips with 7 fill steps 1.2 x.
#ifndef GBSW_TRACE_COLS
#define GBSW_TRACE_COLS 8
#endif
#ifndef GBSW_TRACE_LANES
#define GBSW_TRACE_LANES 8
#endif
constexpr int kTraceColsPerLane = GBSW_TRACE_COLS;
constexpr int kTraceLanes = GBSW_TRACE_LANES;
static_assert(kTraceColsPerLane == 4 || kTraceColsPerLane == 8, "a lane's row fills a 16- or 32-bit word");
static_assert(kTraceLanes == 8 || kTraceLanes == 16 || kTraceLanes == 32, "groups of 8, 16 or 32 lanes");
constexpr int kTraceCols = kTraceLanes * kTraceColsPerLane;

// Direction memory, in 32-bit words, of a pair whose segment is m reference x k
// query symbols: per strip and row, one 4-bit code per column.
__host__ __device__ inline int64_t trace_dir_words(int m, int k) {
    return (int64_t)((m + kTraceCols - 1) / kTraceCols) * (int64_t)k * (kTraceCols / 8);
}

cudaError_t launch_trace(const TraceParams& p, cudaStream_t stream);

// ---- the int16x2 kernel (trace_strips.cu) ----
// Columns a virtual lane holds and columns of a strip.
constexpr int kTrace16Cols = 4;
constexpr int kTrace16Width = strip_width(kTrace16Cols);
// The limits of its values, from the scoring (`best`: the largest score of an
// aligned pair of symbols).  neg: its -inf, as low as the rows of the pipeline's
// fill (131 at most, each up to |ext| lower than the one before) leave room for.
// top: a cell may lie above its upper neighbour by up to best + |open|, so a kernel
// that looks at every sixteenth row sees a value above top before one can wrap.
struct Trace16Limits {
    int neg, top, best;
};
inline Trace16Limits trace16_limits(int best, int open, int ext) {
    return {-32768 - 131 * ext - open + 160, 32767 - 20 * (best - open), best};
}

// Threads of a walk block and lanes per walk.
constexpr int kWalkThreads = 128;
constexpr int kWalkLanes = 8;

// Whether the scoring suits it: int8 scores, match at least mismatch and at most
// 128 above it (DNA), open <= ext (the gap row then follows from the recurrence) and
// small gaps.
inline bool trace16_scores_ok(bool int8_scores, int match, int mismatch, bool protein, int open, int ext) {
    return int8_scores && (protein || (match >= mismatch && match - mismatch <= 128)) && open <= ext && ext >= -16 && open >= -256;
}
// Whether a pair's segment does: every real value lies above -inf, and none above
// top if the score is the pair's (a prefix of the path aligns two substrings, so no
// value exceeds the best local score; results of other inputs are told from it by
// the kernel's own look).
inline bool trace16_pair_ok(const Trace16Limits& lim, int m, int k, int score, int open, int ext) {
    return ((int64_t)lim.best * (m < k ? m : k) <= lim.top || score <= lim.top) &&
           2 * (int64_t)open + (int64_t)ext * ((int64_t)m + k) >= lim.neg + 256;
}
// Direction words (32 bits) of a strip of `lanes` virtual lanes and `pairs` row pairs:
// two per lane and step, steps rounded up to four.
__host__ __device__ inline int64_t trace16_strip_words(int pairs, int lanes) {
    return (int64_t)((pairs + lanes - 1 + 3) / 4) * 256;
}
// Direction words of a pair.
inline int64_t trace16_dir_words(int m, int k) {
    const int strips = (m + kTrace16Width - 1) / kTrace16Width, pairs = (k + 2) / 2;
    const int lanes = (m - (strips - 1) * kTrace16Width + kTrace16Cols - 1) / kTrace16Cols;
    return (strips - 1) * trace16_strip_words(pairs, 64) + trace16_strip_words(pairs, lanes);
}
// ---- its banded form for many DNA pairs (trace_band in trace_strips.cu) ----
// Lanes of a group, columns of its strips (two virtual lanes of 4 columns a lane).
constexpr int kBandLanes = 4;
constexpr int kBandWidth = 2 * kBandLanes * kTrace16Cols;
constexpr int kBandMaxRows = 2048;  // a group's edge buffer holds a word a row
constexpr int kBandNeg = -14000;    // its -inf
// Whether a pair's segment suits it: real values within 12,000 of 0 on both sides, so
// that the difference of any two values, -inf's among them, fits 16 bits (a value below
// -inf has lost at most 16 for each of the 39 rows and columns of a strip and its fill).
inline bool band_pair_ok(int match, int mismatch, int m, int k, int open, int ext) {
    const int64_t both = m < k ? m : k;
    return match > 0 && k < kBandMaxRows && m < kBandMaxRows && match * both <= 12000 &&
           (mismatch < 0 ? mismatch : 0) * both + 2 * (int64_t)open + (int64_t)ext * ((int64_t)m + k) >= -12000;
}
// The diagonals i - j that a path of this score can visit.  A path that leaves those
// between (0, 0) and (k, m) by d has d gap symbols more on both sides and d aligned
// pairs less: match (min(m, k) - d) + 2 open + (|m - k| + 2 d - 2) ext at best.
struct TraceBand {
    int lo, hi;
};
__host__ __device__ inline TraceBand trace_band_of(int m, int k, int score, int match, int open, int ext) {
    const int both = m < k ? m : k, apart = m < k ? k - m : m - k;
    const int64_t spare = (int64_t)(match * both + 2 * open + (apart - 2) * ext) - score;
    const int d = spare > 0 ? (int)spare / (match - 2 * ext) : 0;
    return {(k < m ? k - m : 0) - d, (k > m ? k - m : 0) + d};
}
// First and last row pair of a strip, and its direction words (two per lane and step,
// steps rounded up to four), the same for every strip of the pair.
__host__ __device__ inline int band_first_pair(const TraceBand& b, int strip) {
    const int i = strip * kBandWidth + b.lo;
    return (i > 0 ? i : 0) >> 1;
}
__host__ __device__ inline int band_last_pair(const TraceBand& b, int strip, int k) {
    const int i = strip * kBandWidth + kBandWidth + b.hi;
    return (i < k ? i : k) >> 1;
}
__host__ __device__ inline int64_t band_strip_words(const TraceBand& b, int k) {
    const int all = (k >> 1) + 1, most = (kBandWidth + b.hi - b.lo) / 2 + 2, pairs = all < most ? all : most;
    return (int64_t)((pairs + 2 * kBandLanes - 1 + 3) / 4) * (8 * kBandLanes);
}
cudaError_t band_occupancy(int* blocks_per_sm);
inline int band_groups(int blocks) { return blocks * (128 / kBandLanes); }
// The DP of the pairs p.order[0 .. p.count) in `blocks` blocks (p.queue 0 before the
// launch; `edges`: `rows` / 2 entries per group, rows even and above every k), then
// their walks.
cudaError_t launch_trace_band(const TraceParams& p, uint2* edges, int rows, int blocks, cudaStream_t stream);
cudaError_t trace16_occupancy(bool protein, int* blocks_per_sm);
// The DP of `ntasks` strip tasks (s.tasks, a pair's strips one after another), then
// the walks of the pairs p.order[0 .. p.count), their runs at the ends of their slots.
cudaError_t launch_trace16(const TraceParams& p, const StripParams& s, int ntasks, int blocks, cudaStream_t stream);
// Copies pair k's nops[k] operations from the end of its slot to out + out_off[k].
cudaError_t launch_gather_ops(const uint32_t* ops, const int64_t* slot_off, const int32_t* nops,
                              const int64_t* out_off, uint32_t* out, int64_t n, cudaStream_t stream);

}  // namespace gbsw
