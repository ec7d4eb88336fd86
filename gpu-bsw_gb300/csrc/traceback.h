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
cudaError_t trace16_occupancy(bool protein, int* blocks_per_sm);
// The DP of `ntasks` strip tasks (s.tasks, a pair's strips one after another), then
// the walks of the pairs p.order[0 .. p.count), their runs at the ends of their slots.
cudaError_t launch_trace16(const TraceParams& p, const StripParams& s, int ntasks, int blocks, cudaStream_t stream);
// Copies pair k's nops[k] operations from the end of its slot to out + out_off[k].
cudaError_t launch_gather_ops(const uint32_t* ops, const int64_t* slot_off, const int32_t* nops,
                              const int64_t* out_off, uint32_t* out, int64_t n, cudaStream_t stream);

}  // namespace gbsw
