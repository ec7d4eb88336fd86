// Lower bounds of DNA pairs' scores, before the forward pass: the score of one real
// alignment of each pair, found by seed and extension.  The forward pass then computes
// only the rows of a strip that an alignment of that score can cross (sw_dual.cu).  The
// bound changes no result: a low one (0 where nothing is found) only leaves more rows.
//
// A warp packs a pair's sequences to 2 bits a symbol in shared memory and looks for 8
// anchors of 12 symbols, evenly spaced over the shorter sequence, at every position of
// the longer one.  The place of the anchor nearest to the middle is extended to both sides, a lane
// each, 16 pairs at a time: along the diagonal while symbols agree, 16 at a step; where
// two differ, on past them or past a gap of 1 to 8 on either side, whichever agrees
// best over the 10 symbols behind it.  (On the throughput shape it finds the score itself
// of half the related pairs.)
//
// Bound by issue: a warp takes some 1,000 instructions to pack and scan a read and its
// 700-symbol reference, and 300 for the next difference of 16 pairs.  100,000 of them: 0.30 ms
// (a pair at a time, with 16 places extended each: 1.20).  Gaps of 1 to 3 only lost the
// alignment of one long pair in ten: forward pass of 200,000 mixed pairs 42.9 ms, with 1 to 5
// 36, 1 to 8 32.9, 1 to 10 32.9.
#include <algorithm>

#include "strip_device.cuh"
#include "sw_device.cuh"
#include "sw_kernels.h"

namespace gbsw {
namespace {

constexpr int kSeed = 12, kAnchors = 8, kGap = 8;  // symbols of a seed, seeds of a pair, longest gap of a step
constexpr unsigned kBehindMask = (1u << 20) - 1;  // 10 symbols behind a difference
constexpr unsigned kSeedMask = (1u << (2 * kSeed)) - 1;
constexpr int kBoundRows = 8192, kBoundCols = 4096;  // longer pairs go without a bound
// Smaller ones too: their few strips have little to leave out (140,000 reads of 100-150
// against 300 symbols: forward 1.76 ms, with bounds 1.97).
constexpr int kBoundCells = 1 << 16;
// Of a warp: packed words, and in batches of longer pairs (200,000 mixed pairs, forward: 32.7
// ms with 1,024 words, 31.3 with 4,096, 32.6 with 6,144), pairs to extend together.
constexpr int kBoundWords = 1024, kBoundLongWords = 4096, kBoundPairs = 16;
// A sequence's words and one past the last symbol's.
__host__ __device__ constexpr int bound_words(int len) { return len / 16 + 2; }
static_assert(bound_words(kBoundRows) + bound_words(kBoundCols) <= kBoundWords, "a pair fits");

// Packs the sequence at `s`, part of the buffer [from, to); symbols past its end are
// whatever follows there.
__device__ __forceinline__ void pack_symbols(const uint8_t* s, int len, const uint8_t* from, const uint8_t* to,
                                             unsigned* words, int lane) {
    for (int w = lane; w < bound_words(len); w += 32) {
        const uint8_t* const at = s + 16 * w;
        const uint8_t* const aligned = at - (reinterpret_cast<uintptr_t>(at) & 3u);
        unsigned v = 0;
        if (aligned >= from && aligned + 20 <= to) {
            const unsigned* const x = reinterpret_cast<const unsigned*>(aligned);
            const unsigned sh = 8 * (unsigned)(at - aligned);
            unsigned next = x[0];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned here = next;
                next = x[k + 1];
                unsigned c = (__funnelshift_r(here, next, sh) >> 1) & 0x03030303u;
                c |= c >> 6;
                v |= ((c | (c >> 12)) & 0xffu) << (8 * k);
            }
        } else {
            for (int b = 0; b < 16 && 16 * w + b < len; ++b) v |= (unsigned)dna_code(at[b]) << (2 * b);
        }
        words[w] = v;
    }
}
// 16 symbols from position at >= 0, the first in the low bits.  Reads the word after
// theirs; symbols past the end are whatever it holds.
__device__ __forceinline__ unsigned symbols(const unsigned* s, int at) {
    return __funnelshift_r(s[at >> 4], s[(at >> 4) + 1], 2 * (at & 15));
}
// 16 symbols from position `at` onward in direction dir (bits of backward ones reversed).
__device__ __forceinline__ unsigned window(const unsigned* s, int len, int at, int dir) {
    if (at < 0 || at >= len) return 0;
    if (dir > 0) return symbols(s, at);
    const unsigned v = at >= 15 ? symbols(s, at - 15) : s[0] << (2 * (15 - at));
    return __brev(v);
}
// Bit 2 k set where symbol k of the windows differs.
__device__ __forceinline__ unsigned differ(unsigned a, unsigned b) {
    const unsigned x = a ^ b;
    return (x | (x >> 1)) & 0x55555555u;
}

// Best score of the extension from row i, column j in direction dir.
__device__ int extend(const unsigned* rows, int nrows, const unsigned* cols, int ncols, int i, int j, int dir,
                      const PassParams& p) {
    const int step_off = p.match - p.mismatch, drop = 8 * step_off - p.open;
    int cur = 0, best = 0;
    while (true) {
        const int left = min(min(dir > 0 ? nrows - i : i + 1, dir > 0 ? ncols - j : j + 1), 16);
        if (left <= 0) break;
        const unsigned d = differ(window(rows, nrows, i, dir), window(cols, ncols, j, dir));
        const int run = min(d ? (__ffs((int)d) - 1) >> 1 : 16, left);
        cur += run * p.match;
        best = max(best, cur);
        i += dir * run;
        j += dir * run;
        if (run == left) {
            if (left < 16) break;
            continue;
        }
        // the symbols at (i, j) differ
        const unsigned r0 = window(rows, nrows, i, dir), c0 = window(cols, ncols, j, dir);
        auto gain = [&](unsigned a, unsigned b, int cost) {
            return cost - __popc(differ(a, b) & kBehindMask) * step_off;
        };
        int move_r = 1, move_c = 1, cost = p.mismatch;
        int top = gain(window(rows, nrows, i + dir, dir), window(cols, ncols, j + dir, dir), cost);
#pragma unroll
        for (int n = 1; n <= kGap; ++n) {
            const int gap = p.open + (n - 1) * p.ext;
            const int down = gain(window(rows, nrows, i + dir * n, dir), c0, gap);
            const int right = gain(r0, window(cols, ncols, j + dir * n, dir), gap);
            if (down > top) {
                top = down;
                move_r = n;
                move_c = 0;
                cost = gap;
            }
            if (right > top) {
                top = right;
                move_r = 0;
                move_c = n;
                cost = gap;
            }
        }
        cur += cost;
        i += dir * move_r;
        j += dir * move_c;
        if (cur < best - drop) break;
    }
    return best;
}

struct BoundPair {
    int pid, rows, cols;  // its sequences' words
    int nrows, ncols, row, col;
};

__global__ void __launch_bounds__(kThreads) score_bounds(PassParams p, int2* bound, int room) {
    extern __shared__ unsigned s_words[];  // `room` a warp
    __shared__ BoundPair s_pair[kThreads / 32][kBoundPairs];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned* const words = s_words + warp * room;
    BoundPair* const pair = s_pair[warp];
    int used = 0, pairs = 0;
    auto extend_all = [&] {
        __syncwarp();
        int part = 0;
        if ((lane >> 1) < pairs) {
            const BoundPair x = pair[lane >> 1];
            part = (lane & 1) ? extend(words + x.rows, x.nrows, words + x.cols, x.ncols, x.row - 1, x.col - 1, -1, p)
                              : extend(words + x.rows, x.nrows, words + x.cols, x.ncols, x.row + kSeed, x.col + kSeed, 1, p);
        }
        __syncwarp();
        part += __shfl_xor_sync(kFull, part, 1) + kSeed * p.match;
        if ((lane & 1) == 0 && (lane >> 1) < pairs) {
            const BoundPair& x = pair[lane >> 1];
            bound[x.pid] = make_int2(part, x.row - x.col);
        }
        __syncwarp();
        used = pairs = 0;
    };
    const int64_t warps = (int64_t)gridDim.x * (kThreads / 32);
    for (int64_t pid = (int64_t)blockIdx.x * (kThreads / 32) + warp; pid < p.n; pid += warps) {
        const int64_t ra = p.ref_off[pid], qa = p.query_off[pid];
        const int a = (int)(p.ref_off[pid + 1] - ra), b = (int)(p.query_off[pid + 1] - qa);
        const int nrows = max(a, b), ncols = min(a, b);
        if (lane == 0) bound[pid] = make_int2(0, 0);
        if (ncols < 2 * kSeed || (int64_t)nrows * ncols < kBoundCells || nrows >= kBoundRows || ncols >= kBoundCols) continue;
        const int need = bound_words(nrows) + bound_words(ncols);
        if (pairs == kBoundPairs || used + need > room) extend_all();
        unsigned *const rows = words + used, *const cols = rows + bound_words(nrows);
        const uint8_t *const ref_end = p.ref + p.ref_off[p.n], *const query_end = p.query + p.query_off[p.n];
        const bool flip = a < b;
        pack_symbols(p.ref + ra, a, p.ref, ref_end, flip ? cols : rows, lane);
        pack_symbols(p.query + qa, b, p.query, query_end, flip ? rows : cols, lane);
        __syncwarp();
        unsigned seed[kAnchors];
#pragma unroll
        for (int k = 0; k < kAnchors; ++k) seed[k] = symbols(cols, (ncols - kSeed) * k / (kAnchors - 1)) & kSeedMask;
        // the place found whose anchor lies nearest to the middle: that, anchor, row
        unsigned hit = ~0u;
        for (int at = lane; at <= nrows - kSeed; at += 32) {
            const unsigned v = symbols(rows, at) & kSeedMask;
            bool any = false;
#pragma unroll
            for (int k = 0; k < kAnchors; ++k) any |= v == seed[k];
            if (any) {
#pragma unroll
                for (int k = 0; k < kAnchors; ++k)
                    if (v == seed[k]) hit = min(hit, (unsigned)abs(2 * k - kAnchors + 1) << 24 | (unsigned)k << 16 | (unsigned)at);
            }
        }
        hit = __reduce_min_sync(kFull, hit);
        if (hit != ~0u) {
            const int row = (int)(hit & 0xffffu), k = (int)(hit >> 16) & 0xff;
            if (lane == 0)
                pair[pairs] = BoundPair{(int)pid, used, used + bound_words(nrows), nrows, ncols, row,
                                        (ncols - kSeed) * k / (kAnchors - 1)};
            ++pairs;
            used += need;
        }
        __syncwarp();  // before the next pair's symbols
    }
    extend_all();
}

}  // namespace

cudaError_t launch_score_bounds(const PassParams& p, int2* bound, int sms, cudaStream_t stream) {
    const int64_t want = (p.n + kThreads / 32 - 1) / (kThreads / 32);
    const int room = p.scratch_rows > 1024 ? kBoundLongWords : kBoundWords;
    const size_t dyn = (size_t)(kThreads / 32) * (size_t)room * sizeof(unsigned);
    constexpr int kMost = kThreads / 32 * kBoundLongWords * (int)sizeof(unsigned);  // whatever other calls need
    cudaError_t e = cudaFuncSetAttribute((const void*)score_bounds, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
    if (e != cudaSuccess) return e;
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * 16));
    score_bounds<<<blocks, kThreads, dyn, stream>>>(p, bound, room);
    return cudaGetLastError();
}

}  // namespace gbsw
