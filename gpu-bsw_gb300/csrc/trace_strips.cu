// Traceback in int16x2, strip by strip: the path definition and the tie rules of
// traceback.cu, computed like the strip-parallel passes (sw_strips.cu: 64 virtual
// lanes in a warp, 4 columns each, two rows a step, a strip's right edge handed on
// row by row in tagged words), then walked by a few lanes per pair.
//
// Rows are 0..k: row 0 is computed by the recurrence itself.  Lane 0 takes in
// H(0,0) = 0, E(0,0) = -inf at row 0, and H(i,0), E(i,0) below it; with F(0,j) = -inf
// the E chain gives H(0,j) = open + (j-1) ext (open <= ext).  Before row 0 every value
// is -inf, a value below every real one (trace16_pair_ok) and far enough from the
// type's end that the rows of the fill cannot wrap.  A difference of
// two candidates fits 16 bits wherever its sign is used: neighbouring H differ by
// no more than a few gaps and scores.
//
// Directions.  A cell's four bits are the signs of four packed differences: E opened
// (E + ext < H + open), F opened, F < H, and diagonal < H, so the source of H is the
// diagonal, else F, else E, the first that equals it.  prmt spreads the
// signs of two of them over the four bytes of a word, one LOP3 keeps the cell's
// bit of each byte: a lane's 2 rows x 4 columns x 2 halves make two words, stored
// [strip][step / 4][lane][step % 4], so that a lane fills whole sectors, a warp's
// stores are contiguous although its lanes work on different rows, and a walk
// finds some four cells in a sector.  Row i, column j of a strip are in step
// i / 2 + virtual lane.
//
// Substitution scores.  DNA compares raw bytes in both halves: symbols are kept
// in bits 7-15 of their half, so that the complement of their xor is -1 where they
// are equal and at most -129 where not, and one add-max makes it max(match,
// mismatch) or, 128 or more below match, mismatch; protein reads a strip profile,
// as the passes.  Row 0 and those before it are below every real value whatever
// they add, and no real cell depends on rows and columns outside the pair.
//
// Calls of many DNA pairs run trace_band below, the same cells within a band.
//
// What bounds it: the DP, the ALU pipe (9 ALU and 8 other operations a cell pair,
// where the int32 kernel spent 17 ALU operations on one cell); the walk, a
// chain of one direction word per cell.
#include "strip_device.cuh"
#include "sw_device.cuh"
#include "traceback.h"

namespace gbsw {
namespace {

constexpr int kTraceSteps = 8;               // steps of a chunk
constexpr int kTraceRows = 2 * kTraceSteps;  // their rows, fetched together
constexpr int kTraceFront = 128;             // entries of an edge buffer before row 0 (the pipeline's fill)
constexpr uint32_t kOpI = 1, kOpD = 2, kOpEq = 7, kOpX = 8;
// DNA: a symbol's place in its half, and the row symbol outside the pair (at most 0
// against a padding column, whose symbol is 0, so that no value grows out there)
constexpr int kSymShift = 7;
constexpr unsigned kRowPad = 0x7f;

__device__ __forceinline__ int gap_cost(int open, int ext, int len) { return open + (len - 1) * ext; }

// Two rows of a lane's columns, both halves: the row above in hup (H), hop (H + open) and
// fup (F), H(i-1, left) in diag0, H and E of the left edge's two rows in h_in and e (E:
// on to the right neighbour); leaves the rows' H in first and hup and their direction bits.
template <class Score>
__device__ __forceinline__ void two_rows(unsigned (&hup)[kTrace16Cols], unsigned (&hop)[kTrace16Cols],
                                         unsigned (&fup)[kTrace16Cols], unsigned diag0, const unsigned (&h_in)[2],
                                         unsigned (&e)[2], unsigned open2, unsigned ext2, Score score,
                                         unsigned (&first)[kTrace16Cols], unsigned& bits_ef, unsigned& bits_h) {
    unsigned diag[2] = {diag0, h_in[0]}, left[2] = {__vadd2(h_in[0], open2), __vadd2(h_in[1], open2)};
#pragma unroll
    for (int c = 0; c < kTrace16Cols; ++c) {
        unsigned up = hup[c], upo = hop[c], f = fup[c];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const unsigned d = __vadd2(diag[r], score(r, c));
            const unsigned ee = __vadd2(e[r], ext2), fe = __vadd2(f, ext2);
            e[r] = __vmaxs2(ee, left[r]);  // E(i, j)
            f = __vmaxs2(fe, upo);         // F(i, j)
            const unsigned h = __vimax3_s16x2(d, f, e[r]);
            // signs: E opened, F opened; F < H, diagonal < H
            const unsigned ef = prmt(__vsub2(ee, left[r]), __vsub2(fe, upo), 0xFDB9u);
            const unsigned hh = prmt(__vsub2(f, h), __vsub2(d, h), 0xFDB9u);
            const unsigned bit = 0x01010101u << (4 * r + c);
            bits_ef |= ef & bit;
            bits_h |= hh & bit;
            diag[r] = up;
            up = h;
            upo = left[r] = __vadd2(h, open2);
            if (r == 0) first[c] = h;
        }
        hup[c] = up;
        hop[c] = upo;
        fup[c] = f;
    }
}

template <bool PROTEIN>
__global__ void __launch_bounds__(kThreads, 4) trace_strips(TraceParams p, StripParams s, int ntasks) {
    constexpr int C = kTrace16Cols, W = kTrace16Width;
    static_assert(C == 4, "two words of direction bits a step");
    // what lane 0 takes in at each step: the edge words of its two rows, their codes
    __shared__ __align__(16) uint4 sin_[kThreads / 32][2][kTraceSteps];
    __shared__ int smat[PROTEIN ? kAADim * kAADim : 1];
    __shared__ int senc[PROTEIN ? 128 : 1];
    constexpr unsigned kResidue = kThreads * C;  // bytes from one residue's slice of the profile to the next
    __shared__ __align__(16) unsigned char sprof[PROTEIN ? 2 * kAAProfRows * kResidue : 1];
    __shared__ int s_first;
    if constexpr (PROTEIN) {
        for (int k = threadIdx.x; k < kAADim * kAADim; k += blockDim.x) smat[k] = p.aa_matrix[k];
        for (int k = threadIdx.x; k < 128; k += blockDim.x) senc[k] = k < 91 ? p.aa_encoding[k] : 0;
    }
    if (threadIdx.x == 0) s_first = strip_first_task(s, p.queue, ntasks);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int src = (lane + 31) & 31;
    // lane 0: the injected word's low (or high) half, then lane 31's low half
    const unsigned sel_lo = lane ? 0x3210u : 0x1054u, sel_hi = lane ? 0x3210u : 0x1076u;
    const int open = p.open, ext = p.ext;
    const unsigned open2 = pack16(open, open), ext2 = pack16(ext, ext), neg2 = pack16(p.neg, p.neg);
    const unsigned match_up = pack16(p.match + 1, p.match + 1), mismatch2 = pack16(p.mismatch, p.mismatch);
    int task = s_first + warp;
    auto advance = [&] {
        if (lane == 0) task = atomicAdd(p.queue, 1);
        task = __shfl_sync(kFull, task, 0);
    };
    for (;; advance()) {
        if (task >= ntasks) break;
        const int2 work = s.tasks[task];
        const int pid = work.x, strip = work.y & 0xffff, nstrips = (int)((unsigned)work.y >> 16);
        const bool last = strip + 1 == nstrips;
        const unsigned tag = s.tag_base + (unsigned)task;
        const int rb = p.ref_begin[pid], qb = p.query_begin[pid];
        const int m = p.ref_end[pid] - rb, k = p.query_end[pid] - qb;
        const uint8_t* const R = p.ref + p.ref_off[pid] + rb;
        const uint8_t* const Q = p.query + p.query_off[pid] + qb;
        const bool ref_longer = p.ref_off[pid + 1] - p.ref_off[pid] >= p.query_off[pid + 1] - p.query_off[pid];
        const int j_a = strip * W + lane * C + 1, j_b = j_a + 32 * C;  // first columns (1-based) of the halves
        const int lanes = min(64, (m - strip * W + C - 1) / C);
        const int pairs = (k + 2) / 2;                                 // row pairs of rows 0..k
        const int t_end = pairs + lanes - 1;
        uint2* const dir = reinterpret_cast<uint2*>(p.dir + p.dir_off[pid - p.first]) + (int64_t)strip * trace16_strip_words(pairs, 64) / 2;
        // steps in which this lane holds a row of the pair in one of its halves
        const int keep_end = lane < lanes ? min(t_end, lane + pairs + (lanes > 32 ? 32 : 0)) : 0;
        // where H(k, m) is
        const int vm = ((m - 1) % W) / C, t_fin = last ? (k >> 1) + vm : -1;
        if (!last && !strip_buffer_free(p.error, s, task)) break;
        uint64_t* const e_out = s.edges + (size_t)(task % s.ring) * s.edge_stride;
        const uint64_t* const e_in = s.edges + (size_t)((task + s.ring - 1) % s.ring) * s.edge_stride;
        uint64_t* e_step = e_out + (kTraceFront - 2 * 63);

        unsigned rc[PROTEIN ? 1 : C];  // DNA: this lane's column symbols, both halves
        if constexpr (PROTEIN) {
            unsigned char* const prof = sprof + (size_t)threadIdx.x * C;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                int cc[C];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int j = (x ? j_b : j_a) + c;
                    cc[c] = j <= m ? senc[R[j - 1] & 127] : -1;
                }
                for (int e = 0; e < kAAProfRows; ++e) {
                    unsigned w = 0;
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const int v = (cc[c] < 0 || e == kAAPad)
                                          ? kNegByte
                                          : (ref_longer ? smat[cc[c] * kAADim + e] : smat[e * kAADim + cc[c]]);
                        w |= ((unsigned)v & 0xffu) << (8 * c);
                    }
                    *reinterpret_cast<unsigned*>(prof + (size_t)(x * kAAProfRows + e) * kResidue) = w;
                }
            }
        } else {
#pragma unroll
            for (int c = 0; c < C; ++c)
                rc[c] = ((j_a + c <= m ? (unsigned)R[j_a + c - 1] : 0u) |
                         ((j_b + c <= m ? (unsigned)R[j_b + c - 1] : 0u) << 16)) << kSymShift;
        }

        // code of row i: DNA its symbol, protein its residue's offset in the profile
        auto row_code = [&](int i) -> unsigned {
            const bool real = i >= 1 && i <= k;
            const int v = real ? (int)Q[i - 1] : 0;
            if constexpr (PROTEIN) return (real ? (unsigned)senc[v & 127] : (unsigned)kAAPad) * kResidue;
            return real ? (unsigned)v << kSymShift : kRowPad;
        };
        unsigned ncode = 0;
        uint64_t nedge = 0;
        bool nneeds = false;
        const uint64_t* nat = nullptr;
        auto issue = [&](int t0) {  // lanes 0 .. kTraceRows - 1: rows 2 t0 + lane
            const int i = 2 * t0 + lane;
            const bool mine = lane < kTraceRows;
            ncode = row_code(mine ? i : 0);
            nneeds = mine && strip > 0 && i <= k;
            nat = e_in + (kTraceFront + i);
            if (nneeds) {
                nedge = load_word(nat);
            } else {
                const int h = i <= k ? (i > 0 ? gap_cost(open, ext, i) : 0) : p.neg;
                nedge = pack16(h, p.neg);
            }
        };
        auto commit = [&](int buf) -> bool {
            if (strip > 0 && !strip_wait(p.error, nneeds, nat, tag - 1, nedge)) return false;
            if (lane < kTraceRows) {
                unsigned* at = reinterpret_cast<unsigned*>(&sin_[warp][buf][lane >> 1]);
                at[lane & 1] = (unsigned)nedge;
                reinterpret_cast<unsigned short*>(at + 2)[lane & 1] = (unsigned short)ncode;
            }
            __syncwarp();
            return true;
        };

        unsigned hup[C], hop[C], fup[C];  // the row above: H, H + open, F
#pragma unroll
        for (int c = 0; c < C; ++c) {
            hup[c] = fup[c] = neg2;
            hop[c] = pack16(p.neg + open, p.neg + open);
        }
        unsigned diag0 = neg2, x_h[2] = {neg2, neg2}, x_e[2] = {neg2, neg2}, x_code[2];
        x_code[0] = x_code[1] = row_code(0) * 0x10001u;  // rows before 0
        const unsigned char* const prof = sprof + (size_t)threadIdx.x * C;
        __syncwarp();
        int t = 0, buf = 0;
        issue(0);
        bool ok = commit(0);
        while (ok) {
            issue(t + kTraceSteps);
            uint4 next = sin_[warp][buf][0];  // loaded a step ahead
            uint2 kept[4];
#pragma unroll 4
            for (int u = 0; u < kTraceSteps; ++u) {
                const uint4 in = next;
                next = sin_[warp][buf][(u + 1) % kTraceSteps];
                const unsigned code[2] = {prmt(x_code[0], in.z, sel_lo), prmt(x_code[1], in.z, sel_hi)};
                x_code[0] = __shfl_sync(kFull, code[0], src);
                x_code[1] = __shfl_sync(kFull, code[1], src);
                const unsigned h_in[2] = {prmt(x_h[0], in.x, sel_lo), prmt(x_h[1], in.y, sel_lo)};
                unsigned e[2] = {prmt(x_e[0], in.x, sel_hi), prmt(x_e[1], in.y, sel_hi)};
                unsigned wa[2] = {0, 0}, wb[2] = {0, 0};
                if constexpr (PROTEIN) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        wa[r] = *reinterpret_cast<const unsigned*>(prof + (code[r] & 0xffffu));
                        wb[r] = *reinterpret_cast<const unsigned*>(prof + kAAProfRows * kResidue + (code[r] >> 16));
                    }
                }
                unsigned first[C], bits_ef = 0, bits_h = 0;
                two_rows(
                    hup, hop, fup, diag0, h_in, e, open2, ext2,
                    [&](int r, int c) -> unsigned {
                        if constexpr (PROTEIN) return prmt(wa[r], wb[r], (unsigned)c * 0x1111u + 0xC480u);
                        else return __viaddmax_s16x2(~(code[r] ^ rc[c]), match_up, mismatch2);
                    },
                    first, bits_ef, bits_h);
#pragma unroll
                for (int r = 0; r < 2; ++r) x_e[r] = __shfl_sync(kFull, e[r], src);
                x_h[0] = __shfl_sync(kFull, first[C - 1], src);
                x_h[1] = __shfl_sync(kFull, hup[C - 1], src);
                diag0 = h_in[1];
                kept[u % 4] = make_uint2(bits_ef, bits_h);
                if (u % 4 == 3 && t >= lane && t - 3 < keep_end) {
                    uint4* const at = reinterpret_cast<uint4*>(dir + (int64_t)(t >> 2) * 128 + 4 * lane);
                    at[0] = make_uint4(kept[0].x, kept[0].y, kept[1].x, kept[1].y);
                    at[1] = make_uint4(kept[2].x, kept[2].y, kept[3].x, kept[3].y);
                }
                // rows 2 (t - 63) and the next; rows outside the pair fall into the buffer's margins
                if (!last && lane == 31)
                    store_words(e_step, tag, prmt(first[C - 1], e[0], 0x7632u), prmt(hup[C - 1], e[1], 0x7632u));
                e_step += 2;
                if (t == t_fin) {
                    unsigned h = 0;
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        if (c == (m - 1) % C) h = (k & 1) ? hup[c] : first[c];
                    if (lane == (vm & 31)) p.path_score[pid] = vm >= 32 ? hi16(h) : lo16(h);
                }
                ++t;
            }
            // values that could soon wrap: results of other inputs (trace16_pair_ok)
            unsigned high = hup[0];
#pragma unroll
            for (int c = 1; c < C; ++c) high = __vmaxs2(high, hup[c]);
            if (max(lo16(high), hi16(high)) > p.top) atomicOr(p.error, kErrTrace);
            if (t >= t_end) break;
            ok = commit(buf ^ 1);
            buf ^= 1;
        }
        if (!ok) break;  // a wait ran out: kErrTeam is set, every warp stops
        __syncwarp();
        if (strip > 0 && lane == 0) strip_buffer_read(s, task - 1);
    }
}

// The DP of DNA pairs whose score leaves their paths a narrow band (trace_band_of), many
// pairs at a time: groups of 4 lanes take pairs from the queue and run a pair's strips
// (8 virtual lanes, 32 columns) one after another, over the band's rows only.  A cell
// outside the band counts as -inf.  That leaves every cell of every path of the pair's
// score as it was, a candidate that ties with one among them, and no cell above its
// value, so the walk meets the same choices; a score that is not the segment's gives a
// path value that differs from it, as without a band.  The strip's edge goes through a
// buffer of the group's own, a word a row, in place: rows are read a chunk before they
// are written.
//
// A read of 225 symbols at the throughput shape's error rate keeps 2 x 21 diagonals
// of its 225 rows.  In 256-column strips of a whole warp it took 169 steps of a warp,
// two thirds of their cells outside the segment or the band; here 7 strips of 46 steps
// of an eighth of one.  100,000 such pairs, DP and walks: 4.71 -> 1.67 ms, with 1.8 in
// place of 4.3 GB of directions.  Bound by the ALU pipe, as the strips.
__global__ void __launch_bounds__(kThreads, 4) trace_band(TraceParams p, uint2* edges, int rows) {
    constexpr int C = kTrace16Cols, G = kBandLanes, W = kBandWidth, kGroups = kThreads / G;
    constexpr int kFetch = kTraceSteps / G;  // row pairs a lane fetches for a chunk
    static_assert(kTraceSteps % G == 0 && kThreads == 128, "the fetch and band_groups");
    // what lane 0 takes in at each step: the edge words of its two rows, their codes
    __shared__ __align__(16) uint4 sin_[kGroups][2][kTraceSteps];
    const int lane = threadIdx.x & 31, g = lane % G, grp = threadIdx.x / G;
    const unsigned gmask = ((1u << G) - 1u) << (lane - g);
    const int src = lane - g + (g + G - 1) % G;
    // lane 0: the injected word's low (or high) half, then lane G - 1's low half
    const unsigned sel_lo = g ? 0x3210u : 0x1054u, sel_hi = g ? 0x3210u : 0x1076u;
    const int open = p.open, ext = p.ext;
    const unsigned open2 = pack16(open, open), ext2 = pack16(ext, ext), neg2 = pack16(kBandNeg, kBandNeg);
    const unsigned match_up = pack16(p.match + 1, p.match + 1), mismatch2 = pack16(p.mismatch, p.mismatch);
    uint2* const edge = edges + ((size_t)blockIdx.x * kGroups + grp) * (size_t)(rows / 2);

    // ---- group state ----
    bool busy = false, done = false;
    int pid = 0, m = 0, k = 0, strip = 0, t = 0, t_end = 0, buf = 0;
    int p0 = 0, p1 = -1, have = -1;  // the strip's first and last row pair, the last one its left edge holds
    int keep_end = 0, t_fin = -1, vm = 0, hand_on = 0;  // hand_on: row pairs whose edge the next strip reads
    TraceBand band{0, 0};
    const uint8_t *R = p.ref, *Q = p.query;
    uint2* dir = nullptr;
    // ---- lane state ----
    unsigned hup[C], hop[C], fup[C], rc[C];
    unsigned diag0 = neg2, x_h[2] = {neg2, neg2}, x_e[2] = {neg2, neg2}, x_code[2] = {0, 0};
#pragma unroll
    for (int c = 0; c < C; ++c) {
        hup[c] = hop[c] = fup[c] = neg2;
        rc[c] = 0;
    }

    auto row_code = [&](int i) -> unsigned {
        return i >= 1 && i <= k ? (unsigned)Q[i - 1] << kSymShift : kRowPad;
    };
    uint2 nedge[kFetch];
    unsigned ncode[kFetch];
    auto issue = [&](int t0) {  // lane g: row pairs g, g + G of the chunk
#pragma unroll
        for (int x = 0; x < kFetch; ++x) {
            const int q = p0 + t0 + g + x * G, i = 2 * q;
            ncode[x] = row_code(i) | (row_code(i + 1) << 16);
            if (strip > 0) {
                nedge[x] = q <= have ? __ldcg(edge + q) : make_uint2(neg2, neg2);
            } else {
                nedge[x].x = pack16(i <= k ? (i > 0 ? gap_cost(open, ext, i) : 0) : kBandNeg, kBandNeg);
                nedge[x].y = pack16(i < k ? gap_cost(open, ext, i + 1) : kBandNeg, kBandNeg);
            }
        }
    };
    auto commit = [&](int b) {
#pragma unroll
        for (int x = 0; x < kFetch; ++x)
            sin_[grp][b][g + x * G] = make_uint4(nedge[x].x, nedge[x].y, ncode[x], 0);
    };
    auto setup_strip = [&] {
        const int lanes = min(2 * G, (m - strip * W + C - 1) / C);
        const bool last = (strip + 1) * W >= m;
        have = p1;
        p0 = band_first_pair(band, strip);
        p1 = band_last_pair(band, strip, k);
        const int pairs = p1 - p0 + 1;
        t = 0;
        t_end = pairs + lanes - 1;
        keep_end = g < lanes ? min(t_end, g + pairs + (lanes > G ? G : 0)) : 0;
        vm = ((m - 1) % W) / C;
        t_fin = last ? (k >> 1) - p0 + vm : -1;
        hand_on = last ? 0 : pairs;
        const int j_a = strip * W + g * C + 1, j_b = j_a + G * C;  // first columns (1-based) of the halves
#pragma unroll
        for (int c = 0; c < C; ++c) {
            rc[c] = ((j_a + c <= m ? (unsigned)R[j_a + c - 1] : 0u) |
                     ((j_b + c <= m ? (unsigned)R[j_b + c - 1] : 0u) << 16)) << kSymShift;
            hup[c] = fup[c] = neg2;
            hop[c] = pack16(kBandNeg + open, kBandNeg + open);
        }
        diag0 = x_h[0] = x_h[1] = x_e[0] = x_e[1] = neg2;
        x_code[0] = x_code[1] = kRowPad * 0x10001u;  // rows before the strip's
        buf = 0;
        issue(0);
        commit(0);
    };

    while (true) {
        if (!done && !busy) {
            int at = 0;
            if (g == 0) at = atomicAdd(p.queue, 1);
            at = __shfl_sync(gmask, at, lane - g);
            if (at >= p.count) {
                done = true;
                keep_end = hand_on = 0;
                t_fin = -1;
            } else {
                pid = (int)p.order[at];
                const int score = p.score[pid];
                if (score > 0) {
                    const int rb = p.ref_begin[pid], qb = p.query_begin[pid];
                    m = p.ref_end[pid] - rb;
                    k = p.query_end[pid] - qb;
                    R = p.ref + p.ref_off[pid] + rb;
                    Q = p.query + p.query_off[pid] + qb;
                    band = trace_band_of(m, k, score, p.match, open, ext);
                    dir = reinterpret_cast<uint2*>(p.dir + p.dir_off[pid - p.first]);
                    strip = 0;
                    p1 = -1;
                    busy = true;
                    setup_strip();
                }
            }
            __syncwarp(gmask);
        }
        if (__all_sync(kFull, done)) break;
        if (__any_sync(kFull, !done && !busy)) continue;  // a pair without a path: take the next one

        // ---- kTraceSteps steps, every lane of the warp ----
        if (busy) issue(t + kTraceSteps);
        uint4 next = sin_[grp][buf][0];  // loaded a step ahead
        uint2 kept[4];
#pragma unroll 4
        for (int u = 0; u < kTraceSteps; ++u) {
            const uint4 in = next;
            next = sin_[grp][buf][(u + 1) % kTraceSteps];
            const unsigned code[2] = {prmt(x_code[0], in.z, sel_lo), prmt(x_code[1], in.z, sel_hi)};
            x_code[0] = __shfl_sync(kFull, code[0], src);
            x_code[1] = __shfl_sync(kFull, code[1], src);
            const unsigned h_in[2] = {prmt(x_h[0], in.x, sel_lo), prmt(x_h[1], in.y, sel_lo)};
            unsigned e[2] = {prmt(x_e[0], in.x, sel_hi), prmt(x_e[1], in.y, sel_hi)};
            unsigned first[C], bits_ef = 0, bits_h = 0;
            two_rows(
                hup, hop, fup, diag0, h_in, e, open2, ext2,
                [&](int r, int c) { return __viaddmax_s16x2(~(code[r] ^ rc[c]), match_up, mismatch2); }, first,
                bits_ef, bits_h);
#pragma unroll
            for (int r = 0; r < 2; ++r) x_e[r] = __shfl_sync(kFull, e[r], src);
            x_h[0] = __shfl_sync(kFull, first[C - 1], src);
            x_h[1] = __shfl_sync(kFull, hup[C - 1], src);
            diag0 = h_in[1];
            kept[u % 4] = make_uint2(bits_ef, bits_h);
            if (u % 4 == 3 && t >= g && t - 3 < keep_end) {
                uint4* const at = reinterpret_cast<uint4*>(dir + (t >> 2) * (4 * G) + 4 * g);
                at[0] = make_uint4(kept[0].x, kept[0].y, kept[1].x, kept[1].y);
                at[1] = make_uint4(kept[2].x, kept[2].y, kept[3].x, kept[3].y);
            }
            const int q = t - (2 * G - 1);  // the last virtual lane's row pair
            if (g == G - 1 && (unsigned)q < (unsigned)hand_on)
                __stcg(edge + p0 + q, make_uint2(prmt(first[C - 1], e[0], 0x7632u), prmt(hup[C - 1], e[1], 0x7632u)));
            if (t == t_fin) {
                unsigned h = 0;
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (c == (m - 1) % C) h = (k & 1) ? hup[c] : first[c];
                if (g == vm % G) p.path_score[pid] = vm >= G ? hi16(h) : lo16(h);
            }
            ++t;
        }
        if (busy && t < t_end) {
            buf ^= 1;
            commit(buf);
        } else if (busy) {
            __syncwarp(gmask);  // this strip's edge before the next one reads it
            if ((strip + 1) * W < m) {
                dir += band_strip_words(band, k) / 2;
                ++strip;
                setup_strip();
            } else {
                busy = false;
                keep_end = hand_on = 0;
                t_fin = -1;
            }
        }
        __syncwarp();
    }
}

// The paths of the launch's pairs, in the order of their cost (a warp's walks end
// close together), a group of kWalkLanes lanes each.  The lanes walk in step, so
// that each of them can fetch a part of what comes next: a tile holds, for the
// virtual lane of the current cell and the seven left of it, the eight steps
// around the diagonal's rows there, and the 32 symbols up and left of the cell.
// A walk that leaves its tile (a long gap, the strip's edge, its end) takes the
// next one.  (One thread per pair took 0.92 ms for the walks of 7,001 proteins, most
// of it in one of 32 lanes' misses at every step.)  Runs are written from the
// slot's end backwards, which leaves them in path order.
template <bool BAND>
__global__ void __launch_bounds__(kWalkThreads) walk_paths(TraceParams p) {
    constexpr int L = kWalkLanes, S = 4 * L;  // symbols of a tile
    constexpr int G = BAND ? kBandLanes : 32, W = BAND ? kBandWidth : kTrace16Width;
    __shared__ __align__(16) uint4 s_dir[kWalkThreads / L][L][4];
    __shared__ uint8_t s_r[kWalkThreads / L][S], s_q[kWalkThreads / L][S];
    const int lane = threadIdx.x & 31, g = lane % L, grp = threadIdx.x / L;
    const unsigned gmask = ((1u << L) - 1u) << (lane - g);
    const int64_t at = (int64_t)blockIdx.x * (kWalkThreads / L) + grp;
    if (at >= p.count) return;
    const int64_t pid = p.order[at];
    const int score = p.score[pid];
    if (score <= 0) {
        if (g == 0) p.nops[pid] = p.path_score[pid] = 0;
        return;
    }
    if (p.path_score[pid] != score) {
        if (g == 0) {
            atomicOr(p.error, kErrTrace);
            p.nops[pid] = 0;
        }
        return;
    }
    const int rb = p.ref_begin[pid], qb = p.query_begin[pid];
    const int m = p.ref_end[pid] - rb, k = p.query_end[pid] - qb;
    const uint8_t* const R = p.ref + p.ref_off[pid] + rb;
    const uint8_t* const Q = p.query + p.query_off[pid] + qb;
    const uint4* const dir = reinterpret_cast<const uint4*>(p.dir + p.dir_off[pid - p.first]);
    TraceBand band{0, 0};
    if constexpr (BAND) band = trace_band_of(m, k, score, p.match, p.open, p.ext);
    const int64_t per_strip = (BAND ? band_strip_words(band, k) : trace16_strip_words((k + 2) / 2, 64)) / 4;
    uint32_t* out = p.ops + p.slot_off[pid + 1];
    int i = k, j = m, state = 0, n = 0;
    int ti = 0, tj = 0, tv = 0, tt = 0, ts = -1;  // the tile's first cell, its virtual lane, first step and strip (-1: no tile)
    uint32_t run = 0;  // the run being extended (len << 4 | op)
    auto push = [&](uint32_t op) {
        if ((run & 15u) == op) {
            run += 16u;
        } else {
            if (run) {
                --out;
                ++n;
                if (g == 0) *out = run;
            }
            run = 16u | op;
        }
    };
    while (i > 0 && j > 0) {
        const int strip = (j - 1) / W, c = (j - 1) % W, v = c / kTrace16Cols;
        const int p0 = BAND ? band_first_pair(band, strip) : 0, t = (i >> 1) - p0 + v;
        int l = tv - v;
        // of the two sectors the tile holds for virtual lane tv - l, step / 4 of the second
        int sector = (t >> 2) - ((tt - 3 * l) >> 2) + 1;
        if (strip != ts || (unsigned)l >= (unsigned)L || (unsigned)sector > 1u || (unsigned)((ti - i) | (tj - j)) >= (unsigned)S) {
            ti = i;
            tj = j;
            tv = v;
            ts = strip;
            l = 0;
            // the diagonal enters the columns of virtual lane v - l in row first - 4 l, so
            // in step tt - 1 - 3 l
            tt = ((i + 3 - c % kTrace16Cols) >> 1) - p0 + v + 1;
            sector = (t >> 2) - (tt >> 2) + 1;
            __syncwarp(gmask);  // every lane is done with the old tile
            const int lanes = min(2 * G, (m - strip * W + kTrace16Cols - 1) / kTrace16Cols);
            const int pairs = (BAND ? band_last_pair(band, strip, k) : k >> 1) - p0 + 1;
            const int last_q = (pairs + lanes - 2) >> 2, q = (tt - 3 * g) >> 2;  // the strip's last step / 4
            if (v - g >= 0) {
                const uint4* const src = dir + (int64_t)strip * per_strip + (int64_t)q * (2 * G) + 2 * ((v - g) % G);
                if (q >= 1 && q - 1 <= last_q) {
                    s_dir[grp][g][0] = src[-2 * G];
                    s_dir[grp][g][1] = src[-2 * G + 1];
                }
                if (q >= 0 && q <= last_q) {
                    s_dir[grp][g][2] = src[0];
                    s_dir[grp][g][3] = src[1];
                }
            }
#pragma unroll
            for (int x = g; x < S; x += L) {
                if (j - 1 - x >= 0) s_r[grp][x] = R[j - 1 - x];
                if (i - 1 - x >= 0) s_q[grp][x] = Q[i - 1 - x];
            }
            __syncwarp(gmask);
        }
        const bool same = s_r[grp][tj - j] == s_q[grp][ti - i];
        const uint2 w = reinterpret_cast<const uint2*>(s_dir[grp][l])[4 * sector + (t & 3)];
        const int sh = (v >= G ? 8 : 0) + 4 * (i & 1) + c % kTrace16Cols;
        if (state == 0) {
            if (!((w.y >> (16 + sh)) & 1u)) {
                push(same ? kOpEq : kOpX);
                --i;
                --j;
            } else {
                state = ((w.y >> sh) & 1u) ? 1 : 2;
            }
        }
        if (state == 1) {
            push(kOpD);
            if ((w.x >> sh) & 1u) state = 0;
            --j;
        } else if (state == 2) {
            push(kOpI);
            if ((w.x >> (16 + sh)) & 1u) state = 0;
            --i;
        }
    }
    for (; j > 0; --j) push(kOpD);
    for (; i > 0; --i) push(kOpI);
    if (run) {
        ++n;
        if (g == 0) *--out = run;
    }
    if (g == 0) p.nops[pid] = n;
}

}  // namespace

namespace {
unsigned walk_blocks(int64_t pairs) {
    constexpr int kPerBlock = kWalkThreads / kWalkLanes;
    return (unsigned)((pairs + kPerBlock - 1) / kPerBlock);
}
}  // namespace

cudaError_t trace16_occupancy(bool protein, int* blocks_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        blocks_per_sm, protein ? (const void*)trace_strips<true> : (const void*)trace_strips<false>, kThreads, 0);
}

cudaError_t launch_trace16(const TraceParams& p, const StripParams& s, int ntasks, int blocks, cudaStream_t stream) {
    if (p.count <= 0) return cudaSuccess;
    if (ntasks > 0) {
        if (p.protein)
            trace_strips<true><<<blocks, kThreads, 0, stream>>>(p, s, ntasks);
        else
            trace_strips<false><<<blocks, kThreads, 0, stream>>>(p, s, ntasks);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    walk_paths<false><<<walk_blocks(p.count), kWalkThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t band_occupancy(int* blocks_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, (const void*)trace_band, kThreads, 0);
}

cudaError_t launch_trace_band(const TraceParams& p, uint2* edges, int rows, int blocks, cudaStream_t stream) {
    if (p.count <= 0) return cudaSuccess;
    trace_band<<<blocks, kThreads, 0, stream>>>(p, edges, rows);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    walk_paths<true><<<walk_blocks(p.count), kWalkThreads, 0, stream>>>(p);
    return cudaGetLastError();
}

}  // namespace gbsw
