// Dual-pair passes: two pairs per lane group, in the two 16-bit halves of
// every register (int16x2 DPX instructions), for DNA pairs made only of
// A/C/G/T and for protein pairs.
//
// The pass kernels are bound by the integer ALU pipe; packing two pairs into
// one register halves the ALU instructions per cell.  A group of G lanes
// owns a unit of two pairs (the schedule puts pairs of the same strip count
// and nearly the same row count next to each other); lane g holds C columns
// of both pairs.  The unit is as tall as its taller pair and as many strips
// wide as its wider pair: in the forward pass each pair is left-padded to the
// unit's width with score -128 (exactly the matrix boundary, as in the int32
// kernel), in the reverse pass padded on the right (as the int32 kernel's
// reverse), and the rows past a pair's last row are simply not looked at by
// its half.
//
// Two rows a step.  Rows stream through the group as a pipeline: at step t lane g
// works on rows 2 (t - g) + 1 and the next one, both halves, and takes H + open
// and E of its left neighbour's last column by shuffle; row codes travel the same
// way, four bytes a step, so each is fetched and converted once per group.  Two
// rows of 8 columns hold as many cells as one row of 16 with half the column state
// (H, F and the profiles), and pay shuffles' latency, the argmax test, the loop and
// the strip edge's store once for both.  All lanes of a warp run a chunk of steps
// together (a group without work runs on padding), so that the shuffles' mask is
// constant.
//
// Overflow: with gap values in [-16384, 0], every term the cell update forms
// stays inside int16 while the true H values stay at or below
// dual_limit = 32767 - m, where m is the largest single-cell score (DNA
// max(match, mismatch, 0), protein the matrix's largest entry).  The first cell
// whose true H exceeds dual_limit is still computed exactly (its inputs are
// exact and it exceeds them by at most m), so a pass whose best score is at
// most dual_limit was exact throughout, and a pair whose reported best exceeds
// it may have wrapped: the forward pass then writes no result for it, queues it
// for the int32 pass (PassParams::rerun) and moves it to int32 class 0, whose
// reverse pass it then takes as well.  The reverse pass never overflows: its
// scores are bounded by the forward score.
//
// Substitution scores, both halves with one prmt per cell:
//   DNA: each column keeps the packed int8 scores of its base against A, C, G,
//     T for both pairs; the two row codes pick one byte of each;
//   protein: the group keeps an int8 profile of both pairs' strips (24 residue
//     rows each) in shared memory; per row a lane loads its C scores of pair A's
//     row residue and of pair B's and interleaves byte c of each.
// Each thread builds and reads only its own slice of the profiles, laid out
// [half][residue][thread][C bytes] so that the loads of a warp stay
// conflict-free whatever residues its rows hold.
//
// Per cell (both halves at once; E = E(i,j) from the left, Ho = H + open):
//   s   = the two pairs' scores of this cell
//   F'  = max(F + ext, Ho_up, 0)
//   T   = max(F' + open, Ho_diag + s)
//   Ho  = max(E + open, T)
//   E'  = max(E + max(ext, open), T, 0)          (= max(E + ext, Ho, 0))
// which is the int32 kernel's recurrence (see sw_pass.cuh) evaluated per half.
// The plain packed add of T's second term runs beside the ALU pipe, which takes
// a warp instruction every other cycle (measured: a viaddmax alone 1.01 ns per
// warp and scheduler, with a packed add beside it 1.01, with a second viaddmax,
// vimax3 or prmt 2.02).
//
// Argmax.  Forward: a lane keeps the running max of its cells and the step of the
// chunk in which it last grew; the chunk's rows stay in shared memory, and where a max
// grew the two rows of that step are saved (rows past a pair's last one may seem to grow
// it: the chunk that holds the last row looks at its rows one by one).  A strip's maxima
// start one below the best cell of the strips before it, which no smaller cell can beat:
// the random growth of unrelated strips no longer saves anything.  Reverse: one test a
// step for a half that reaches its score, once per lane.  The rules are the int32
// kernel's, as are the transposed reverse pass and its band (reverse_band,
// reverse_low_band): a unit's strips start and end at the rows its wider band needs, and
// both halves compute every row between.
//
// Score bounds (LIVE, DNA forward): with a score F that the pair is known to reach
// (sw_bound.cu, or the best of the strips before), a strip need only compute rows that an
// alignment scoring F or more can visit.  From a row of the left edge whose H lies below
// F - match x (the columns from there on), no alignment reaches F: the others are live.
// Once no alignment can begin in the strip either (F above match x its and later columns),
// it starts at the first live row and ends where the last one's can have got to: the
// strip's columns further down, and as many gap symbols as its H has to spare.  Rows left
// out count as empty ones, which only lowers cells that no such alignment visits, so the
// best cells, all of them, stay.  A unit computes the rows of both halves, and the schedule
// brings together pairs with like diagonals.  100,000 reads, four of five related: forward
// 4.19 -> 3.70 ms without that order, with it 3.26; long pairs of the mixed shape 55.7 -> 27.
// The reverse pass (LIVE) knows its score.  Its alignments begin in the first column
// (reverse_band), so that none begins in a later strip, and a row of a strip's edge is live
// if its H and match x (the rows from there on) reach the score: of the band, which has
// the same width in every strip, that leaves half.
//
// Measured, 100,000 reads against contigs (8 lanes): forward 4.65 -> 4.19 ms, reverse
// (16 lanes) 1.92 -> 1.49 against one row of 16 columns a step with a row test in every
// step; long DNA pairs of the mixed shape 58.3 -> 55.7 and 23.2 -> 18.4 ms; 27,000
// proteins of 32 lanes 1.75 -> 1.17, reverse of 16 lanes 1.29 -> 0.77.  The ALU pipe is
// busy 81% (reverse 87%) of the forward pass; the cell block is 5.5 of its 7 instructions
// a cell pair.  Slower: chunks of 8 steps forward (their rows leave room for two blocks an
// SM, 4.71 ms), of 2 steps (5.16), 16 columns a lane (5.04), the max of every step kept in
// shared memory in place of the step test (4.54).
#include "strip_device.cuh"
#include "sw_device.cuh"
#include "sw_kernels.h"

namespace gbsw {
namespace {

constexpr int kDualCols = 8;  // columns a lane (protein in 32 lanes: 4)
// Steps of a chunk: its rows are fetched together and forward kept in shared memory,
// 4 KB a row and block at 8 columns, where 8 rows still let four blocks share an SM.
template <bool REVERSE, bool AA, int G>
__host__ __device__ constexpr int dual_steps() {
    return REVERSE || (AA && G == 32) ? 8 : 4;
}
constexpr unsigned kPadCode = 4;  // DNA row code outside the pair
// Selector byte of a row code: base q selects byte q sign-extended; kPadCode the
// sign of byte 0 twice, a score of 0 or -1, so a padding row never scores above 0.
// + 0x44: the same of pair B's scores (bytes 4-7).
constexpr unsigned kSelTableLo = 0xB3A29180u, kSelTableHi = 0x88u;

// One pair of a unit, as the kernel reads it (shared memory).
struct Half {
    const uint8_t* rowseq;
    const uint8_t* colseq;
    int pid;                 // -1: empty slot
    int nrows, ncols;
    int ncols_run;           // columns computed (reverse: bounded, see reverse_columns)
    int pad;
    int band, low;           // reverse: reverse_band, reverse_low_band (-1: every row)
    int target;              // reverse: the forward score
    int floor;               // forward: a score the pair reaches (0: none known)
    int a_short;
};

// The unit's band (reverse_band) and its other side: the larger of its halves'
// (-1: a half without one).
__device__ __forceinline__ int unit_band(const Half& a, const Half& b) {
    const bool has_a = a.nrows > 0, has_b = b.nrows > 0;
    if ((has_a && a.band < 0) || (has_b && b.band < 0)) return -1;
    return max(has_a ? a.band : 0, has_b ? b.band : 0);
}
__device__ __forceinline__ int unit_low_band(const Half& a, const Half& b) {
    const bool has_a = a.nrows > 0, has_b = b.nrows > 0;
    if ((has_a && a.low < 0) || (has_b && b.low < 0)) return -1;
    return max(has_a ? a.low : 0, has_b ? b.low : 0);
}

// Dynamic shared memory: forward, the chunk's rows; protein, the strip profiles.
template <bool REVERSE, bool AA, int G, int C>
__host__ __device__ constexpr size_t dual_row_bytes() {
    return REVERSE ? 0 : (size_t)2 * dual_steps<REVERSE, AA, G>() * kThreads * C * sizeof(int);
}
template <bool REVERSE, bool AA, int G, int C>
constexpr size_t dual_smem() {
    return dual_row_bytes<REVERSE, AA, G, C>() + (AA ? (size_t)2 * kAAProfRows * kThreads * C : 0);
}

template <bool REVERSE, bool LIVE>
__device__ __forceinline__ void load_half(const PassParams& p, Half& h, int pid) {
    h = Half{};
    h.pid = pid;
    h.rowseq = h.colseq = p.ref;
    h.band = h.low = -1;
    if (pid < 0) return;
    const int64_t ra = p.ref_off[pid], rb = p.ref_off[pid + 1];
    const int64_t qa = p.query_off[pid], qb = p.query_off[pid + 1];
    const uint8_t* A = p.ref + ra;
    const uint8_t* B = p.query + qa;
    const int a = (int)(rb - ra), b = (int)(qb - qa);
    if constexpr (!REVERSE) {
        if (max(a, b) > p.scratch_rows) {
            atomicOr(p.error, kErrBounds);
            return;
        }
        h.a_short = a < b;  // kernel.cpp:248
        h.colseq = h.a_short ? A : B;
        h.rowseq = h.a_short ? B : A;
        h.ncols = h.ncols_run = h.a_short ? a : b;
        h.nrows = h.a_short ? b : a;
        if (LIVE) h.floor = min(p.bound[pid].x, p.dual_limit);
    } else {
        const int target = p.score[pid];
        const int na = p.ref_end[pid], nb = p.query_end[pid];
        if (target <= 0) return;  // begins were written by the forward pass
        if (na < 1 || na > a || nb < 1 || nb > b || a > p.scratch_rows || b > p.scratch_rows) {
            atomicOr(p.error, kErrBounds);
            return;
        }
        h.target = target;
        h.a_short = na < nb;  // kernel.cpp:444; transposed: rows = shorter prefix
        h.rowseq = h.a_short ? A : B;
        h.colseq = h.a_short ? B : A;
        h.nrows = h.a_short ? na : nb;
        h.ncols = h.a_short ? nb : na;
        h.ncols_run = reverse_columns(a, b, na, nb, target, p.match, p.rev_p);
        h.band = reverse_band(a, b, na, nb, target, p.match, p.rev_p);
        h.low = reverse_low_band(a, b, na, nb, target, p.match, p.rev_p);
    }
}

template <bool REVERSE, bool LIVE>
__device__ __forceinline__ void write_half(const PassParams& p, const Half& h, uint64_t best) {
    const int pid = h.pid;
    if (pid < 0) return;
    if constexpr (!REVERSE) {
        const int v = (int)(best >> 32);
        if (LIVE && v < h.floor) atomicOr(p.error, kErrNoHit);
        if (v > p.dual_limit) {  // may have wrapped in int16: rerun in int32
            p.rerun[2 + atomicAdd(p.rerun + 1, 1)] = pid;
            p.pair_cls[pid] = 0;
            return;
        }
        if (v <= 0) {
            p.score[pid] = 0;
            p.ref_end[pid] = p.query_end[pid] = -1;
            p.ref_begin[pid] = p.query_begin[pid] = -1;
            return;
        }
        const int row = 0xFFFF - (int)((best >> 16) & 0xFFFF);
        const int col = tie_key(0xFFFF - (int)(best & 0xFFFF)) + 1;
        p.score[pid] = v;
        p.query_end[pid] = h.a_short ? row : col;  // kernel.cpp:381-392
        p.ref_end[pid] = h.a_short ? col : row;
    } else {
        if (h.target <= 0 || best == ~0ull) {
            if (h.target > 0) atomicOr(p.error, kErrNoHit);
            p.ref_begin[pid] = p.query_begin[pid] = -1;
            return;
        }
        const int begin_s = h.nrows - (int)(best >> 32);           // kernel.cpp:580
        const int begin_l = h.ncols - (int)(best & 0xffffffffu);   // kernel.cpp:579
        p.ref_begin[pid] = h.a_short ? begin_s : begin_l;          // kernel.cpp:591-600
        p.query_begin[pid] = h.a_short ? begin_l : begin_s;
    }
}

template <bool REVERSE, bool AA, int G, int C, bool LIVE>
__global__ void __launch_bounds__(kThreads, REVERSE && !AA ? 5 : 4) sw_pass_dual(PassParams p) {
    let_next_start();
    constexpr int W = G * C, kGroups = kThreads / G;
    constexpr int kDualSteps = dual_steps<REVERSE, AA, G>(), kDualRows = 2 * kDualSteps;
    constexpr int kDualUnroll = !REVERSE && !AA ? 4 : 2;
    static_assert(G >= 4 && G <= 32 && (G & (G - 1)) == 0 && (C == 4 || C == 8 || C == 16), "group geometry");
    constexpr int kSaved = REVERSE ? 1 : 2;
    constexpr int kFetch = (kDualRows + G - 1) / G;  // rows a lane fetches for a chunk
    // what lane 0 takes in at each step of this and the next chunk: {H + open, E} of
    // the strip edge in its two rows, and the row codes (A, B, A, B)
    __shared__ __align__(16) uint4 s_edge[kGroups][2][kDualSteps];
    __shared__ unsigned s_code[kGroups][2][kDualSteps];
    __shared__ Half s_half[kGroups][2];
    // per half, the two rows where this lane's max last grew (reverse: the row that reached the score)
    __shared__ __align__(16) int4 ssave[2][kSaved][C / 4][kThreads];
    __shared__ unsigned s_floor[kThreads];
    // forward: the Ho from which a row of this strip's edge is live (both halves), and the
    // rows of the next strip that live ones reach
    __shared__ unsigned s_thr[LIVE && !REVERSE ? kGroups : 1];
    __shared__ int2 s_live[LIVE ? kGroups : 1];
    __shared__ uint64_t s_best[2][kThreads];
    extern __shared__ __align__(16) unsigned char sdyn[];
    int4(*const srow)[C / 4][kThreads] = reinterpret_cast<int4(*)[C / 4][kThreads]>(sdyn);
    unsigned char* const prof = sdyn + dual_row_bytes<REVERSE, AA, G, C>() + (size_t)threadIdx.x * C;
    constexpr unsigned kResidue = kThreads * C;  // bytes from one residue's slice to the next
    __shared__ int smat[AA ? kAADim * kAADim : 1];
    __shared__ int senc[AA ? 128 : 1];
    if constexpr (AA) {
        // forward: rows carry the longer sequence = the matrix's first index;
        // reverse (transposed): rows carry the shorter one = the second index
        for (int k = threadIdx.x; k < kAADim * kAADim; k += blockDim.x) {
            const int r = k / kAADim, c = k % kAADim;
            smat[k] = REVERSE ? p.aa_matrix[c * kAADim + r] : p.aa_matrix[k];
        }
        // symbol -> matrix index (driver.cpp:252-258); bytes outside the table were
        // flagged by the schedule and read as 'A'
        for (int k = threadIdx.x; k < 128; k += blockDim.x) senc[k] = k < 91 ? p.aa_encoding[k] : 0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, g = lane % G, grp = threadIdx.x / G;
    const unsigned gmask = G == 32 ? kFull : (((1u << (G & 31)) - 1u) << (lane - g));
    const int src = g > 0 ? lane - 1 : lane;
    const long long group_id = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G;
    int2* const bnd = p.scratch + (size_t)group_id * (size_t)p.scratch_rows;
    const int open = p.open, ext = p.ext, max_score = max(p.match, max(p.mismatch, 0));
    const unsigned open2 = pack16(open, open), ext2 = pack16(ext, ext);
    const unsigned gmax2 = pack16(max(open, ext), max(open, ext));  // E' = max(E + gmax, T, 0)
    const int qbegin = p.class_range[2 * p.cls], qend = p.class_range[2 * p.cls + 1];
    Half* const half = s_half[grp];

    // ---- group state ----
    bool busy = false, done = false, last_strip = true;
    int nstrips = 0, strip = 0, t = 0, t_end = 0, buf = 0;
    int nrows = 0;      // the taller pair's rows
    int have = 0;       // rows the previous strip's edge holds
    int last_rows = 0;  // live rows: the previous strip's last row
    int write_rows = 0; // rows whose edge goes to the next strip (0: last strip)
    // ---- lane state ----
    unsigned ho[C], f[C], pa[AA ? 1 : C], pb[AA ? 1 : C];
    unsigned diag0 = open2, x_ho[2] = {open2, open2}, x_e[2] = {0, 0}, x_code = 0, mx = open2;
    int mi_a = 0, mi_b = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        ho[c] = open2;
        f[c] = 0;
        if constexpr (!AA) pa[c] = pb[c] = 0x80808080u;
    }

    // groups that never get a unit run on these (protein: they index the profiles)
    for (int k = g; k < 2 * kDualSteps; k += G) (&s_code[grp][0][0])[k] = 0;
    __syncwarp();

    // code of row i of half x: DNA a selector byte, protein a residue
    auto row_code = [&](int x, int i) -> unsigned {
        const Half& h = half[x];
        const bool real = i >= 1 && i <= h.nrows;
        const int v = real ? (int)h.rowseq[REVERSE ? h.nrows - i : i - 1] : 0;
        if constexpr (AA) return real ? (unsigned)senc[v & 127] : (unsigned)kAAPad;
        return prmt(kSelTableLo, kSelTableHi, real ? (unsigned)dna_code(v) : kPadCode) & 0xffu;
    };
    // The rows of the chunk that starts at step t0: lane g fetches rows 2 t0 + 1 + g
    // (+ G), a chunk before they are needed.
    int sym[kFetch][2];
    int2 edge[kFetch];
    auto issue = [&](int t0) {
#pragma unroll
        for (int k = 0; k < kFetch; ++k) {
            const int j = g + k * G, i = 2 * t0 + 1 + j;
            edge[k] = make_int2((int)open2, 0);
            sym[k][0] = sym[k][1] = -1;
            if (j < kDualRows) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const Half& h = half[x];
                    if (i <= h.nrows) sym[k][x] = (int)h.rowseq[REVERSE ? h.nrows - i : i - 1];
                }
                if (strip > 0 && i <= have) edge[k] = __ldcg(bnd + (i - 1));
            }
        }
    };
    auto commit = [&](int b) {
#pragma unroll
        for (int k = 0; k < kFetch; ++k) {
            const int j = g + k * G;
            if (j < kDualRows) {
                reinterpret_cast<int2*>(&s_edge[grp][b][j >> 1])[j & 1] = edge[k];
                unsigned c[2];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int v = sym[k][x];
                    if constexpr (AA) c[x] = v < 0 ? (unsigned)kAAPad : (unsigned)senc[v & 127];
                    else c[x] = prmt(kSelTableLo, kSelTableHi, v < 0 ? kPadCode : (unsigned)dna_code(v)) & 0xffu;
                }
                reinterpret_cast<unsigned short*>(&s_code[grp][b][j >> 1])[j & 1] = (unsigned short)(c[0] | (c[1] << 8));
            }
        }
    };

    auto setup_strip = [&]() {
        const int t_a = strip * W + g * C - half[0].pad, t_b = strip * W + g * C - half[1].pad;
        if constexpr (AA) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const Half& h = half[x];
                int cc[C];  // matrix column of each of this lane's columns; -1: padding
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int k = (x ? t_b : t_a) + c;
                    cc[c] = (k >= 0 && k < h.ncols) ? senc[h.colseq[REVERSE ? h.ncols - 1 - k : k] & 127] : -1;
                }
                for (int e = 0; e < kAAProfRows; ++e) {  // the last: the padding row
#pragma unroll
                    for (int q = 0; q < C / 4; ++q) {
                        unsigned w = 0;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int c = 4 * q + j;
                            const int v = (cc[c] < 0 || e == kAAPad) ? kNegByte : smat[e * kAADim + cc[c]];
                            w |= ((unsigned)v & 0xffu) << (8 * j);
                        }
                        *reinterpret_cast<unsigned*>(prof + (size_t)(x * kAAProfRows + e) * kResidue + 4 * q) = w;
                    }
                }
            }
        } else {
            auto column_profile = [&](const Half& h, int k) -> unsigned {
                if (k < 0 || k >= h.ncols) return 0x80808080u;  // padding: -128 against every base
                const int code = dna_code(h.colseq[REVERSE ? h.ncols - 1 - k : k]);
                unsigned w = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) w |= ((unsigned)(code == q ? p.match : p.mismatch) & 0xffu) << (8 * q);
                return w;
            };
#pragma unroll
            for (int c = 0; c < C; ++c) {
                pa[c] = column_profile(half[0], t_a + c);
                pb[c] = column_profile(half[1], t_b + c);
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            ho[c] = open2;
            f[c] = 0;
        }
        diag0 = x_ho[0] = x_ho[1] = open2;
        x_e[0] = x_e[1] = 0;
        mi_a = mi_b = 0;
        last_strip = strip + 1 == nstrips;
        int lanes = G, last_row = nrows;
        if constexpr (REVERSE) {
            const int band = unit_band(half[0], half[1]), low = unit_low_band(half[0], half[1]);
            last_row = band_last_row(strip * W + W, low, nrows);
            have = band_last_row(strip * W, low, nrows);
            int first_row = min(band_first_row(strip * W + 1, band), last_row);
            if constexpr (LIVE) {
                if (strip > 0) {
                    first_row = max(first_row, s_live[grp].x);
                    last_row = min(last_row, s_live[grp].y);
                    have = last_rows;
                }
                last_rows = last_row;
                if (!last_strip) {
                    // halves without a band may begin an alignment in any strip
                    int2 live = make_int2(nrows + 1, 0);
#pragma unroll
                    for (int x = 0; x < 2; ++x)
                        if (half[x].nrows > 0 && half[x].band < 0) live = make_int2(1, max(live.y, half[x].nrows));
                    __syncwarp(gmask);  // s_live is read
                    if (g == 0) s_live[grp] = live;
                }
            }
            t = (first_row - 1) / 2;
            lanes = min(G, (max(half[0].ncols_run, half[1].ncols_run) - strip * W + C - 1) / C);
            // one below the score a half looks for, which it so passes once
            mx = pack16(half[0].target > 0 ? half[0].target - 1 + open : 0x7fff,
                        half[1].target > 0 ? half[1].target - 1 + open : 0x7fff);
        } else {
            have = LIVE ? last_rows : nrows;
            // lanes of padding only are the matrix boundary whatever the row
            t = strip == 0 ? min(half[0].pad, half[1].pad) / C : 0;
            if (LIVE && strip > 0) {
                t = (s_live[grp].x - 1) / 2;
                last_row = s_live[grp].y;
            }
            last_rows = last_row;
            if (LIVE && !last_strip) {
                unsigned thr = 0;
                int2 live = make_int2(nrows + 1, 0);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int fl = (x ? hi16(s_floor[threadIdx.x]) : lo16(s_floor[threadIdx.x])) - open + 1;
                    const int gain = max_score * (half[x].ncols - max(0, (strip + 1) * W - half[x].pad));
                    const bool all = half[x].nrows > 0 && gain >= fl;
                    if (all) live = make_int2(1, max(live.y, half[x].nrows));
                    thr |= (unsigned)(unsigned short)(all || half[x].nrows == 0 ? 0x7fff : fl - gain + open) << (16 * x);
                }
                __syncwarp(gmask);  // s_live is read
                if (g == 0) {
                    s_thr[grp] = thr;
                    s_live[grp] = live;
                }
            }
        }
        t_end = (last_row + 1) / 2 + lanes - 1;
        write_rows = last_strip ? 0 : last_row;
        issue(t);
        // what each lane would have worked on a step before: its right neighbour takes it
        const int i = 2 * (t - 1 - g) + 1;
        x_code = row_code(0, i) | (row_code(1, i) << 8) | (row_code(0, i + 1) << 16) | (row_code(1, i + 1) << 24);
        buf = 0;
        commit(0);
    };

    // Forward: saves the two rows of the step in which half x last grew its max (u: that
    // step; before: the max before the chunk) and returns the first one; 0: none that counts.
    auto settle = [&](int x, int t0, int u, unsigned before) -> int {
        const int r0 = 2 * (t0 - g) + 1;  // the lane's first row of the chunk
        const int rows = half[x].nrows - r0 + 1;
        if (rows < kDualRows) {
            int k = -1, top = x ? hi16(before) : lo16(before);
            for (int j = max(0, 1 - r0); j < rows; ++j) {
                int m = -32768;
#pragma unroll
                for (int q = 0; q < C / 4; ++q) {
                    const int4 v = srow[j][q][threadIdx.x];
                    const unsigned w = __vmaxs2(__vmaxs2((unsigned)v.x, (unsigned)v.y), __vmaxs2((unsigned)v.z, (unsigned)v.w));
                    m = max(m, x ? hi16(w) : lo16(w));
                }
                if (m > top) {
                    top = m;
                    k = j;
                }
            }
            if (k < 0) return 0;
            u = k >> 1;
        }
        const int second = min(2 * u + 1, rows - 1);  // a row past the last one doesn't count
#pragma unroll
        for (int q = 0; q < C / 4; ++q) {
            ssave[x][0][q][threadIdx.x] = srow[2 * u][q][threadIdx.x];
            ssave[x][kSaved - 1][q][threadIdx.x] = srow[second][q][threadIdx.x];
        }
        return r0 + 2 * u;
    };
    // Reverse: looks for the scores in row i.
    auto check_row = [&](int i, const unsigned (&h)[C]) {
        unsigned row = h[0];
#pragma unroll
        for (int c = 1; c < C; ++c) row = __vmaxs2(row, h[c]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            if ((x ? hi16(row) > hi16(mx) : lo16(row) > lo16(mx)) && (unsigned)(i - 1) < (unsigned)half[x].nrows) {
                (x ? mi_b : mi_a) = i;
                mx = prmt(mx, row, x ? 0x7610u : 0x3254u);
#pragma unroll
                for (int k = 0; k < C / 4; ++k)
                    ssave[x][0][k][threadIdx.x] =
                        make_int4((int)h[4 * k], (int)h[4 * k + 1], (int)h[4 * k + 2], (int)h[4 * k + 3]);
            }
        }
    };

    while (true) {
        if (!done && !busy) {
            int q = 0;
            if (g == 0) q = atomicAdd(p.queue, 1);
            q = __shfl_sync(gmask, q, lane - g);
            const int k0 = qbegin + 2 * q;
            if (k0 >= qend) {
                done = true;
                write_rows = 0;
                if (g < 2) half[g].nrows = 0;  // the rest of the warp's chunks run on padding
                __syncwarp(gmask);
            } else {
                if (g < 2) load_half<REVERSE, LIVE>(p, half[g], k0 + g < qend ? p.order[k0 + g] : -1);
                __syncwarp(gmask);
                nrows = max(half[0].nrows, half[1].nrows);
                nstrips = (max(half[0].ncols_run, half[1].ncols_run) + W - 1) / W;
                if (nrows == 0 || nstrips == 0) {
                    if (g < 2) write_half<REVERSE, LIVE>(p, half[g], REVERSE ? ~0ull : 0ull);
                } else {
                    // forward: left-padded; reverse: padded on the right, which keeps
                    // the band's first rows those of the real columns
                    if (g < 2) half[g].pad = REVERSE ? 0 : nstrips * W - half[g].ncols_run;
                    s_best[0][threadIdx.x] = s_best[1][threadIdx.x] = REVERSE ? ~0ull : 0ull;
                    __syncwarp(gmask);
                    strip = 0;
                    if constexpr (!REVERSE)
                        mx = s_floor[threadIdx.x] = LIVE ? pack16(max(half[0].floor - 1, 0) + open, max(half[1].floor - 1, 0) + open) : open2;
                    busy = true;
                    setup_strip();
                }
                __syncwarp(gmask);
            }
        }
        if (__all_sync(kFull, done)) break;
        if (__any_sync(kFull, !done && !busy)) continue;  // an empty unit: take the next one

        // ---- kDualSteps steps, every lane of the warp ----
        if (busy) issue(t + kDualSteps);
        const unsigned before = mx;
        int grew_a = -1, grew_b = -1;
#pragma unroll kDualUnroll
        for (int u = 0; u < kDualSteps; ++u) {
            unsigned code = __shfl_sync(kFull, x_code, src);
            unsigned ho_in[2] = {__shfl_sync(kFull, x_ho[0], src), __shfl_sync(kFull, x_ho[1], src)};
            unsigned e[2] = {__shfl_sync(kFull, x_e[0], src), __shfl_sync(kFull, x_e[1], src)};
            if (g == 0) {
                const uint4 in = s_edge[grp][buf][u];
                ho_in[0] = in.x;
                e[0] = in.y;
                ho_in[1] = in.z;
                e[1] = in.w;
                code = s_code[grp][buf][u];
            }
            x_code = code;
            // DNA: the selectors of both rows, pair B's from bytes 4-7
            const unsigned sel[2] = {code + 0x44004400u, (code + 0x44004400u) >> 16};
            unsigned wa[2][AA ? C / 4 : 1], wb[2][AA ? C / 4 : 1];
            if constexpr (AA) {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const unsigned char* at_a = prof + ((code >> (16 * r)) & 0xffu) * kResidue;
                    const unsigned char* at_b = prof + (kAAProfRows + ((code >> (16 * r + 8)) & 0xffu)) * kResidue;
                    if constexpr (C == 8) {
                        const uint2 va = *reinterpret_cast<const uint2*>(at_a), vb = *reinterpret_cast<const uint2*>(at_b);
                        wa[r][0] = va.x;
                        wa[r][C / 4 - 1] = va.y;
                        wb[r][0] = vb.x;
                        wb[r][C / 4 - 1] = vb.y;
                    } else {
                        wa[r][0] = *reinterpret_cast<const unsigned*>(at_a);
                        wb[r][0] = *reinterpret_cast<const unsigned*>(at_b);
                    }
                }
            }
            unsigned diag[2] = {diag0, ho_in[0]}, first[C];  // first: H + open of the first row
            unsigned grow = mx;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                unsigned up = ho[c], fv = f[c];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const unsigned s2 = AA ? prmt(wa[r][c / 4], wb[r][c / 4], (c % 4) * 0x1111u + 0xC480u)
                                           : prmt(pa[AA ? 0 : c], pb[AA ? 0 : c], sel[r]);
                    fv = __viaddmax_s16x2_relu(fv, ext2, up);                // F(i,j)
                    const unsigned u2 = __vadd2(diag[r], s2);                // Ho_diag + s
                    const unsigned tv = __viaddmax_s16x2(fv, open2, u2);     // max(F + open, .)
                    const unsigned hov = __viaddmax_s16x2(e[r], open2, tv);  // Ho(i,j)
                    e[r] = __viaddmax_s16x2_relu(e[r], gmax2, tv);           // E(i,j+1)
                    diag[r] = up;
                    up = hov;
                    if (r == 0) first[c] = hov;
                }
                ho[c] = up;
                f[c] = fv;
                grow = __vimax3_s16x2(grow, first[c], up);
            }
            x_e[0] = e[0];
            x_e[1] = e[1];
            x_ho[0] = first[C - 1];
            x_ho[1] = ho[C - 1];
            diag0 = ho_in[1];
            const int i = 2 * (t + u - g) + 1;
            if (g == G - 1 && (unsigned)(i - 1) < (unsigned)write_rows)
                __stcg(reinterpret_cast<int4*>(bnd + (i - 1)),
                       make_int4((int)first[C - 1], (int)e[0], (int)ho[C - 1], (int)e[1]));
            if constexpr (REVERSE) {
                // a half reaches its score once, so the branch is rarely taken
                if (grow != mx) {
                    check_row(i, first);
                    check_row(i + 1, ho);
                }
            } else {
                if (((grow ^ mx) & 0xffffu) != 0) grew_a = u;
                if (((grow ^ mx) & 0xffff0000u) != 0) grew_b = u;
                mx = grow;
#pragma unroll
                for (int q = 0; q < C / 4; ++q) {
                    srow[2 * u][q][threadIdx.x] = make_int4((int)first[4 * q], (int)first[4 * q + 1],
                                                            (int)first[4 * q + 2], (int)first[4 * q + 3]);
                    srow[2 * u + 1][q][threadIdx.x] =
                        make_int4((int)ho[4 * q], (int)ho[4 * q + 1], (int)ho[4 * q + 2], (int)ho[4 * q + 3]);
                }
            }
        }
        if (!REVERSE && grew_a >= 0) {
            const int row = settle(0, t, grew_a, before);
            mi_a = row > 0 ? row : mi_a;
        }
        if (!REVERSE && grew_b >= 0) {
            const int row = settle(1, t, grew_b, before);
            mi_b = row > 0 ? row : mi_b;
        }
        if constexpr (LIVE) {
            if (g == G - 1 && write_rows > 0) {
                // Live rows among the chunk's: none of its edge values (E is at most H) lies
                // further above its last row's H than a gap down to there costs.
                const int r0 = 2 * (t - g) + 1;  // the chunk's first row here
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    int over = (x ? hi16(ho[C - 1]) : lo16(ho[C - 1])) - (open + (kDualRows - 2) * ext);
                    int each = -max(open, ext);  // a gap symbol's least cost
                    bool live_rows = true;
                    if constexpr (REVERSE) {
                        // the score must be reached over the rows that are left, and a gap takes some
                        const int rows = half[x].nrows - r0 + 1;
                        over += max_score * rows - half[x].target - open;
                        each += max_score;
                        live_rows = rows > 0 && half[x].band >= 0;
                    } else {
                        over -= x ? hi16(s_thr[grp]) : lo16(s_thr[grp]);
                    }
                    if (live_rows && over >= 0) {
                        const int reach = each > 0 ? over / each : nrows;
                        int2 live = s_live[grp];
                        live.x = min(live.x, max(r0, 1));
                        live.y = max(live.y, min(nrows, r0 + kDualRows - 1 + W + reach));
                        s_live[grp] = live;
                    }
                }
            }
        }
        t += kDualSteps;
        if (busy && t < t_end) {
            buf ^= 1;
            commit(buf);
        } else if (busy) {
            // ---- end of strip: this lane's candidates ----
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int mi = x ? mi_b : mi_a;
                if (mi > 0) {
                    const int t0 = strip * W + g * C - half[x].pad;
#pragma unroll
                    for (int r = 0; r < kSaved; ++r) {
                        int v[C], want = -32768;
#pragma unroll
                        for (int k = 0; k < C / 4; ++k) {
                            const int4 w = ssave[x][r][k][threadIdx.x];
                            const int ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                v[4 * k + j] = x ? hi16((unsigned)ww[j]) : lo16((unsigned)ww[j]);
                                want = max(want, v[4 * k + j]);
                            }
                        }
                        // the columns that hold the row's max: forward the first in tie
                        // order, reverse the leftmost
                        int pick = REVERSE ? C : 0x7fffffff;
#pragma unroll
                        for (int c = 0; c < C; ++c)
                            if (v[c] == want) pick = min(pick, REVERSE ? c : tie_key(t0 + c));
                        const uint64_t cand = REVERSE ? (((uint64_t)(uint32_t)mi << 32) | (uint32_t)(t0 + pick + 1))
                                                      : pack_fwd(want - open, mi + r, pick);
                        const uint64_t best = s_best[x][threadIdx.x];
                        if (REVERSE ? cand < best : cand > best) s_best[x][threadIdx.x] = cand;
                    }
                }
            }
            if constexpr (!REVERSE) {
                // a cell below the best of the strips so far can't win: the next strip's
                // max starts one below it (a cell equal to it may come first in the tie order)
                unsigned top = mx;
#pragma unroll
                for (int off = G / 2; off > 0; off >>= 1) top = __vmaxs2(top, __shfl_xor_sync(gmask, top, off, G));
                mx = __vmaxs2(s_floor[threadIdx.x], __vsub2(top, 0x00010001u));
                s_floor[threadIdx.x] = mx;
            }
            __syncwarp(gmask);  // this strip's edge before the next one reads it
            ++strip;
            if (strip < nstrips && (!LIVE || s_live[grp].x <= s_live[grp].y)) {
                setup_strip();
            } else {
                uint64_t a = s_best[0][threadIdx.x], b = s_best[1][threadIdx.x];
#pragma unroll
                for (int off = G / 2; off > 0; off >>= 1) {
                    const uint64_t oa = __shfl_xor_sync(gmask, a, off, G), ob = __shfl_xor_sync(gmask, b, off, G);
                    a = REVERSE ? (oa < a ? oa : a) : (oa > a ? oa : a);
                    b = REVERSE ? (ob < b ? ob : b) : (ob > b ? ob : b);
                }
                if (g < 2) write_half<REVERSE, LIVE>(p, half[g], g ? b : a);
                busy = false;
                write_rows = 0;
            }
        }
        __syncwarp();
    }
    end_after_previous(p);
}

template <bool AA, int G, int C>
const void* dual_pass(bool reverse, bool live, size_t* dyn) {
    *dyn = reverse ? dual_smem<true, AA, G, C>() : dual_smem<false, AA, G, C>();
    if constexpr (!AA) {
        if (live) return reverse ? (const void*)sw_pass_dual<true, AA, G, C, true> : (const void*)sw_pass_dual<false, AA, G, C, true>;
    }
    return reverse ? (const void*)sw_pass_dual<true, AA, G, C, false> : (const void*)sw_pass_dual<false, AA, G, C, false>;
}

// Kernel and dynamic shared memory of a dual variant (`live`: DNA, live rows only);
// nullptr if none.  DNA widths name a strip of 16 columns a lane (64, 128, 256
// columns); the kernel runs it with twice the lanes of 8 columns.
const void* pick_dual(bool reverse, bool aa, int width, bool live, size_t* dyn) {
    *dyn = 0;
    if (!aa) {
        if (width == 4) return dual_pass<false, 8, kDualCols>(reverse, live, dyn);
        if (width == 8) return dual_pass<false, 16, kDualCols>(reverse, live, dyn);
        if (width == 16) return dual_pass<false, 32, kDualCols>(reverse, live, dyn);
        return nullptr;
    }
    if (width == 16) return dual_pass<true, 16, 8>(reverse, live, dyn);
    if (width == 32) return dual_pass<true, 32, 4>(reverse, live, dyn);
    return nullptr;
}

cudaError_t prepare(bool reverse, bool aa, int width, bool live, const void** fn, size_t* dyn) {
    *fn = pick_dual(reverse, aa, width, live, dyn);
    if (!*fn) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(*fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*dyn);
}

}  // namespace

int dual_lanes(bool aa, int width) { return aa ? width : 2 * width; }

bool has_dual(bool aa, int width) {
    size_t dyn;
    return pick_dual(false, aa, width, false, &dyn) != nullptr;
}

cudaError_t launch_pass_dual(bool reverse, bool aa, int width, const PassParams& p, int blocks,
                             cudaStream_t stream) {
    // Reverse: where strips are many.  Long pairs of the mixed shape 18.4 -> 14.8 ms; 100,000
    // reads 1.49 -> 1.56, 200,000 pairs of 100-150 against 200-500 symbols 1.16 -> 1.36.
    const bool live = reverse ? p.cls == kRangeLong : p.bound != nullptr;
    size_t dyn = 0;
    const void* fn = nullptr;
    cudaError_t e = prepare(reverse, aa, width, live, &fn, &dyn);
    if (e != cudaSuccess) return e;
    void* args[] = {(void*)&p};
    return launch_beside(fn, blocks, kThreads, args, dyn, stream, p.join != 0);
}

cudaError_t pass_dual_occupancy(bool reverse, bool aa, int width, int* blocks_per_sm) {
    size_t dyn = 0;
    const void* fn = nullptr;
    cudaError_t e = prepare(reverse, aa, width, false, &fn, &dyn);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, kThreads, dyn);
}

}  // namespace gbsw
