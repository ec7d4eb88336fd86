// Strip-parallel passes: every column strip of every pair is a task of its own,
// and a warp runs a strip in int16x2, for batches too small to fill the GPU with
// pairs (one long read, a handful of them, a thousand short ones).
//
// 64 lanes in a warp.  A strip is 64 * C columns.  Lane g holds columns
// [g * C, g * C + C) in the low halves of its registers (virtual lane g) and the C
// columns 32 * C further right in the high halves (virtual lane 32 + g).  Rows
// stream through the 64 virtual lanes as a pipeline, two at a time: at step t
// virtual lane v works on rows 2 (t - v) + 1 and 2 (t - v) + 2, so the high halves
// run 64 rows behind the low ones.  One rotating shuffle per value moves it on:
// lane g takes both halves of lane g - 1, and lane 0 takes the strip's left edge
// into its low half and lane 31's low half into its high half (one prmt).  Row
// symbols travel the same way, so each is fetched and converted once per warp.
// The cell update and the overflow rule are the two-pair kernels' (sw_dual.cu):
// half the ALU instructions of an int32 cell, from one pair.
//
// Two rows a step: such batches leave about one warp to a scheduler, whose time is
// a step's chain of shuffle (26 cycles), lane 0's prmt and the C serial updates of
// E (4 each); a second row adds one link to the chain and doubles its work.
//
// Tasks.  A pair's strips are consecutive tasks, pairs longest first; warps take
// tasks in order from one counter.  Strip s + 1 needs strip s's right edge row by
// row: its virtual lane 63 writes each row's H + open and E as one 8-byte word
// with the task's tag, and strip s + 1 polls that word, so data and readiness
// arrive together and no fence is needed.  A task only ever waits for tasks with
// lower numbers, which running warps hold already, so every wait ends; each is
// bounded all the same (kErrTeam).  Task k writes edge buffer k % ring, after the
// reader of that buffer's previous task is done with it.  The best of strips
// 0..s travels with the edges, and a pair's last strip writes its results.
//
// Forward pairs are padded to their strips on the left (as in sw_dual.cu); lanes
// that hold only padding are the matrix boundary whatever the row, so a pair's
// first strip starts at the step where its first real lane meets row 1.  Reverse
// strips cover the rows of the band (reverse_band, reverse_low_band) and end when
// the last lane that holds a real column has passed them.
//
// Why: the block-per-pair int32 team it replaces gave a pair four warps of 256
// columns each, so 61 long reads ran on 61 SMs, a warp to a scheduler, each step
// issuing twice the instructions; batches of some thousand pairs ran two pairs to
// a group and waited for the longest.  Measured (forward / reverse pass with their
// schedules): 61 reads of 3-12 kb 26.4 / 26.9 -> 2.35 / 1.69 ms; 3,000 mixed DNA pairs
// 2,834 / 1,549 -> 1,435 / 717 us; 6,000 DNA pairs of the throughput shape 875 / 513 ->
// 481 / 289; 500 proteins 290 / 510 -> 180 / 150; 6,000 proteins 1,175 / 1,427 -> 506 / 422.
// What bounds it: with a warp to a scheduler a step's dependent chain (215 cycles
// for some 75 ALU instructions at 4 columns), with more the ALU pipe.
#include <algorithm>

#include "sw_common.cuh"
#include "strip_device.cuh"
#include "sw_device.cuh"
#include "sw_strips.h"

namespace gbsw {
namespace {

constexpr int kStripSteps = 8;                // steps of a chunk
constexpr int kStripRows = 2 * kStripSteps;   // their rows, fetched together
constexpr int kHalfLag = 64;                  // rows the high halves run behind the low ones
// Entries of an edge buffer before row 1: the rows the last lane passes while
// the pipeline fills (even: a step's two rows are stored together).
constexpr int kEdgeFront = 128;
constexpr unsigned kPadCode = 4;  // DNA row code outside the pair
constexpr unsigned kSelTableLo = 0xB3A29180u, kSelTableHi = 0x88u;  // selector byte of a row code (sw_dual.cu)

// One pair as a pass sees it: rows stream, columns are held in registers.
struct PairView {
    const uint8_t* rowseq;
    const uint8_t* colseq;
    int nrows, ncols, ncols_run;  // ncols_run: columns computed (reverse: bounded, reverse_columns)
    int band, low;                // reverse: reverse_band, reverse_low_band (-1: none)
    int target;                   // reverse: the forward score
    bool a_short;
    int error;                    // error flag to raise, 0 if the pair is sound
};

template <bool REVERSE>
__device__ __forceinline__ PairView view_pair(const PassParams& p, int pid) {
    PairView v{};
    v.band = v.low = -1;
    const int64_t ra = p.ref_off[pid], rb = p.ref_off[pid + 1];
    const int64_t qa = p.query_off[pid], qb = p.query_off[pid + 1];
    const uint8_t* A = p.ref + ra;
    const uint8_t* B = p.query + qa;
    const int a = (int)(rb - ra), b = (int)(qb - qa);
    if constexpr (!REVERSE) {
        v.a_short = a < b;  // kernel.cpp:248
        v.colseq = v.a_short ? A : B;
        v.rowseq = v.a_short ? B : A;
        v.ncols = v.ncols_run = v.a_short ? a : b;
        v.nrows = v.a_short ? b : a;
        if (v.nrows > p.scratch_rows) v.error = kErrBounds;
    } else {
        v.target = p.score[pid];
        const int na = p.ref_end[pid], nb = p.query_end[pid];
        if (v.target <= 0) return v;
        if (na < 1 || na > a || nb < 1 || nb > b || a > p.scratch_rows || b > p.scratch_rows) {
            v.error = kErrBounds;
            return v;
        }
        v.a_short = na < nb;  // kernel.cpp:444; transposed: rows = shorter prefix
        v.rowseq = v.a_short ? A : B;
        v.colseq = v.a_short ? B : A;
        v.nrows = v.a_short ? na : nb;
        v.ncols = v.a_short ? nb : na;
        v.ncols_run = reverse_columns(a, b, na, nb, v.target, p.match, p.rev_p);
        v.band = reverse_band(a, b, na, nb, v.target, p.match, p.rev_p);
        v.low = reverse_low_band(a, b, na, nb, v.target, p.match, p.rev_p);
    }
    if (v.error) v.nrows = v.ncols = v.ncols_run = 0;
    return v;
}

// The pair's results from its combined key (forward: packed argmax; reverse:
// packed first hit, ~0 if none); one thread.
template <bool REVERSE>
__device__ __forceinline__ void write_result(const PassParams& p, int pid, const PairView& v, uint64_t best) {
    if constexpr (!REVERSE) {
        const int score = (int)(best >> 32);
        if (score > p.dual_limit) {  // may have wrapped in int16: rerun in int32
            p.rerun[2 + atomicAdd(p.rerun + 1, 1)] = pid;
            p.pair_cls[pid] = 0;
            return;
        }
        if (score <= 0) {
            p.score[pid] = 0;
            p.ref_end[pid] = p.query_end[pid] = -1;
            p.ref_begin[pid] = p.query_begin[pid] = -1;
            return;
        }
        const int row = 0xFFFF - (int)((best >> 16) & 0xFFFF);
        const int col = tie_key(0xFFFF - (int)(best & 0xFFFF)) + 1;
        p.score[pid] = score;
        p.query_end[pid] = v.a_short ? row : col;  // kernel.cpp:381-392
        p.ref_end[pid] = v.a_short ? col : row;
    } else {
        if (v.target <= 0 || best == ~0ull) {
            if (v.target > 0 && !v.error) atomicOr(p.error, kErrNoHit);
            p.ref_begin[pid] = p.query_begin[pid] = -1;
            return;
        }
        const int begin_s = v.nrows - (int)(best >> 32);           // kernel.cpp:580
        const int begin_l = v.ncols - (int)(best & 0xffffffffu);   // kernel.cpp:579
        p.ref_begin[pid] = v.a_short ? begin_s : begin_l;          // kernel.cpp:591-600
        p.query_begin[pid] = v.a_short ? begin_l : begin_s;
    }
}

__host__ __device__ constexpr size_t strip_row_bytes(int columns) {
    return (size_t)kStripRows * kThreads * columns * sizeof(int);
}

template <bool REVERSE, bool AA, int C>
__global__ void __launch_bounds__(kThreads, 4) sw_strips(PassParams p, StripParams s) {
    let_next_start();
    constexpr int W = strip_width(C);
    static_assert(C % 4 == 0 && kStripRows <= 32, "geometry");
    // what lane 0 takes in at each step of this and the next chunk: the edge words
    // of the step's two rows and their codes (bytes 0 and 2)
    __shared__ __align__(16) uint4 sin_[kThreads / 32][2][kStripSteps];
    // per half, the row where this lane's max last grew (reverse: reached the score)
    __shared__ __align__(16) int4 ssave[2][C / 4][kThreads];
    // dynamic: H + open of the chunk's rows, [row][quad of columns][thread], then
    // (protein) this thread's C profile bytes per half and residue
    extern __shared__ __align__(16) unsigned char sdyn[];
    int4(*const srow)[C / 4][kThreads] = reinterpret_cast<int4(*)[C / 4][kThreads]>(sdyn);
    __shared__ int smat[AA ? kAADim * kAADim : 1];
    __shared__ int senc[AA ? 128 : 1];
    constexpr unsigned kResidue = kThreads * C;  // bytes from one residue's slice to the next
    if constexpr (AA) {
        // forward: rows carry the longer sequence = the matrix's first index;
        // reverse (transposed): the shorter one = the second index
        for (int k = threadIdx.x; k < kAADim * kAADim; k += blockDim.x) {
            const int r = k / kAADim, c = k % kAADim;
            smat[k] = REVERSE ? p.aa_matrix[c * kAADim + r] : p.aa_matrix[k];
        }
        for (int k = threadIdx.x; k < 128; k += blockDim.x) senc[k] = k < 91 ? p.aa_encoding[k] : 0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int src = (lane + 31) & 31;
    // lane 0 takes the injected word into its low half and lane 31's low half into
    // its high half; the others take their left neighbour's word as it is
    const unsigned sel_ho = lane ? 0x3210u : 0x1054u;
    const unsigned sel_e = lane ? 0x3210u : 0x1076u;
    // code word: the low and the high half's row code of the step's first row, then
    // of its second one, a byte each (DNA a selector byte, protein a residue)
    const unsigned sel_code = lane ? 0x3210u : 0x2604u;
    const int open = p.open, ext = p.ext;
    const unsigned open2 = pack16(open, open), ext2 = pack16(ext, ext);
    const unsigned gmax2 = pack16(max(open, ext), max(open, ext));
    const unsigned zero_edge = (unsigned)open & 0xffffu;  // H = 0, E = 0
    const int ntasks = min(*s.ntasks, s.max_tasks);
    __shared__ int s_first;
    if (threadIdx.x == 0) s_first = strip_first_task(s, p.queue, ntasks);
    __syncthreads();
    int task = s_first + warp;

    unsigned char* const prof = sdyn + (REVERSE ? 0 : strip_row_bytes(C)) + (size_t)threadIdx.x * C;

    auto wait_words = [&](bool needs, const uint64_t* at, unsigned tag, uint64_t& v) -> bool {
        return strip_wait(p.error, needs, at, tag, v);
    };

    // the next task (every warp runs its tasks in increasing order)
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
        const PairView pv = view_pair<REVERSE>(p, pid);
        if (pv.nrows == 0 || pv.ncols_run == 0) {  // one task, nothing to compute
            if (lane == 0) {
                if (pv.error) atomicOr(p.error, pv.error);
                write_result<REVERSE>(p, pid, pv, REVERSE ? ~0ull : 0ull);
            }
            continue;
        }
        const int nrows = pv.nrows, ncols = pv.ncols;
        const int pad = REVERSE ? 0 : nstrips * W - pv.ncols_run;
        const int t_a = strip * W + lane * C - pad;  // real column (0-based) of the low half's first column
        const int t_b = t_a + 32 * C;
        // rows [.., last_row] of this strip, rows the previous strip's edge holds
        // and the first step
        int last_row = nrows, have = nrows, t = 0, lanes = 64;
        if constexpr (REVERSE) {
            last_row = band_last_row(strip * W + W, pv.low, nrows);
            have = band_last_row(strip * W, pv.low, nrows);
            t = (min(band_first_row(strip * W + 1, pv.band), last_row) - 1) / 2;  // the band's first row is odd
            lanes = min(64, (pv.ncols_run - strip * W + C - 1) / C);
        } else if (strip == 0) {
            t = pad / C;
        }
        const int t_end = (last_row + 1) / 2 + lanes - 1;
        // entry of row r: kEdgeFront + r - 1
        uint64_t* const e_out = s.edges + (size_t)(task % s.ring) * s.edge_stride;
        const uint64_t* const e_in = s.edges + (size_t)((task + s.ring - 1) % s.ring) * s.edge_stride;
        const bool writes = lane == 31;
        uint64_t* e_step = e_out + (kEdgeFront + 2 * (t - 63));
        if (!last && !strip_buffer_free(p.error, s, task)) break;

        // ---- column profiles ----
        unsigned pa[AA ? 1 : C], pb[AA ? 1 : C];
        if constexpr (AA) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                int cc[C];  // matrix column of this lane's columns; -1: padding
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int k = (x ? t_b : t_a) + c;
                    cc[c] = (k >= 0 && k < ncols) ? senc[pv.colseq[REVERSE ? ncols - 1 - k : k] & 127] : -1;
                }
                for (int e = 0; e < kAAProfRows; ++e) {  // the last: the padding row
#pragma unroll
                    for (int k = 0; k < C / 4; ++k) {
                        unsigned w = 0;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int c = 4 * k + j;
                            const int v = (cc[c] < 0 || e == kAAPad) ? kNegByte : smat[e * kAADim + cc[c]];
                            w |= ((unsigned)v & 0xffu) << (8 * j);
                        }
                        *reinterpret_cast<unsigned*>(prof + (size_t)(x * kAAProfRows + e) * kResidue + 4 * k) = w;
                    }
                }
            }
        } else {
            auto column_profile = [&](int k) -> unsigned {
                if (k < 0 || k >= ncols) return 0x80808080u;  // padding: -128 against every base
                const int code = dna_code(pv.colseq[REVERSE ? ncols - 1 - k : k]);
                unsigned w = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q) w |= ((unsigned)(code == q ? p.match : p.mismatch) & 0xffu) << (8 * q);
                return w;
            };
#pragma unroll
            for (int c = 0; c < C; ++c) {
                pa[c] = column_profile(t_a + c);
                pb[c] = column_profile(t_b + c);
            }
        }

        // ---- row symbols and the left edge, a chunk ahead ----
        auto row_symbol = [&](int i) -> int {
            return (i >= 1 && i <= last_row) ? (int)pv.rowseq[REVERSE ? nrows - i : i - 1] : -1;
        };
        // its code as the steps use it: DNA a selector byte, protein the residue
        auto row_code = [&](int v) -> unsigned {
            if constexpr (AA) return v < 0 ? (unsigned)kAAPad : (unsigned)senc[v & 127];
            return prmt(kSelTableLo, kSelTableHi, v < 0 ? kPadCode : (unsigned)dna_code(v)) & 0xffu;
        };
        int nsym = -1;
        uint64_t nedge = 0;
        bool nneeds = false;
        const uint64_t* nat = nullptr;
        auto issue = [&](int t0) {  // lanes 0 .. kStripRows - 1: rows 2 t0 + 1 + lane
            const int i = 2 * t0 + 1 + lane;
            const bool mine = lane < kStripRows;
            nsym = mine ? row_symbol(i) : -1;
            nneeds = mine && strip > 0 && i <= have;
            nat = e_in + (kEdgeFront - 1 + i);
            if (nneeds) nedge = load_word(nat);
        };
        auto commit = [&](int buf) -> bool {
            const unsigned code = row_code(nsym);
            if (strip > 0 && !wait_words(nneeds, nat, tag - 1, nedge)) return false;
            if (lane < kStripRows) {
                unsigned* at = reinterpret_cast<unsigned*>(&sin_[warp][buf][lane >> 1]);
                at[lane & 1] = nneeds ? (unsigned)nedge : zero_edge;
                reinterpret_cast<unsigned short*>(at + 2)[lane & 1] = (unsigned short)code;
            }
            __syncwarp();
            return true;
        };

        // ---- the zero state every strip starts from ----
        unsigned ho[C], f[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            ho[c] = open2;
            f[c] = 0;
        }
        unsigned diag0 = open2;
        // the left neighbour's words of the next step: what it hands on is shuffled as
        // soon as it is known, before the step's checks and stores
        unsigned x_ho[2] = {open2, open2}, x_e[2] = {0, 0}, x_code;
        {
            const int i = 2 * (t - 1 - lane) + 1;
            x_code = row_code(row_symbol(i)) | (row_code(row_symbol(i - kHalfLag)) << 8) |
                     (row_code(row_symbol(i + 1)) << 16) | (row_code(row_symbol(i + 1 - kHalfLag)) << 24);
            x_code = __shfl_sync(kFull, x_code, src);
        }
        // running max of both halves in the H + open domain (reverse: one below the
        // score, which a half so passes once) and the rows that set it
        unsigned mx = REVERSE ? pack16(pv.target - 1 + open, pv.target - 1 + open) : open2;
        int mi_a = 0, mi_b = 0;
        // Reverse: looks for it in a row, i for the low half.
        auto check_row = [&](int i, const unsigned (&h)[C]) {
            unsigned row = h[0];
#pragma unroll
            for (int c = 1; c < C; ++c) row = __vmaxs2(row, h[c]);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int j = i - kHalfLag * x;
                if ((x ? hi16(row) > hi16(mx) : lo16(row) > lo16(mx)) && (unsigned)(j - 1) < (unsigned)last_row) {
                    (x ? mi_b : mi_a) = j;
                    mx = prmt(mx, row, x ? 0x7610u : 0x3254u);
#pragma unroll
                    for (int k = 0; k < C / 4; ++k)
                        ssave[x][k][threadIdx.x] =
                            make_int4((int)h[4 * k], (int)h[4 * k + 1], (int)h[4 * k + 2], (int)h[4 * k + 3]);
                }
            }
        };
        // Forward: the rows that set it are found once a chunk, from the rows it kept: a
        // half's max last grew in step u of the chunk's (u < 0: not at all).  Rows past
        // the last one may seem to grow it; the chunk that holds the last row looks at
        // its own rows one by one.
        auto settle = [&](int x, int t0, int u, unsigned before) -> int {
            const int r0 = 2 * (t0 - lane) + 1 - kHalfLag * x;  // the half's first row of the chunk
            const int rows = last_row - r0 + 1;
            auto half_max = [&](int k) -> int {
                int m = -32768;
#pragma unroll
                for (int q = 0; q < C / 4; ++q) {
                    const int4 v = srow[k][q][threadIdx.x];
                    const unsigned w = __vmaxs2(__vmaxs2((unsigned)v.x, (unsigned)v.y), __vmaxs2((unsigned)v.z, (unsigned)v.w));
                    m = max(m, x ? hi16(w) : lo16(w));
                }
                return m;
            };
            int k = -1;
            if (rows >= kStripRows) {
                if (u >= 0) k = 2 * u + (half_max(2 * u) == (x ? hi16(mx) : lo16(mx)) ? 0 : 1);
            } else if (rows > 0) {
                int top = x ? hi16(before) : lo16(before);
                for (int j = max(0, 1 - r0); j < rows; ++j) {
                    const int m = half_max(j);
                    if (m > top) {
                        top = m;
                        k = j;
                    }
                }
            }
            if (k < 0) return 0;
#pragma unroll
            for (int q = 0; q < C / 4; ++q) ssave[x][q][threadIdx.x] = srow[k][q][threadIdx.x];
            return r0 + k;
        };

        __syncwarp();
        issue(t);
        bool ok = commit(0);
        int buf = 0;
        while (ok) {
            issue(t + kStripSteps);
            uint4 next = sin_[warp][buf][0];  // loaded a step ahead
            const unsigned before = mx;
            int grew_a = -1, grew_b = -1;
#pragma unroll 2
            for (int u = 0; u < kStripSteps; ++u) {
                const uint4 in = next;
                next = sin_[warp][buf][(u + 1) % kStripSteps];
                const unsigned code = prmt(x_code, in.z, sel_code);
                x_code = __shfl_sync(kFull, code, src);
                const unsigned ho_in[2] = {prmt(x_ho[0], in.x, sel_ho), prmt(x_ho[1], in.y, sel_ho)};
                unsigned e[2] = {prmt(x_e[0], in.x, sel_e), prmt(x_e[1], in.y, sel_e)};
                // DNA: the selectors of both rows, a high half's from bytes 4-7
                const unsigned sel[2] = {code + 0x44004400u, (code + 0x44004400u) >> 16};
                unsigned wa[2][AA ? C / 4 : 1], wb[2][AA ? C / 4 : 1];
                if constexpr (AA) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const unsigned char* at_a = prof + ((code >> (16 * r)) & 0xffu) * kResidue;
                        const unsigned char* at_b = prof + (kAAProfRows + ((code >> (16 * r + 8)) & 0xffu)) * kResidue;
#pragma unroll
                        for (int k = 0; k < C / 4; ++k) {
                            wa[r][k] = *reinterpret_cast<const unsigned*>(at_a + 4 * k);
                            wb[r][k] = *reinterpret_cast<const unsigned*>(at_b + 4 * k);
                        }
                    }
                }
                unsigned diag[2] = {diag0, ho_in[0]}, first[C];  // first: H + open of the first row
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
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) x_e[r] = __shfl_sync(kFull, e[r], src);
                x_ho[0] = __shfl_sync(kFull, first[C - 1], src);
                x_ho[1] = __shfl_sync(kFull, ho[C - 1], src);
                diag0 = ho_in[1];
                // rows 2 (t - 63) + 1 and the next; rows outside the strip fall into the buffer's margins
                if (!last && writes) store_words(e_step, tag, prmt(first[C - 1], e[0], 0x7632u), prmt(ho[C - 1], e[1], 0x7632u));
                e_step += 2;
                unsigned grow = mx;
#pragma unroll
                for (int c = 0; c < C; ++c) grow = __vimax3_s16x2(grow, first[c], ho[c]);
                if constexpr (REVERSE) {
                    // a half reaches the score once, so the branch is rarely taken
                    if (grow != mx) {
                        check_row(2 * (t + u - lane) + 1, first);
                        check_row(2 * (t + u - lane) + 2, ho);
                    }
                    continue;
                }
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
            if (!REVERSE && grew_a >= 0) {
                const int row = settle(0, t, grew_a, before);
                mi_a = row > 0 ? row : mi_a;
            }
            if (!REVERSE && grew_b >= 0) {
                const int row = settle(1, t, grew_b, before);
                mi_b = row > 0 ? row : mi_b;
            }
            t += kStripSteps;
            if (t >= t_end) break;
            ok = commit(buf ^ 1);
            buf ^= 1;
        }
        if (!ok) break;  // a wait ran out: kErrTeam is set, every warp stops

        // ---- the strip's best, joined with that of the strips to its left ----
        uint64_t best = REVERSE ? ~0ull : 0ull;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int mi = x ? mi_b : mi_a;
            if (mi > 0) {
                const int t0 = x ? t_b : t_a;
                // the row's max (the running one may hold a row past the last)
                int want = -32768;
#pragma unroll
                for (int k = 0; k < C / 4; ++k) {
                    const int4 v = ssave[x][k][threadIdx.x];
                    const unsigned w = __vmaxs2(__vmaxs2((unsigned)v.x, (unsigned)v.y), __vmaxs2((unsigned)v.z, (unsigned)v.w));
                    want = max(want, x ? hi16(w) : lo16(w));
                }
                int pick = REVERSE ? C : 0x7fffffff;
#pragma unroll
                for (int k = 0; k < C / 4; ++k) {
                    const int4 v = ssave[x][k][threadIdx.x];
                    const int vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int val = x ? hi16((unsigned)vv[j]) : lo16((unsigned)vv[j]);
                        if (val == want) pick = min(pick, REVERSE ? 4 * k + j : tie_key(t0 + 4 * k + j));
                    }
                }
                const uint64_t cand = REVERSE ? (((uint64_t)(uint32_t)mi << 32) | (uint32_t)(t0 + pick + 1))
                                              : pack_fwd(want - open, mi, pick);
                best = REVERSE ? (cand < best ? cand : best) : (cand > best ? cand : best);
            }
        }
        best = REVERSE ? group_min_u64<32>(best, kFull) : group_max_u64<32>(best, kFull);
        if (strip > 0) {
            const uint64_t* at = e_in + (s.edge_stride - 2) + (lane & 1);
            uint64_t v = load_word(at);
            if (!wait_words(true, at, tag - 1, v)) break;
            const uint64_t left = ((uint64_t)__shfl_sync(kFull, (unsigned)v, 1) << 32) |
                                  __shfl_sync(kFull, (unsigned)v, 0);
            best = REVERSE ? (left < best ? left : best) : (left > best ? left : best);
            if (lane == 0) strip_buffer_read(s, task - 1);
        }
        if (!last) {
            if (lane == 0)
                store_words(e_out + (s.edge_stride - 2), tag, (unsigned)best, (unsigned)(best >> 32));
        } else if (lane == 0) {
            write_result<REVERSE>(p, pid, pv, best);
        }
    }
    end_after_previous(p);
}

// Inclusive scan over the block's 1,024 threads; every thread gets its sum, *total
// the block's.
__device__ __forceinline__ int scan_1024(int v, int* sums, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(kFull, v, off);
        if (lane >= off) v += x;
    }
    __syncthreads();  // an earlier scan's sums are read
    if (lane == 31) sums[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int w = sums[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int x = __shfl_up_sync(kFull, w, off);
            if (lane >= off) w += x;
        }
        sums[lane] = w;
    }
    __syncthreads();
    *total = sums[31];
    return v + (warp > 0 ? sums[warp - 1] : 0);
}

// The tasks of range p.cls: the strips of its pairs, in schedule order.  One
// block: the launches it serves hold few pairs.
template <bool REVERSE>
__global__ void __launch_bounds__(1024) list_strips(PassParams p, StripParams s, int width) {
    __shared__ int sums[32];
    const int begin = p.class_range[2 * p.cls], end = p.class_range[2 * p.cls + 1];
    int total = 0;
    for (int base = begin; base < end; base += 1024) {
        const int k = base + (int)threadIdx.x;
        int pid = 0, strips = 0, all = 0;
        if (k < end) {
            pid = p.order[k];
            strips = max(1, (view_pair<REVERSE>(p, pid).ncols_run + width - 1) / width);
        }
        const int at = total + scan_1024(strips, sums, &all) - strips;
        for (int x = 0; x < strips && at + x < s.max_tasks; ++x)
            s.tasks[at + x] = make_int2(pid, x | (strips << 16));
        total += all;
    }
    if (threadIdx.x == 0) *s.ntasks = total;
    for (int k = (int)threadIdx.x; k < kStripSmSlots; k += 1024) s.on_sm[k] = 0;
}

// The whole schedule of a small batch in one block: a counting sort over four
// groups (binned, raw bytes, int32, idle) x 256 cost levels (eight per doubling) in
// shared memory, then the list of strips.  The large batches' schedule clears and
// scans 36,864 buckets in three kernels: 21 us a pass for 1,000 pairs, this one 8.
template <bool REVERSE>
__global__ void __launch_bounds__(1024) small_schedule(PassParams p, StripParams s, int* order, int* class_range,
                                                       int width) {
    constexpr int kPer = kSmallSchedule / 1024;
    __shared__ int at[1024], sums[32], long_pairs;
    __shared__ int ranked[kSmallSchedule];
    __shared__ unsigned short strips_of[kSmallSchedule];
    const int t = (int)threadIdx.x, n = (int)p.n;
    at[t] = 0;
    if (t == 0) long_pairs = 0;
    for (int k = t; k < kStripSmSlots; k += 1024) s.on_sm[k] = 0;
    __syncthreads();
    int bucket[kPer];
#pragma unroll
    for (int x = 0; x < kPer; ++x) {
        const int k = t + 1024 * x;
        bucket[x] = -1;
        if (k < n) {
            const PairView v = view_pair<REVERSE>(p, k);
            const int cls = p.pair_cls[k];
            int group = is_bin_class(cls) ? 0 : (cls == 1 ? 1 : 2);
            if (REVERSE) group = p.score[k] <= 0 ? 3 : (group == 0 && v.target > p.dual_limit ? 2 : group);
            const int strips = max(1, (v.ncols_run + 255) / 256);
            strips_of[k] = (unsigned short)(width > 0 ? max(1, (v.ncols_run + width - 1) / width) : 0);
            const unsigned cost = (unsigned)strips * (unsigned)(v.nrows / 2 + 64);
            const int e = 31 - __clz(cost);
            bucket[x] = 256 * group + 255 - min(255, 8 * e + (int)((cost >> (e - 3)) & 7));  // cost >= 64
            atomicAdd(&at[bucket[x]], 1);
            if (group == 0 && cls == kClassLong) atomicAdd(&long_pairs, 1);
        }
    }
    __syncthreads();
    int total;
    const int mine = at[t], end = scan_1024(mine, sums, &total);
    at[t] = end - mine;
    __syncthreads();
    if (t == 0) {
        const int raw = at[256], wide = at[512], idle = at[768];
        auto range = [&](int r, int a, int b) {
            class_range[2 * r] = a;
            class_range[2 * r + 1] = b;
        };
        range(kClassBinned, 0, raw);
        range(1, raw, wide);
        range(0, wide, idle);
        range(kClassIdle, idle, n);
        range(kRangeLong, 0, long_pairs);
        range(kRangeShort, long_pairs, raw);
        if (!REVERSE) p.rerun[0] = p.rerun[1] = 0;
    }
    const int binned = at[256];
    __syncthreads();
#pragma unroll
    for (int x = 0; x < kPer; ++x)
        if (bucket[x] >= 0) {
            const int pos = atomicAdd(&at[bucket[x]], 1);
            order[pos] = t + 1024 * x;
            ranked[pos] = t + 1024 * x;
        }
    if (width <= 0) return;
    __syncthreads();
    int tasks = 0;
    for (int base = 0; base < binned; base += 1024) {
        const int k = base + t, pid = k < binned ? ranked[k] : 0, strips = k < binned ? strips_of[pid] : 0;
        const int to = tasks + scan_1024(strips, sums, &total) - strips;
        for (int x = 0; x < strips && to + x < s.max_tasks; ++x) s.tasks[to + x] = make_int2(pid, x | (strips << 16));
        tasks += total;
    }
    if (t == 0) *s.ntasks = tasks;
}

const void* pick_strips(bool reverse, bool aa, int columns, size_t* dyn) {
    *dyn = (reverse ? 0 : strip_row_bytes(columns)) + (aa ? (size_t)2 * kAAProfRows * kThreads * columns : 0);
    if (aa) return reverse ? (const void*)sw_strips<true, true, 4> : (const void*)sw_strips<false, true, 4>;
    if (columns == 8) return reverse ? (const void*)sw_strips<true, false, 8> : (const void*)sw_strips<false, false, 8>;
    return reverse ? (const void*)sw_strips<true, false, 4> : (const void*)sw_strips<false, false, 4>;
}

}  // namespace

cudaError_t strips_occupancy(bool reverse, bool aa, int columns, int* blocks_per_sm) {
    size_t dyn = 0;
    const void* fn = pick_strips(reverse, aa, columns, &dyn);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, kThreads, dyn);
}

cudaError_t launch_small_schedule(bool reverse, const PassParams& p, const StripParams& s, int* order, int* class_range,
                                  int columns, cudaStream_t stream) {
    const int width = columns > 0 ? strip_width(columns) : 0;
    if (reverse)
        small_schedule<true><<<1, 1024, 0, stream>>>(p, s, order, class_range, width);
    else
        small_schedule<false><<<1, 1024, 0, stream>>>(p, s, order, class_range, width);
    return cudaGetLastError();
}

cudaError_t launch_list_strips(bool reverse, int columns, const PassParams& p, const StripParams& s, cudaStream_t stream) {
    if (reverse)
        list_strips<true><<<1, 1024, 0, stream>>>(p, s, strip_width(columns));
    else
        list_strips<false><<<1, 1024, 0, stream>>>(p, s, strip_width(columns));
    return cudaGetLastError();
}

cudaError_t launch_strips(bool reverse, bool aa, int columns, const PassParams& p, const StripParams& s, int blocks,
                          cudaStream_t stream) {
    size_t dyn = 0;
    const void* fn = pick_strips(reverse, aa, columns, &dyn);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    void* args[] = {(void*)&p, (void*)&s};
    return launch_beside(fn, blocks, kThreads, args, dyn, stream, p.join != 0);
}

}  // namespace gbsw
