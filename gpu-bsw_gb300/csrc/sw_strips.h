// Strip-parallel int16x2 passes (sw_strips.cu): host interface.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "sw_common.cuh"

namespace gbsw {

// Counters of blocks per SM (SM ids wrap around them).
constexpr int kStripSmSlots = 512;

// Work and buffers of a strip-parallel launch.
struct StripParams {
    int2* tasks;           // x: pair, y: strip | strips of the pair << 16; a pair's strips follow one another
    int* ntasks;           // tasks in the list
    int* on_sm;            // kStripSmSlots counters: blocks started, by SM
    int max_tasks;         // room of the list
    unsigned* freed;       // per task: its tag once its edge buffer has been read
    uint64_t* edges;       // edge buffers, edge_stride entries each: (tag << 32) | (E << 16) | (H + open) by row,
                           // and in the last two entries the halves of the best so far
    int edge_stride;
    int ring;              // edge buffers (>= 2): task k uses k % ring
    int sms;               // multiprocessors of the device
    unsigned tag_base;     // task k's tag is tag_base + k; no other task has it until the buffers are cleared
};

// Entries of an edge buffer for sequences of up to `rows` symbols: the rows, 128
// before them and 16 after (the pipeline's fill and the rest of the last chunk: up
// to 7 steps of two rows past the step of the last row, 15 with an odd last row),
// and the two words of the best.
inline int strip_edge_stride(int rows) { return (rows + 128 + 16 + 2 + 1) & ~1; }
// Columns of a strip with `columns` (4 or 8) columns a lane.
__host__ __device__ constexpr int strip_width(int columns) { return 64 * columns; }
// Columns a lane holds: 8 where there is a kernel for them and `wide` is asked for.
inline int strip_columns(bool aa, bool wide) { return wide && !aa ? 8 : 4; }

// Most pairs of the one-block schedule below.
constexpr int kSmallSchedule = 4096;
// Orders up to kSmallSchedule pairs whose binned ones all run strip by strip: their
// classes (p.pair_cls; reverse: those above p.dual_limit take class 0), each by
// descending cost, into p.order and p.class_range (writable copies of the
// pointers), lists the strips of the binned ones (`columns` a lane; 0: none) and
// clears the rerun count.
cudaError_t launch_small_schedule(bool reverse, const PassParams& p, const StripParams& s, int* order, int* class_range,
                                  int columns, cudaStream_t stream);
cudaError_t strips_occupancy(bool reverse, bool aa, int columns, int* blocks_per_sm);
// Lists the strips of range p.cls of the schedule, and runs the listed ones.
cudaError_t launch_list_strips(bool reverse, int columns, const PassParams& p, const StripParams& s, cudaStream_t stream);
cudaError_t launch_strips(bool reverse, bool aa, int columns, const PassParams& p, const StripParams& s, int blocks,
                          cudaStream_t stream);

}  // namespace gbsw
