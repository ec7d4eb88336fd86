// Device helpers of the strip-parallel kernels (sw_strips.cu, trace_strips.cu):
// packed halves, the tagged words of a strip's edge and the bounded waits on them.
#pragma once
#include <cstdint>

#include "sw_common.cuh"
#include "sw_strips.h"

namespace gbsw {
namespace {

// Polls of a wait before it gives up (each sleeps about 40 ns, so over a second).
constexpr int kStripSpin = 1 << 25;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned prmt(unsigned a, unsigned b, unsigned sel) {
    unsigned r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ int lo16(unsigned x) { return (int)(short)(x & 0xffffu); }
__device__ __forceinline__ int hi16(unsigned x) { return (int)(short)(x >> 16); }
__device__ __forceinline__ unsigned pack16(int lo, int hi) {
    return (unsigned)(lo & 0xffff) | ((unsigned)hi << 16);
}
__device__ __forceinline__ uint64_t load_word(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_words(uint64_t* p, unsigned tag, unsigned v, unsigned w) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(((uint64_t)tag << 32) | v),
                 "l"(((uint64_t)tag << 32) | w)
                 : "memory");
}

// Polls until every lane of the warp that `needs` a word has it at `at` with
// `tag`; false if the wait ran out (kErrTeam is set) or another one did.
__device__ __forceinline__ bool strip_wait(int* error, bool needs, const uint64_t* at, unsigned tag, uint64_t& v) {
    bool ready = !needs || (unsigned)(v >> 32) == tag;
    for (int it = 0; !__all_sync(kFull, ready); ++it) {
        const bool stop = it == kStripSpin || ((it & 1023) == 1023 && (*(volatile int*)error & kErrTeam));
        if (__any_sync(kFull, stop)) {
            if ((threadIdx.x & 31) == 0) atomicOr(error, kErrTeam);
            return false;
        }
        __nanosleep(40);
        if (!ready) {
            v = load_word(at);
            ready = (unsigned)(v >> 32) == tag;
        }
    }
    return true;
}

// Waits until the reader of the edge buffer's previous task is done with it (the
// task `ring` before this one, if it had a reader); false as above.
__device__ __forceinline__ bool strip_buffer_free(int* error, const StripParams& s, int task) {
    if (task < s.ring) return true;
    const int before = s.tasks[task - s.ring].y;
    if ((before & 0xffff) + 1 >= (int)((unsigned)before >> 16)) return true;  // a last strip: no reader
    const unsigned* f = s.freed + (task - s.ring);
    const unsigned want = s.tag_base + (unsigned)(task - s.ring);
    bool ok = false;
    for (int it = 0; it < kStripSpin && !ok; ++it) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
        ok = v == want;
        if (!ok && (it & 1023) == 1023 && (*(volatile int*)error & kErrTeam)) break;
        if (!ok) __nanosleep(40);
    }
    if (__all_sync(kFull, ok)) return true;
    if ((threadIdx.x & 31) == 0) atomicOr(error, kErrTeam);
    return false;
}

// Marks task `task`'s edge buffer as read; one thread of the reader.
__device__ __forceinline__ void strip_buffer_read(const StripParams& s, int task) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(s.freed + task), "r"(s.tag_base + (unsigned)task)
                 : "memory");
}

// The first of a block's tasks (one per warp), or `ntasks` if the block is to
// leave; one thread.  Warps that share a scheduler slow the chain of the longest
// pair, so few tasks keep one or two blocks to an SM (measured by tasks per
// scheduler: 500 proteins, 1.2 of them, forward 178 us at one block, 225 at two,
// 262 at four; 1,000 mixed DNA pairs, 5 of them, 893, 762, 752 at three).
__device__ __forceinline__ int strip_first_task(const StripParams& s, int* queue, int ntasks) {
    const int warps = (int)blockDim.x / 32, schedulers = s.sms * 4;
    const int per_sm = ntasks <= 2 * schedulers ? 1 : (ntasks <= 4 * schedulers ? 2 : 64);
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    return atomicAdd(s.on_sm + sm % kStripSmSlots, 1) < per_sm ? atomicAdd(queue, warps) : ntasks;
}

}  // namespace
}  // namespace gbsw
