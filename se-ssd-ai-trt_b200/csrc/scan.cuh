// Numbering in one pass: exclusive prefix sums over the chunks of a frame, handed from chunk to chunk through global
// memory while the kernel runs (no counting pass, no second read of the input).
//
// A block takes chunks from a ticket counter, so every chunk before its own belongs to a block that is already running.
// It publishes its chunk's total, adds up the totals published before it - a warp looks at 32 chunks at a time and stops
// at the first one whose running total is known - and publishes its own running total. Tickets go through the frames
// of a batch side by side (chunk-major), so that a chunk's predecessors are usually finished when it starts. The wait for
// a predecessor is bounded by a clock limit, after which the call reports SESSD_STATUS_TIMEOUT.
#pragma once

#include "common.cuh"

namespace sessd {

constexpr unsigned long long kScanTotal = 1ull << 32, kScanPrefix = 2ull << 32;   // state words: flag | value

__device__ __forceinline__ void scan_publish(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long scan_peek(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Sum of the totals of chunks 0 .. c - 1 of the frame whose state words start at `state`; `total` is chunk c's own.
// Called by one whole warp; the words must be zero before the kernel.
__device__ __forceinline__ int scan_prefix(unsigned long long* state, int c, int total, int32_t* status) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) scan_publish(state + c, (c == 0 ? kScanPrefix : kScanTotal) | (unsigned)total);
    int prefix = 0;
    bool complete = c == 0;
    for (int base = c - 1; !complete; base -= 32) {
        const int i = base - lane;
        const long long t0 = clock64();
        unsigned long long v = i >= 0 ? scan_peek(state + i) : kScanPrefix;   // before chunk 0: a running total of 0
        int last;
        for (;;) {
            const uint32_t have_prefix = __ballot_sync(0xFFFFFFFFu, v >= kScanPrefix);
            const uint32_t have_any = __ballot_sync(0xFFFFFFFFu, v >= kScanTotal);
            last = have_prefix ? __ffs((int)have_prefix) - 1 : 31;
            const uint32_t needed = last == 31 ? 0xFFFFFFFFu : (2u << last) - 1u;
            if ((have_any & needed) == needed) {
                complete = have_prefix != 0u;
                break;
            }
            if (__any_sync(0xFFFFFFFFu, clock64() - t0 > 100000000LL)) {   // some 50 ms; real waits are microseconds
                if (lane == 0) atomicOr(status, SESSD_STATUS_TIMEOUT);
                complete = true;
                break;
            }
            if (v < kScanTotal) v = scan_peek(state + i);
        }
        prefix += __reduce_add_sync(0xFFFFFFFFu, lane <= last ? (int)(unsigned)v : 0);
    }
    if (lane == 0 && c > 0) scan_publish(state + c, kScanPrefix | (unsigned)(prefix + total));
    return prefix;
}

// Exclusive position of the calling thread's `count` things among those of all chunks before and of its own block
// (kThreads threads); *chunk_end gets the running total including the chunk. The whole block calls it.
__device__ __forceinline__ int scan_position(unsigned long long* state, int c, int count, int* chunk_end, int32_t* status) {
    __shared__ int s_prefix;
    int total;
    const int before = block_exclusive_scan(count, &total);
    if (threadIdx.x < 32) {
        const int p = scan_prefix(state, c, total, status);
        if (threadIdx.x == 0) s_prefix = p;
    }
    __syncthreads();
    const int prefix = s_prefix;
    *chunk_end = prefix + total;
    return prefix + before;
}

// Next ticket of the block, -1 when all `items` are taken.
__device__ __forceinline__ int scan_ticket(uint32_t* counter, int items) {
    __shared__ int s_ticket;
    __syncthreads();                 // the previous ticket and prefix have been read
    if (threadIdx.x == 0) s_ticket = (int)atomicAdd(counter, 1u);
    __syncthreads();
    return s_ticket < items ? s_ticket : -1;
}

}  // namespace sessd
