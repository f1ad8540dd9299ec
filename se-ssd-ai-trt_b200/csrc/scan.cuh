// Numbering in one pass: exclusive prefix sums over the chunks of a frame, handed from chunk to chunk through global
// memory while the kernel runs (no counting pass, no second read of the input).
//
// A block publishes its chunk's total and adds up the totals of all chunks before it: every thread polls up to four of
// them, so that the sum is one round trip once the slowest has published (a chain of running totals, 32 chunks a step,
// took 10 us for the levels of a single frame). Chunks come in groups of 1024; the last chunk of a group publishes the
// running total instead, which the next groups start from. Blocks take their chunks from a ticket counter, so that a chunk's
// predecessors belong to blocks that are already running, whatever order the blocks start in and however many are
// resident. The wait for a predecessor is bounded by a clock limit, after which the call reports SESSD_STATUS_TIMEOUT.
#pragma once

#include "common.cuh"

namespace sessd {

constexpr int kScanGroup = 4 * kThreads;
constexpr unsigned long long kScanReady = 1ull << 32;   // state words: flag | total (or running total)

__device__ __forceinline__ void scan_publish(unsigned long long* p, int v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(kScanReady | (unsigned)v) : "memory");
}
__device__ __forceinline__ unsigned long long scan_peek(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int scan_await(const unsigned long long* p, unsigned long long v, int32_t* status) {
    if (v < kScanReady) {
        const long long t0 = clock64();
        while ((v = scan_peek(p)) < kScanReady)
            if (clock64() - t0 > 100000000LL) {   // some 50 ms; real waits are microseconds
                atomicOr(status, SESSD_STATUS_TIMEOUT);
                break;
            }
    }
    return (int)(unsigned)v;
}

// Sum of the totals of the chunks before chunk c of the frame whose state words start at `state` (zero before the kernel);
// `total` is chunk c's own. The whole block (kThreads threads) calls it.
__device__ __forceinline__ int scan_prefix(unsigned long long* state, int c, int total, int32_t* status) {
    const bool closes_group = c % kScanGroup == kScanGroup - 1;
    if (threadIdx.x == 0 && !closes_group) scan_publish(state + c, total);
    int prefix = 0;
    if (c > 0) {
        const int g0 = c / kScanGroup * kScanGroup;
        unsigned long long v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = g0 + i * kThreads + threadIdx.x;
            v[i] = j < c ? scan_peek(state + j) : kScanReady;
        }
        int sum = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = g0 + i * kThreads + threadIdx.x;
            if (j < c) sum += scan_await(state + j, v[i], status);
        }
        if (threadIdx.x == 0 && g0 > 0) sum += scan_await(state + g0 - 1, 0ull, status);
        prefix = block_sum(sum);
    }
    if (threadIdx.x == 0 && closes_group) scan_publish(state + c, prefix + total);
    return prefix;
}

// Exclusive position of the calling thread's `count` things among those of all chunks before chunk c and of its own block;
// *chunk_end gets the running total including the chunk.
__device__ __forceinline__ int scan_position(unsigned long long* state, int c, int count, int* chunk_end, int32_t* status) {
    int total;
    const int before = block_exclusive_scan(count, &total);
    const int prefix = scan_prefix(state, c, total, status);
    *chunk_end = prefix + total;
    return prefix + before;
}

// The chunks of a block, out of `items` over all `blocks` blocks that number: for (int t = scan_first(..); t >= 0; t =
// scan_next(..)). The first ticket may be taken before pdl_wait() where the counter is older than the preceding kernel: the
// trip to the counter is then over by the time that kernel is.
__device__ __forceinline__ int scan_ticket(uint32_t* counter, int items) {
    __shared__ int s_ticket;
    __syncthreads();                 // the previous ticket has been read
    if (threadIdx.x == 0) s_ticket = (int)atomicAdd(counter, 1u);
    __syncthreads();
    return s_ticket < items ? s_ticket : -1;
}
__device__ __forceinline__ int scan_first(uint32_t* counter, int items) { return scan_ticket(counter, items); }
__device__ __forceinline__ int scan_next(uint32_t* counter, int items, int blocks) {
    return items <= blocks ? -1 : scan_ticket(counter, items);
}

}  // namespace sessd
