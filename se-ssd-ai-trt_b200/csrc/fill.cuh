// Device pieces of the resets: ranges of 16-byte words, and the rows of output tensors past a frame's row count.
#pragma once

#include "common.cuh"

namespace sessd {

// Every range of `f` and the status block, spread over the whole grid.
__device__ __forceinline__ void fill_ranges(const FillRanges& f) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t first = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
#pragma unroll
    for (int r = 0; r < FillRanges::kMax; ++r) {
        const uint32_t v = f.ones[r] ? kEmpty : 0u;
        uint4* p = f.ptr[r];
        const size_t n = f.n16[r];
        for (size_t i = first; i < n; i += stride) p[i] = make_uint4(v, v, v, v);
    }
    if (f.status && first >= (size_t)f.status_from && first < (size_t)kStatusInts) f.status[first] = 0;
}

template <typename V>
__device__ __forceinline__ void zero_rows(void* tensor, int units, const TailRows& t) {
    constexpr int PER = 4;                              // stores per thread and item
    const int64_t per_frame = (int64_t)t.max_rows * units;
    const int threads = (int)blockDim.x;
    const int chunks = (int)((per_frame + threads * PER - 1) / (threads * PER));
    V zero;
    memset(&zero, 0, sizeof(V));
    for (int64_t it = blockIdx.x; it < (int64_t)t.batch * chunks; it += gridDim.x) {
        const int b = (int)(it / chunks), c = (int)(it - (int64_t)b * chunks);
        const int most = min(t.most, t.max_rows), n = max(0, min(load_late(t.counts + b), most));
        const int64_t low = (int64_t)n * units, at = (int64_t)c * threads * PER;
        if (at + threads * PER <= low) continue;       // uniform over the block
        V* base = static_cast<V*>(tensor) + (int64_t)b * per_frame;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int64_t i = at + j * threads + threadIdx.x;
            if (i >= low && i < per_frame) base[i] = zero;
        }
    }
}

// The rows of `t`.
__device__ __forceinline__ void zero_tails(const TailRows& t) {
#pragma unroll
    for (int i = 0; i < TailRows::kMax; ++i) {
        if (!t.tensor[i]) continue;
        const int rb = t.row_bytes[i];
        if (rb % 16 == 0) zero_rows<uint4>(t.tensor[i], rb / 16, t);
        else if (rb % 8 == 0) zero_rows<uint2>(t.tensor[i], rb / 8, t);
        else if (rb % 4 == 0) zero_rows<uint32_t>(t.tensor[i], rb / 4, t);
        else zero_rows<uint16_t>(t.tensor[i], rb / 2, t);
    }
}

}  // namespace sessd
