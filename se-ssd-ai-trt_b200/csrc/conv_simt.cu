// Output-stationary sparse convolution on CUDA cores (fp32 and fp16 storage, fp32 accumulate).
//
// Replaces the reference's per-offset gather / multiply / atomicAdd kernel, launched kvol times per
// layer with one thread per rulebook pair and Cout global atomics per pair
// (submConv3dlayer.cu:479-518, :632-638). Here one launch covers the layer: a thread owns two, four or eight
// output channels of one output row, walks the row's present neighbours, and for each of them
// accumulates s = sum_ci in[ci]*W[k][ci][co] as one fused-multiply-add chain (ci ascending),
// then acc += s with k ascending. That is the arithmetic of the reference kernel with the order of
// the atomic additions fixed, so fp32 results are reproducible bit for bit. BatchNorm scale/shift and
// ReLU (a separate TensorRT scale + activation layer in the reference, se-ssd-ai-trt.cpp:808-856)
// run in the epilogue, and the last layer can scatter straight into the dense BEV map.
//
// This path serves the memory-bound small-channel layers (4->16; in fp32 also 16->16 and 16->32) in calls of few rows (larger ones,
// but for 16->32, are in conv_rows.cu) and, with a kernel that takes its channel counts at run time, every pair of channel counts
// without a kernel of its own. The wide fp32 layers are in conv_f32.cu, the wide fp16 layers in conv_umma.cu.
#include <string>
#include <type_traits>

#include "common.cuh"

namespace sessd {

namespace {

template <typename T, int N>
struct RowLoader;

template <int N>
struct RowLoader<float, N> {
    static __device__ __forceinline__ void load(const float* __restrict__ p, float (&x)[N]) {
        static_assert(N % 4 == 0, "row length must be a multiple of 4");
        const float4* v = reinterpret_cast<const float4*>(p);
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            const float4 t = __ldg(v + i);
            x[4 * i + 0] = t.x; x[4 * i + 1] = t.y; x[4 * i + 2] = t.z; x[4 * i + 3] = t.w;
        }
    }
};

template <int N>
struct RowLoader<__half, N> {
    static __device__ __forceinline__ void load(const __half* __restrict__ p, float (&x)[N]) {
        static_assert(N % 4 == 0, "row length must be a multiple of 4");
        if constexpr (N % 8 == 0) {
            const uint4* v = reinterpret_cast<const uint4*>(p);
#pragma unroll
            for (int i = 0; i < N / 8; ++i) {
                const uint4 t = __ldg(v + i);
                const __half2* h = reinterpret_cast<const __half2*>(&t);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __half22float2(h[j]);
                    x[8 * i + 2 * j] = f.x; x[8 * i + 2 * j + 1] = f.y;
                }
            }
        } else {
            const uint2* v = reinterpret_cast<const uint2*>(p);
#pragma unroll
            for (int i = 0; i < N / 4; ++i) {
                const uint2 t = __ldg(v + i);
                const __half2* h = reinterpret_cast<const __half2*>(&t);
                const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
                x[4 * i] = a.x; x[4 * i + 1] = a.y; x[4 * i + 2] = b.x; x[4 * i + 3] = b.y;
            }
        }
    }
};

template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }

__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__half v) { return __half2float(v); }

template <int N>
__device__ __forceinline__ void store_channels(float* p, const float (&y)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) *reinterpret_cast<float2*>(p + i) = make_float2(y[i], y[i + 1]);
    }
}
template <int N>
__device__ __forceinline__ void store_channels(__half* p, const float (&y)[N]) {
    __align__(16) __half2 h[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) h[i] = __floats2half2_rn(y[2 * i], y[2 * i + 1]);
    if constexpr (N % 8 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 8) *reinterpret_cast<uint4*>(p + i) = *reinterpret_cast<const uint4*>(h + i / 2);
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 4) *reinterpret_cast<uint2*>(p + i) = *reinterpret_cast<const uint2*>(h + i / 2);
    }
}

// N weights from shared memory.
template <int N>
__device__ __forceinline__ void load_weights(const float* p, float (&w)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int c = 0; c < N; c += 4) {
            const float4 t = *reinterpret_cast<const float4*>(p + c);
            w[c] = t.x, w[c + 1] = t.y, w[c + 2] = t.z, w[c + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int c = 0; c < N; c += 2) {
            const float2 t = *reinterpret_cast<const float2*>(p + c);
            w[c] = t.x, w[c + 1] = t.y;
        }
    }
}
template <int N>
__device__ __forceinline__ void load_weights(const __half* p, float (&w)[N]) {
    using V = typename std::conditional<N % 8 == 0, uint4, uint2>::type;
    constexpr int E = sizeof(V) / 2;                     // halves per read
#pragma unroll
    for (int c = 0; c < N; c += E) {
        const V t = *reinterpret_cast<const V*>(p + c);
        const __half2* h = reinterpret_cast<const __half2*>(&t);
#pragma unroll
        for (int j = 0; j < E / 2; ++j) {
            const float2 f = __half22float2(h[j]);
            w[c + 2 * j] = f.x, w[c + 2 * j + 1] = f.y;
        }
    }
}

// Narrow layers. Little arithmetic per row (4 to 5 of 27 neighbours at full resolution) behind three dependent reads
// (row count, map entry, input row), so the kernel lives on rows in flight: COUT / OC threads share a row, a block takes
// ROWS rows at a time and reads their map entries side by side (coalesced over rows, all in flight, those of its next
// rows while it works on the present ones); every thread then walks its row's present neighbours in ascending k. The
// weights sit in shared memory as they come (a warp's rows are at different offsets, so that their reads are what the
// multiply-adds wait for: as halves instead of floats a frame of 20,000 points took 257 instead of 262 us), 16 bytes of
// padding per offset so that rows at different offsets meet in fewer banks. How many channels a thread has is the
// dispatch's choice.
template <typename T, int CIN, int COUT, int OC_>
struct Narrow {
    static constexpr int OC = OC_;                       // output channels per thread
    static constexpr int TPR = COUT / OC;                // threads per output row
    static constexpr int ROWS = kThreads / TPR;          // a divisor of the map's 128-row tile
    // Resident per SM (registers, weights). A small frame's chunks should all be resident: 545 of them as three blocks per SM made a
    // second round for a quarter (16->16, 20,000 points: 33.6 us a call, with four 30.6; 4 x 120,000 points 321 and 307).
    static constexpr int BLOCKS = CIN <= 4 || (OC <= 2 && COUT <= 16) ? 4 : 3;
    static constexpr int KVOL_MAX = 27;                  // 3 x 3 x 3 is the largest kernel the geometry code accepts
    static constexpr int W_STRIDE = CIN * COUT + 16 / (int)sizeof(T);   // elements from one offset's weights to the next offset's
    static constexpr int smem(int kvol) { return kvol * W_STRIDE * (int)sizeof(T) + KVOL_MAX * ROWS * 4; }
};

template <typename T, int CIN, int COUT, int OC_>
__global__ void __launch_bounds__(kThreads, (Narrow<T, CIN, COUT, OC_>::BLOCKS))
conv_narrow_kernel(const T* __restrict__ in, T* __restrict__ out, const int32_t* __restrict__ nbr,
                   const uint32_t* __restrict__ tile_mask, const int32_t* __restrict__ order,
                   const int32_t* __restrict__ out_num, const T* __restrict__ weights, const float* __restrict__ scale,
                   const float* __restrict__ shift, int relu, int batch, int max_voxels, int kvol,
                   T* __restrict__ dense, const int4* __restrict__ out_coors, int D, int H, int W) {
    using N = Narrow<T, CIN, COUT, OC_>;
    constexpr int TPR = N::TPR, ROWS = N::ROWS, OC = N::OC;
    constexpr int LOADS = (N::KVOL_MAX * ROWS + kThreads - 1) / kThreads;   // map entries a thread reads
    constexpr int NP = 2;                                                   // input rows in flight per thread
    extern __shared__ __align__(16) uint8_t narrow_smem[];
    T* s_w = reinterpret_cast<T*>(narrow_smem);
    int32_t* s_idx = reinterpret_cast<int32_t*>(s_w + kvol * N::W_STRIDE);           // [KVOL_MAX][ROWS]
    const int tid = threadIdx.x, r = tid / TPR, cq = tid % TPR;
    const int chunks = (max_voxels + ROWS - 1) / ROWS;
    const int items = batch * chunks, tiles = (max_voxels + 127) / 128;
    // the block's next rows: frame, first row, row count of the frame; entry[j] = the map entries this thread reads for
    // them, entry e = (offset e / ROWS, row e % ROWS)
    int next = blockIdx.x, b_next = 0, o_next = 0, n_next = 0, row_next = 0;
    int entry[LOADS];
    auto fetch = [&]() {
        for (; next < items; next += gridDim.x) {
            b_next = next / chunks;
            o_next = (next - b_next * chunks) * ROWS;
            n_next = load_late(out_num + b_next);
            n_next = n_next > max_voxels ? max_voxels : n_next;
            if (o_next < n_next) break;
        }
        if (next >= items) return;
        const uint32_t mask = __ldg(tile_mask + (size_t)b_next * tiles + (o_next >> 7));
        row_next = order && o_next + r < n_next ? __ldg(order + (size_t)b_next * max_voxels + o_next + r) : o_next + r;
        const int32_t* nb = nbr + nbr_index(kvol, max_voxels, b_next, 0, o_next);   // ROWS rows of one 128-row tile
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int e = tid + j * kThreads, k = e / ROWS, row = e % ROWS;
            entry[j] = k < kvol && ((mask >> k) & 1u) && o_next + row < n_next ? __ldg(nb + k * kNbrRun + row) : -1;
        }
    };
    // the weights are older than any preceding kernel
    for (int e = tid; e < kvol * CIN * COUT; e += kThreads) {
        const int k = e / (CIN * COUT);
        s_w[k * N::W_STRIDE + (e - k * (CIN * COUT))] = __ldg(weights + e);
    }
    pdl_enter();
    fetch();
    while (next < items) {
        const int b = b_next, o = row_next;
        const bool live = o_next + r < n_next;
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int e = tid + j * kThreads;
            if (e < N::KVOL_MAX * ROWS) s_idx[e] = entry[j];
        }
        __syncthreads();
        next += gridDim.x;
        fetch();
        // the row's present offsets, its threads looking at every TPR-th slot
        uint32_t present = 0;
#pragma unroll
        for (int k0 = 0; k0 < N::KVOL_MAX; k0 += TPR) {
            const int k = k0 + cq;
            if (k < N::KVOL_MAX && s_idx[k * ROWS + r] >= 0) present |= 1u << k;
        }
#pragma unroll
        for (int d = 1; d < TPR; d <<= 1) present |= __shfl_xor_sync(0xFFFFFFFFu, present, d);
        float acc[OC];
#pragma unroll
        for (int c = 0; c < OC; ++c) acc[c] = 0.f;
        const T* in_b = in + (size_t)b * max_voxels * CIN;
        while (present) {
            int ks[NP];
            float x[NP][CIN];
#pragma unroll
            for (int u = 0; u < NP; ++u) {
                ks[u] = present ? __ffs((int)present) - 1 : -1;
                present &= present - 1u;          // no-op when nothing is left
                if (ks[u] >= 0) RowLoader<T, CIN>::load(in_b + (size_t)s_idx[ks[u] * ROWS + r] * CIN, x[u]);
            }
#pragma unroll
            for (int u = 0; u < NP; ++u) {
                if (ks[u] < 0) continue;
                // one neighbour: sum_ci x[ci] * W[k][ci][:] as a fused chain, then added to the row's sum
                float s[OC];
#pragma unroll
                for (int c = 0; c < OC; ++c) s[c] = 0.f;
                const T* wk = s_w + ks[u] * N::W_STRIDE + cq * OC;
#pragma unroll
                for (int ci = 0; ci < CIN; ++ci) {
                    float w[OC];
                    load_weights(wk + ci * COUT, w);
#pragma unroll
                    for (int c = 0; c < OC; ++c) s[c] = fmaf(x[u][ci], w[c], s[c]);
                }
#pragma unroll
                for (int c = 0; c < OC; ++c) acc[c] = __fadd_rn(acc[c], s[c]);
            }
        }
        if (live) {
#pragma unroll
            for (int c = 0; c < OC; ++c) {
                float v = acc[c];
                if (scale) v = fmaf(v, __ldg(scale + cq * OC + c), shift ? __ldg(shift + cq * OC + c) : 0.f);
                if (relu) v = v > 0.f ? v : 0.f;
                acc[c] = v;
            }
            store_channels(out + ((size_t)b * max_voxels + o) * COUT + cq * OC, acc);
            if (dense) {
                // Fused BEV scatter (sparse2Dense.cu:201-206): channel c*D + z, pixel (y, x).
                const int4 c4 = __ldg(&out_coors[(size_t)b * max_voxels + o]);
                T* d = dense + (size_t)b * COUT * D * H * W + ((size_t)c4.y * H + c4.z) * W + c4.w;
#pragma unroll
                for (int c = 0; c < OC; ++c) d[(size_t)(cq * OC + c) * D * H * W] = from_float<T>(acc[c]);
            }
        }
        __syncthreads();     // the rows' entries have been used
    }
}

// Any channel counts (the reference's kernel takes in_channel and out_channel as run-time values,
// submConv3dlayer.cu:479-518): one warp per output row, lane = output channel (in rounds of 32), the same order of
// additions as above - per neighbour a fused chain over ci, neighbours added in ascending k. The pairs of the
// network's schedule never come here; this keeps the plugin entry points usable for other layer shapes.
template <typename T>
__global__ void __launch_bounds__(kThreads)
conv_generic_kernel(const T* __restrict__ in, T* __restrict__ out, const int32_t* __restrict__ nbr,
                    const uint32_t* __restrict__ tile_mask, const int32_t* __restrict__ order,
                    const int32_t* __restrict__ out_num, const T* __restrict__ weights, const float* __restrict__ scale,
                    const float* __restrict__ shift, int relu, int batch, int max_voxels, int kvol, int cin, int cout,
                    T* __restrict__ dense, const int4* __restrict__ out_coors, int D, int H, int W) {
    pdl_enter();
    constexpr int ROWS = kThreads / 32;
    const int lane = threadIdx.x & 31, wrow = threadIdx.x >> 5;
    const int chunks = (max_voxels + ROWS - 1) / ROWS;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int p = (it - b * chunks) * ROWS + wrow;
        int n = load_late(out_num + b);
        n = n > max_voxels ? max_voxels : n;
        if (p >= n) continue;
        const int32_t* nb = nbr + nbr_index(kvol, max_voxels, b, 0, p);
        const uint32_t mask = __ldg(tile_mask + (size_t)b * ((max_voxels + 127) / 128) + (p >> 7));
        const int o = order ? __ldg(order + (size_t)b * max_voxels + p) : p;
        const T* in_b = in + (size_t)b * max_voxels * cin;
        T* d = nullptr;
        if (dense) {
            const int4 c4 = __ldg(&out_coors[(size_t)b * max_voxels + o]);
            d = dense + (size_t)b * cout * D * H * W + ((size_t)c4.y * H + c4.z) * W + c4.w;
        }
        for (int co = lane; co < cout; co += 32) {
            float acc = 0.f;
            for (int k = 0; k < kvol; ++k) {
                // the entry is read whether the mask has the offset or not, so that reads run ahead of the loop (behind the mask:
                // 4 x 120,000 points, 8 -> 24 channels 670 us instead of 640); what it holds counts only where the mask has it
                const int entry = __ldg(nb + k * kNbrRun), idx = (mask >> k) & 1u ? entry : -1;
                if (idx < 0) continue;
                const T* x = in_b + (size_t)idx * cin;
                const T* wk = weights + (size_t)k * cin * cout + co;
                float sum = 0.f;
                for (int ci = 0; ci < cin; ++ci) sum = fmaf(to_float(x[ci]), to_float(wk[(size_t)ci * cout]), sum);
                acc = __fadd_rn(acc, sum);
            }
            if (scale) acc = fmaf(acc, __ldg(scale + co), shift ? __ldg(shift + co) : 0.f);
            if (relu) acc = acc > 0.f ? acc : 0.f;
            const T v = from_float<T>(acc);
            out[((size_t)b * max_voxels + o) * cout + co] = v;
            if (d) d[(size_t)co * D * H * W] = v;
        }
    }
}

template <typename T>
int launch_generic(const ConvLaunch& c, cudaStream_t stream) {
    SESSD_LAUNCH_NAMED(sizeof(T) == 4 ? "conv_generic<f32>" : "conv_generic<f16>", conv_generic_kernel<T>,
                       persistent_grid(8), kThreads, 0, stream, static_cast<const T*>(c.in), static_cast<T*>(c.out), c.nbr, c.tile_mask, c.order,
                       c.out_num, static_cast<const T*>(c.weights), c.scale, c.shift, c.relu, c.batch, c.max_voxels,
                       c.kvol, c.cin, c.cout, static_cast<T*>(c.dense), reinterpret_cast<const int4*>(c.out_coors), c.D,
                       c.H, c.W);
    return SESSD_OK;
}

template <typename T, int CIN, int COUT, int OC>
int launch_narrow(const ConvLaunch& c, cudaStream_t stream) {
    using N = Narrow<T, CIN, COUT, OC>;
    static const std::string name = std::string("conv_narrow<") + (sizeof(T) == 4 ? "f32," : "f16,") +
                                    std::to_string(CIN) + "," + std::to_string(COUT) + ">";
    if (N::smem(N::KVOL_MAX) > 48 * 1024) {
        // the attribute belongs to the device's context: set it once per device (repeating it is harmless)
        static std::atomic<uint64_t> configured{0};
        int dev = 0;
        SESSD_CUDA(cudaGetDevice(&dev));
        const uint64_t bit = 1ull << (dev & 63);
        if (!(configured.load(std::memory_order_acquire) & bit)) {
            SESSD_CUDA(cudaFuncSetAttribute(conv_narrow_kernel<T, CIN, COUT, OC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            N::smem(N::KVOL_MAX)));
            configured.fetch_or(bit, std::memory_order_release);
        }
    }
    SESSD_LAUNCH_NAMED(name.c_str(), (conv_narrow_kernel<T, CIN, COUT, OC>), persistent_grid(N::BLOCKS), kThreads, N::smem(c.kvol),
                       stream, static_cast<const T*>(c.in), static_cast<T*>(c.out), c.nbr, c.tile_mask,
                       c.order, c.out_num,
                       static_cast<const T*>(c.weights), c.scale, c.shift, c.relu, c.batch, c.max_voxels, c.kvol,
                       static_cast<T*>(c.dense), reinterpret_cast<const int4*>(c.out_coors), c.D, c.H, c.W);
    return SESSD_OK;
}

template <typename T>
int dispatch(const ConvLaunch& c, cudaStream_t stream) {
    // Half the channels per thread (a thread is through its row's neighbours sooner, and twice as many blocks share out the rows with
    // the longest lists) is the faster way for small calls: front end of 1 x 20,000 points, fp16 254 us and 258 with all of them, fp32
    // 992 and 1000. With all the channels half as many threads walk a list, which pays from a million rows on. 4 -> 16 in us, half and
    // all: 32 x 20,000 points 125 and 113, 16 x 120,000 320 and 282, fp32 111 and 93, 275 and 230 (calls of that size are conv_rows.cu's
    // where all weights are finite numbers). fp32 16 -> 16 is faster with half at any size (16 x 120,000 779 and 846). fp32 16 -> 32 stays
    // here at every size: a submanifold layer (the network has none of these) gains from between 4 and 8 x 20,000 points (4 x 120,000:
    // 523 and 460), the network's strided one from a million rows on (8 x 120,000 18097 and 18062, the whole front end).
    const bool few = (int64_t)c.batch * c.max_voxels <= 1000000;
    if (c.cin == 4 && c.cout == 16) {
        // (eight halves leave in 16 bytes; rows that start at other multiples of eight are taken, too, where all of them are in use)
        const bool wide = !few && reinterpret_cast<uintptr_t>(c.out) % 16 == 0;
        return wide ? launch_narrow<T, 4, 16, 8>(c, stream) : launch_narrow<T, 4, 16, 4>(c, stream);
    }
    if (sizeof(T) == 4) {   // in fp16 the tensor-core kernel takes these
        if (c.cin == 16 && c.cout == 16) return launch_narrow<float, 16, 16, 2>(c, stream);
        if (c.cin == 16 && c.cout == 32) return few ? launch_narrow<float, 16, 32, 2>(c, stream) : launch_narrow<float, 16, 32, 4>(c, stream);
    }
    return launch_generic<T>(c, stream);   // any other pair of channel counts
}

}  // namespace

bool conv_simt_supported(int cin, int cout) { return cin >= 1 && cout >= 1 && cin <= 4096 && cout <= 4096; }

int launch_conv_simt(const ConvLaunch& c, cudaStream_t stream) {
    return c.dtype == SESSD_F32 ? dispatch<float>(c, stream) : dispatch<__half>(c, stream);
}

}  // namespace sessd
