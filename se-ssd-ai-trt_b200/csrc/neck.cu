// What lies between the dense convolutions of the 2D neck and head (the layer graph of se-ssd-ai-trt.cpp:1262-1440): layout,
// bias, ReLU, residual sum, the attention that fuses the two branches, and the 1x1 heads. The 3x3 convolutions themselves are
// library calls. Activations are fp16, channels last.
//
// All of it is memory traffic on maps of a few megabytes that stay in L2, so what counts is the number of passes and
// launches: as separate tensor operations (a strided copy, a broadcast addition and a ReLU after each of thirteen
// convolutions, fourteen more for the attention and the heads) they took 245 of the 350 us of neck and head on a single
// 128 x 200 x 176 map.
#include "common.cuh"

namespace sessd {

namespace {

constexpr int kTilePixels = 64;

__device__ __forceinline__ void unpack8(const uint4& v, float (&x)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        x[2 * i] = f.x, x[2 * i + 1] = f.y;
    }
}

__device__ __forceinline__ float round_half(float x) { return __half2float(__float2half_rn(x)); }

// [B][C][pixels] -> [B][pixels][C], 64 pixels x 64 channels at a time. Reads and writes are runs of 128 bytes; rows of 66
// halves in shared memory, so that neither the 2-byte writes (a warp: 32 pixels of a channel) nor the 4-byte reads (eight
// lanes per pixel) meet in a bank.
__global__ void __launch_bounds__(kThreads)
channels_last_kernel(const __half* __restrict__ in, __half* __restrict__ out, int batch, int channels, int pixels) {
    pdl_enter();
    constexpr int STRIDE = 66;
    __shared__ __half s[kTilePixels * STRIDE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p_tiles = (pixels + kTilePixels - 1) / kTilePixels, c_tiles = (channels + 63) / 64;
    for (int it = blockIdx.x; it < batch * p_tiles * c_tiles; it += gridDim.x) {
        const int c0 = it % c_tiles * 64, p0 = it / c_tiles % p_tiles * kTilePixels, b = it / (c_tiles * p_tiles);
        const __half* src = in + (size_t)b * channels * pixels;
        __half v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int c = c0 + warp + 8 * (i >> 1), p = p0 + lane + 32 * (i & 1);
            v[i] = c < channels && p < pixels ? load_late(src + (size_t)c * pixels + p) : __half(0.f);
        }
        __syncthreads();                       // the previous tile has been written out
#pragma unroll
        for (int i = 0; i < 16; ++i) s[(lane + 32 * (i & 1)) * STRIDE + warp + 8 * (i >> 1)] = v[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = threadIdx.x + i * kThreads, p = e >> 3, c = (e & 7) * 8;
            if (p0 + p >= pixels || c0 + c >= channels) continue;
            const uint32_t* row = reinterpret_cast<const uint32_t*>(s + p * STRIDE + c);
            *reinterpret_cast<uint4*>(out + ((size_t)b * pixels + p0 + p) * channels + c0 + c) =
                make_uint4(row[0], row[1], row[2], row[3]);
        }
    }
}

// y = relu(y + bias) (+ add), in place; rounded where the separate operations round, and a NaN stays one as with them. A thread's vectors of eight channels
// are whole blocks apart, and 8 * kThreads is a multiple of `channels`, so its bias stays in registers.
__global__ void __launch_bounds__(kThreads)
bias_relu_kernel(__half* __restrict__ y, const __half* __restrict__ bias, const __half* __restrict__ add, int64_t vectors,
                 int channels) {
    pdl_enter();                               // (the bias, too, may be the preceding kernel's work)
    float bv[8];
    unpack8(load_late(reinterpret_cast<const uint4*>(bias) + threadIdx.x % (channels / 8)), bv);
    const int64_t stride = (int64_t)gridDim.x * kThreads;
    for (int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x; e < vectors; e += 2 * stride) {
        uint4 v[2], a[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (e + i * stride >= vectors) break;
            v[i] = reinterpret_cast<const uint4*>(y)[e + i * stride];
            if (add) a[i] = load_late(reinterpret_cast<const uint4*>(add) + e + i * stride);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (e + i * stride >= vectors) break;
            float x[8], r[8];
            unpack8(v[i], x);
            if (add) unpack8(a[i], r);
            uint4 o;
            __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                h[j] = __hmax2_nan(__floats2half2_rn(x[2 * j] + bv[2 * j], x[2 * j + 1] + bv[2 * j + 1]), __half2(0.f, 0.f));
                if (add) {
                    const float2 f = __half22float2(h[j]);
                    h[j] = __floats2half2_rn(f.x + r[2 * j], f.y + r[2 * j + 1]);
                }
            }
            reinterpret_cast<uint4*>(y)[e + i * stride] = o;
        }
    }
}

// The two branches' attention (a 1x1 convolution to one channel each, softmax over the two, weighted sum) and the four
// 1x1 heads, 64 pixels at a time: sums in fp32, rounded to fp16 where the separate operations round. Sixteen lanes share a
// pixel for the attention. The heads are a 64 x 22 x 128 product per tile: too small for tcgen05 (a launch has 3.7 tiles per
// SM), so warps 0-3 take sixteen pixels each with mma.sync. (With one pixel and six outputs per thread
// and fp32 weights in shared memory the kernel took 20 us on a 200 x 176 map, the weights' reads alone 8; so 8.8.)
constexpr int kNeckChannels = 128, kHeadChannels = 22;
struct HeadOut {
    float* out[4];          // [pixels][width]: the heads' outputs as the post-processing takes them (null: not wanted)
    int first[4], width[4];
};
__global__ void __launch_bounds__(kThreads, 4)
neck_tail_kernel(const __half* __restrict__ o0, const __half* __restrict__ o1, const __half* __restrict__ gate_w,
                 const __half* __restrict__ gate_b, const __half* __restrict__ head_w, const __half* __restrict__ head_b,
                 __half* __restrict__ features, const __grid_constant__ HeadOut heads, int64_t pixels) {
    constexpr int C = kNeckChannels, STRIDE = C + 8;   // 17 x 16 bytes: eight rows' words of a fragment lie in different banks
    constexpr int NT = (kHeadChannels + 7) / 8;         // eight output channels each
    __shared__ __align__(16) __half s_x[kTilePixels * STRIDE];
    __shared__ __align__(16) __half s_w[NT * 8 * STRIDE];
    __shared__ float s_out[kTilePixels * kHeadChannels];
    const int tid = threadIdx.x, l16 = tid & 15, lane = tid & 31, warp = tid >> 5;
    const bool want_heads = heads.out[0] != nullptr;
    pdl_enter();                               // (the weights are arguments: they, too, may be the preceding kernel's work)
    float g0[8], g1[8];
    unpack8(load_late(reinterpret_cast<const uint4*>(gate_w) + l16), g0);
    unpack8(load_late(reinterpret_cast<const uint4*>(gate_w + C) + l16), g1);
    const float b0 = __half2float(load_late(gate_b)), b1 = __half2float(load_late(gate_b + 1));
    if (want_heads)
        for (int e = tid; e < NT * 8 * (C / 8); e += kThreads) {
            const int o = e / (C / 8), c = e % (C / 8) * 8;
            *reinterpret_cast<uint4*>(s_w + o * STRIDE + c) =
                o < kHeadChannels ? load_late(reinterpret_cast<const uint4*>(head_w + o * C + c)) : make_uint4(0u, 0u, 0u, 0u);
        }
    const int64_t tiles = (pixels + kTilePixels - 1) / kTilePixels;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t p0 = t * kTilePixels;
        const int rows = pixels - p0 < kTilePixels ? (int)(pixels - p0) : kTilePixels;
        uint4 v0[4], v1[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = (tid >> 4) + 16 * i;
            v0[i] = v1[i] = make_uint4(0u, 0u, 0u, 0u);
            if (p < rows) {
                v0[i] = load_late(reinterpret_cast<const uint4*>(o0 + (p0 + p) * C) + l16);
                v1[i] = load_late(reinterpret_cast<const uint4*>(o1 + (p0 + p) * C) + l16);
            }
        }
        __syncthreads();                       // the previous tile's rows and outputs have been used
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = (tid >> 4) + 16 * i;
            float x0[8], x1[8], d0 = 0.f, d1 = 0.f;
            unpack8(v0[i], x0);
            unpack8(v1[i], x1);
#pragma unroll
            for (int j = 0; j < 8; ++j) d0 = fmaf(x0[j], g0[j], d0), d1 = fmaf(x1[j], g1[j], d1);
#pragma unroll
            for (int d = 8; d; d >>= 1) {
                d0 += __shfl_xor_sync(0xFFFFFFFFu, d0, d);
                d1 += __shfl_xor_sync(0xFFFFFFFFu, d1, d);
            }
            const float g0s = round_half(round_half(d0) + b0), g1s = round_half(round_half(d1) + b1);
            const float top = fmaxf(g0s, g1s), e0 = expf(g0s - top), e1 = expf(g1s - top);
            const __half2 w0 = __float2half2_rn(e0 / (e0 + e1)), w1 = __float2half2_rn(e1 / (e0 + e1));
            uint4 o;
            __half2* h = reinterpret_cast<__half2*>(&o);
            const __half2 *h0 = reinterpret_cast<const __half2*>(&v0[i]), *h1 = reinterpret_cast<const __half2*>(&v1[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = __hadd2_rn(__hmul2_rn(h0[j], w0), __hmul2_rn(h1[j], w1));
            if (features && p < rows) reinterpret_cast<uint4*>(features + (p0 + p) * C)[l16] = o;
            *reinterpret_cast<uint4*>(s_x + p * STRIDE + l16 * 8) = o;
        }
        if (!want_heads) continue;
        __syncthreads();
        if (warp < kTilePixels / 16) {
            float acc[NT][4] = {};
            const __half* row = s_x + (warp * 16 + lane / 4) * STRIDE + (lane & 3) * 2;
            const __half* w = s_w + lane / 4 * STRIDE + (lane & 3) * 2;   // of output 8 nt + lane / 4
#pragma unroll
            for (int k = 0; k < C / 16; ++k) {
                uint32_t a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    a[i] = *reinterpret_cast<const uint32_t*>(row + (i & 1) * 8 * STRIDE + k * 16 + (i >> 1) * 8);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint32_t b0 = *reinterpret_cast<const uint32_t*>(w + nt * 8 * STRIDE + k * 16);
                    const uint32_t b1 = *reinterpret_cast<const uint32_t*>(w + nt * 8 * STRIDE + k * 16 + 8);
                    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                                 : "+f"(acc[nt][0]), "+f"(acc[nt][1]), "+f"(acc[nt][2]), "+f"(acc[nt][3])
                                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
                }
            }
            // each head's part of the tile is one run of s_out, as it is of the output
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int o = nt * 8 + (lane & 3) * 2 + (i & 1), p = warp * 16 + lane / 4 + (i >> 1) * 8;
                    if (o >= kHeadChannels) continue;
                    const float v = round_half(round_half(acc[nt][i]) + __half2float(load_late(head_b + o)));
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int ch = o - heads.first[q];
                        if (ch >= 0 && ch < heads.width[q]) s_out[heads.first[q] * kTilePixels + p * heads.width[q] + ch] = v;
                    }
                }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q)
            for (int e = tid; e < rows * heads.width[q]; e += kThreads)
                heads.out[q][p0 * heads.width[q] + e] = s_out[heads.first[q] * kTilePixels + e];
    }
}

int grid_for(int64_t items, int per_sm) {
    const int64_t most = persistent_grid(per_sm);
    return (int)(items < 1 ? 1 : (items < most ? items : most));
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

}  // namespace sessd

using namespace sessd;

extern "C" {

int sessd_channels_last_enqueue(const void* in, void* out, int batch, int channels, int pixels, void* stream) {
    if (!in || !out || batch < 1 || channels < 8 || channels % 8 || pixels < 1 || !aligned16(out)) return SESSD_ERR_PARAM;
    const int64_t items = (int64_t)batch * ((pixels + kTilePixels - 1) / kTilePixels) * ((channels + 63) / 64);
    if (items > INT32_MAX) return SESSD_ERR_PARAM;
    SESSD_LAUNCH(channels_last_kernel, grid_for(items, 8), kThreads, 0, static_cast<cudaStream_t>(stream),
                 static_cast<const __half*>(in), static_cast<__half*>(out), batch, channels, pixels);
    return SESSD_OK;
}

int sessd_bias_relu_enqueue(void* y, const void* bias, const void* add, long long pixels, int channels, void* stream) {
    if (!y || !bias || pixels < 1 || channels < 8 || channels % 8 || (8 * kThreads) % channels || !aligned16(y) ||
        !aligned16(bias) || !aligned16(add))
        return SESSD_ERR_PARAM;
    const int64_t vectors = (int64_t)pixels * (channels / 8);
    SESSD_LAUNCH(bias_relu_kernel, grid_for((vectors + 2 * kThreads - 1) / (2 * kThreads), 8), kThreads, 0,
                 static_cast<cudaStream_t>(stream), static_cast<__half*>(y), static_cast<const __half*>(bias),
                 static_cast<const __half*>(add), vectors, channels);
    return SESSD_OK;
}

int sessd_neck_tail_enqueue(const void* const* inputs, void* const* outputs, long long pixels, void* stream) {
    if (!inputs || !outputs || pixels < 1) return SESSD_ERR_PARAM;
    for (int i = 0; i < 6; ++i)
        if (!inputs[i] || ((i < 3 || i == 4) && !aligned16(inputs[i]))) return SESSD_ERR_PARAM;
    const bool heads = outputs[1] != nullptr;
    HeadOut h{{nullptr, nullptr, nullptr, nullptr}, {0, 14, 16, 18}, {14, 2, 2, 4}};
    for (int q = 0; q < 4; ++q) {
        if ((outputs[1 + q] != nullptr) != heads) return SESSD_ERR_PARAM;
        h.out[q] = static_cast<float*>(outputs[1 + q]);
    }
    if ((!heads && !outputs[0]) || !aligned16(outputs[0])) return SESSD_ERR_PARAM;
    SESSD_LAUNCH(neck_tail_kernel, grid_for((pixels + kTilePixels - 1) / kTilePixels, 4), kThreads, 0,
                 static_cast<cudaStream_t>(stream), static_cast<const __half*>(inputs[0]), static_cast<const __half*>(inputs[1]),
                 static_cast<const __half*>(inputs[2]), static_cast<const __half*>(inputs[3]),
                 static_cast<const __half*>(inputs[4]), static_cast<const __half*>(inputs[5]),
                 static_cast<__half*>(outputs[0]), h, (int64_t)pixels);
    return SESSD_OK;
}

}  // extern "C"
