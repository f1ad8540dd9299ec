// Output-stationary sparse convolution of the narrow layers in calls with room for many rows: 4 -> 16 channels in fp16 and fp32,
// 16 -> 16 in fp32.
//
// Same arithmetic as conv_simt.cu, bit for bit: per present neighbour a fused-multiply-add chain over ci (ascending) in fp32, the
// neighbours' sums added in ascending kernel offset (submConv3dlayer.cu:503-515 with the order of its atomic additions fixed).
//
// A warp owns a run of 64 consecutive positions of the map (two per lane) and 16 (or 8) output channels, and goes through the offsets
// that any of the run's positions has. All lanes are then at the same offset, so that a weight is read once per warp (a broadcast of
// four from shared memory) and used for 64 rows; a lane without the neighbour multiplies zeros, which adds nothing. Where every row
// walks its own list of neighbours instead (conv_narrow_kernel), rows at different offsets read different weights, which is what
// bounds that kernel, and a warp takes as many steps as its longest list has.
//   - Multiply-adds go two channels per instruction (each rounded like fmaf).
//   - The map's entries of the next run are copied in (cp.async) while the present one is worked on, and the mask of the one after
//     that is read; input rows are requested DEPTH offsets ahead.
// What bounds it is latency, with sixteen warps per SM (twelve with 16 input channels; 128 registers: with one position per lane, twenty
// warps and twice the reads of weights 176 us instead of 164). 4 -> 16 in fp16, 32 frames of 120,000 points (2.6 M rows with 4.8 neighbours; 230 MB, 35 us): 289 us
// before, now 164; of 20,000 points 74 and 50. fp32, 4 x 120,000 points: 4 -> 16 52 and 37, 16 -> 16 144 and 101.
#include <string>

#include "common.cuh"

namespace sessd {

namespace {

constexpr int ROWS_KVOL_MAX = 27;

template <typename T, int CIN>
struct Rows {
    static constexpr int COUT = 16;
    static constexpr int RPL = 2;                        // positions of a lane
    static constexpr int RUN = 32 * RPL;
    static constexpr int CH = CIN == 4 ? 16 : 8;         // channels of a warp
    static constexpr int PARTS = COUT / CH;              // warps that share a run
    static constexpr int WARPS = 4;
    static constexpr int THREADS = WARPS * 32;
    static constexpr int DEPTH = CIN == 4 ? 2 : 1;       // offsets whose rows are requested together, while as many are worked on
    static constexpr int BLOCKS = CIN == 4 ? 4 : 3;                     // per SM
    static constexpr int ROUND = 16;                     // offsets whose entries a run's buffer holds (runs with more are few)
    static constexpr int SLOTS = ROUND + DEPTH;          // .. and those that are requested ahead of the last
    static constexpr int BUFFER = SLOTS * RUN * 4;
    static_assert(ROUND % (2 * DEPTH) == 0 && 4 % DEPTH == 0, "whole steps");
    static constexpr int smem(int kvol) { return kvol * CIN * COUT * 4 + COUT * 8 + WARPS * 2 * BUFFER; }
};

struct RowsArgs {
    const void* in;
    void* out;
    const int32_t* nbr;
    const int32_t* order;
    const uint32_t* tile_mask;
    const int32_t* out_num;
    const void* weights;
    const float *scale, *shift;
    int relu, batch, max_voxels, kvol;
    void* dense;
    const int4* out_coors;
    int D, H, W, maps_ready;
};

using Pair = unsigned long long;                         // two floats
__device__ __forceinline__ Pair pair(float a, float b) {
    Pair v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 unpair(Pair v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
    Pair d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// An input row as it comes, zeros for a missing neighbour. (No branch: behind one, a row was waited for before the next was
// requested.)
template <typename T, int CIN>
struct Row;
template <>
struct Row<__half, 4> {
    uint2 v;
    __device__ __forceinline__ void load(const __half* in, int row) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t"
            "@p ld.global.nc.v2.b32 {%0, %1}, [%2];\n\t}"
            : "=&r"(v.x), "=&r"(v.y)
            : "l"(in + (size_t)(uint32_t)row * 4), "r"(row));
    }
    __device__ __forceinline__ float get(int ci) const {
        const uint32_t w = ci < 2 ? v.x : v.y;
        const __half2 h = *reinterpret_cast<const __half2*>(&w);
        return ci & 1 ? __high2float(h) : __low2float(h);
    }
};
template <int CIN>
struct Row<float, CIN> {
    float4 v[CIN / 4];
    __device__ __forceinline__ void load(const float* in, int row) {
        const float* p = in + (size_t)(uint32_t)row * CIN;
#pragma unroll
        for (int i = 0; i < CIN / 4; ++i)
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                "@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                : "=&f"(v[i].x), "=&f"(v[i].y), "=&f"(v[i].z), "=&f"(v[i].w)
                : "l"(p + 4 * i), "r"(row));
    }
    __device__ __forceinline__ float get(int ci) const {
        const float4& f = v[ci / 4];
        return (ci & 3) == 0 ? f.x : ((ci & 3) == 1 ? f.y : ((ci & 3) == 2 ? f.z : f.w));
    }
};

__device__ __forceinline__ float weight_as_float(float w) { return w; }
__device__ __forceinline__ float weight_as_float(__half w) { return __half2float(w); }

// Channels of an output row.
template <int N>
__device__ __forceinline__ void store_channels(float* p, const float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}
template <int N>
__device__ __forceinline__ void store_channels(__half* p, const float (&v)[N]) {
    __align__(16) __half2 h[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < N / 8; ++i) reinterpret_cast<uint4*>(p)[i] = reinterpret_cast<const uint4*>(h)[i];
}

template <typename T, int CIN>
__global__ void __launch_bounds__((Rows<T, CIN>::THREADS), (Rows<T, CIN>::BLOCKS))
conv_rows_kernel(const __grid_constant__ RowsArgs a) {
    using R = Rows<T, CIN>;
    constexpr int COUT = R::COUT, DEPTH = R::DEPTH, RPL = R::RPL, NP = R::CH / 2;
    extern __shared__ __align__(16) uint8_t rows_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* s_w = reinterpret_cast<float*>(rows_smem);                            // [kvol][CIN][COUT]
    float2* s_epi = reinterpret_cast<float2*>(s_w + a.kvol * CIN * COUT);        // scale and shift of a channel
    uint8_t* s_buf = reinterpret_cast<uint8_t*>(s_epi + COUT) + warp * (2 * R::BUFFER);
    // weights, scale and shift are older than any preceding kernel
    for (int e = tid; e < a.kvol * CIN * COUT; e += R::THREADS) s_w[e] = weight_as_float(__ldg(static_cast<const T*>(a.weights) + e));
    if (tid < COUT)
        s_epi[tid] = make_float2(a.scale ? __ldg(a.scale + tid) : 1.f, a.scale && a.shift ? __ldg(a.shift + tid) : 0.f);
    __syncthreads();
    // map, masks and row counts are older than the preceding kernel where maps_ready says so
    if (!a.maps_ready) pdl_enter();

    // Runs, numbered over the frames: a walk that only moves forward, 32 frames at a time (lane = frame), the same in all lanes.
    const int tiles_per_frame = (a.max_voxels + 127) / 128, stride = (int)gridDim.x * (R::WARPS / R::PARTS);
    int f0 = 0, before = 0, rows = 0, incl = 0;
    auto load_frames = [&]() {
        rows = f0 + lane < a.batch ? load_late(a.out_num + f0 + lane) : 0;
        rows = rows > a.max_voxels ? a.max_voxels : (rows < 0 ? 0 : rows);
        incl = (rows + R::RUN - 1) / R::RUN;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += v;
        }
    };
    load_frames();
    struct Run { int frame, pos, rows; uint32_t mask; };     // frame (-1: there is none), first position, rows of the frame, offsets
    auto locate = [&](int it) {
        int total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        while (it >= before + total && f0 + 32 < a.batch) {
            before += total;
            f0 += 32;
            load_frames();
            total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        if (it >= before + total) return Run{-1, 0, 0, 0u};
        const int src = __ffs((int)__ballot_sync(0xFFFFFFFFu, it < before + incl)) - 1;
        const int n = __shfl_sync(0xFFFFFFFFu, rows, src);
        const int pos = (it - before - (__shfl_sync(0xFFFFFFFFu, incl, src) - (n + R::RUN - 1) / R::RUN)) * R::RUN;
        const int32_t* runs = a.nbr + nbr_runs_index(a.kvol, a.max_voxels, f0 + src, pos);
        const int offsets = load_late(runs) | (pos + 32 < n ? load_late(runs + 1) : 0);
        return Run{f0 + src, pos, n,
                   load_late(a.tile_mask + (size_t)(f0 + src) * tiles_per_frame + (pos >> 7)) & (uint32_t)offsets};
    };
    // Offsets go through a run's buffer up to ROUND at a time: `more` gets those that are left.
    auto split = [&](uint32_t mask, uint32_t* more) {
        uint32_t rest = 0;
        if (__popc(mask) > R::ROUND) {
            rest = mask;
#pragma unroll
            for (int i = 0; i < R::ROUND; ++i) rest &= rest - 1u;
        }
        *more = rest;
        return mask & ~rest;
    };
    // Entries of a run under the offsets of `mask`, one after the other, and -1 for those that are only requested. Sixteen lanes copy an
    // offset's 256 bytes.
    auto copy_entries = [&](const Run& r, uint32_t mask, uint8_t* buffer) {
        constexpr int LANES = R::RUN / 4;
        const int32_t* at = a.nbr + nbr_index(a.kvol, a.max_voxels, r.frame, 0, r.pos) + 4 * (lane % LANES);
        uint32_t dst = (uint32_t)__cvta_generic_to_shared(buffer) + lane * 16;
        const int n = (__popc(mask) + 2 * DEPTH - 1) / (2 * DEPTH) * (2 * DEPTH) + DEPTH;
        for (int i = 0; i < lane / LANES; ++i) mask &= mask - 1u;
        for (int i = lane / LANES; i < n; i += 32 / LANES, dst += 512) {
            if (mask)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(at + (__ffs((int)mask) - 1) * kNbrRun) : "memory");
            else
                asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(-1) : "memory");
#pragma unroll
            for (int j = 0; j < 32 / LANES; ++j) mask &= mask - 1u;
        }
        __syncwarp();
    };
    const int part = warp % R::PARTS * R::CH;                   // first channel of the warp
    int it = (int)blockIdx.x * (R::WARPS / R::PARTS) + warp / R::PARTS, buffer = 0;
    uint32_t more;
    Run next = locate(it), after = next;
    if (next.frame >= 0) {
        copy_entries(next, split(next.mask, &more), s_buf);
        after = locate(it += stride);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (a.maps_ready) pdl_enter();
    for (; next.frame >= 0; buffer ^= 1) {
        // the run, whose entries are on their way; the one after it, whose entries start now; and the one after that, whose mask does
        const Run cur = next;
        next = after;
        uint8_t* buf = s_buf + buffer * R::BUFFER;
        if (next.frame >= 0) {
            copy_entries(next, split(next.mask, &more), s_buf + (buffer ^ 1) * R::BUFFER);
            after = locate(it += stride);
        }
        bool live[RPL];
        int out_row[RPL];
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            const int pos = cur.pos + 32 * i + lane;
            live[i] = pos < cur.rows;
            out_row[i] = a.order && live[i] ? __ldg(a.order + (size_t)cur.frame * a.max_voxels + pos) : pos;
        }
        const T* in = static_cast<const T*>(a.in) + (size_t)cur.frame * a.max_voxels * CIN;
        Pair acc[RPL][NP];
#pragma unroll
        for (int i = 0; i < RPL; ++i)
#pragma unroll
            for (int p = 0; p < NP; ++p) acc[i][p] = 0ull;
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        uint32_t mask = split(cur.mask, &more);
        for (;;) {
#pragma unroll
            for (int i = 0; i < RPL; ++i)
                if (!live[i])                                // positions past the frame's rows hold anything
                    for (int j = 0; j < __popc(mask); ++j) *reinterpret_cast<int*>(buf + j * (R::RUN * 4) + (32 * i + lane) * 4) = -1;
            const uint8_t* slot = buf + lane * 4;
            Row<T, CIN> x[2][DEPTH][RPL];
            auto request = [&](Row<T, CIN> (&r)[DEPTH][RPL]) {
#pragma unroll
                for (int i = 0; i < DEPTH; ++i)
#pragma unroll
                    for (int j = 0; j < RPL; ++j) r[i][j].load(in, *reinterpret_cast<const int*>(slot + i * (R::RUN * 4) + j * 128));
                slot += DEPTH * R::RUN * 4;
            };
            auto work = [&](const Row<T, CIN> (&r)[DEPTH][RPL]) {
#pragma unroll
                for (int i = 0; i < DEPTH; ++i) {
                    if (!mask) break;                        // (uniform over the warp)
                    const float4* w = reinterpret_cast<const float4*>(s_w + (__ffs((int)mask) - 1) * (CIN * COUT) + part);
                    mask &= mask - 1u;
                    Pair s[RPL][NP];
#pragma unroll
                    for (int ci = 0; ci < CIN; ++ci) {
#pragma unroll
                        for (int p = 0; p < NP; p += 2) {
                            const float4 f = w[ci * (COUT / 4) + p / 2];
#pragma unroll
                            for (int j = 0; j < RPL; ++j) {
                                const Pair v = pair(r[i][j].get(ci), r[i][j].get(ci));
                                s[j][p] = fma2(v, pair(f.x, f.y), ci ? s[j][p] : 0ull);
                                s[j][p + 1] = fma2(v, pair(f.z, f.w), ci ? s[j][p + 1] : 0ull);
                            }
                        }
                    }
#pragma unroll
                    for (int j = 0; j < RPL; ++j)
#pragma unroll
                        for (int p = 0; p < NP; ++p) acc[j][p] = add2(acc[j][p], s[j][p]);
                }
            };
            request(x[0]);
            while (mask) {
                request(x[1]);
                work(x[0]);
                request(x[0]);
                work(x[1]);
            }
            __syncwarp();                                    // the buffer has been read
            if (!more) break;
            mask = split(more, &more);
            copy_entries(cur, mask, buf);
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
            __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            if (!live[i]) continue;
            float v[R::CH];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const float4 e = *reinterpret_cast<const float4*>(s_epi + part + 2 * p);
                const float2 f = unpair(acc[i][p]);
                v[2 * p] = fmaf(f.x, e.x, e.y), v[2 * p + 1] = fmaf(f.y, e.z, e.w);
                if (a.relu) v[2 * p] = v[2 * p] > 0.f ? v[2 * p] : 0.f, v[2 * p + 1] = v[2 * p + 1] > 0.f ? v[2 * p + 1] : 0.f;
            }
            const size_t row = (size_t)cur.frame * a.max_voxels + out_row[i];
            store_channels(static_cast<T*>(a.out) + row * COUT + part, v);
            if (a.dense) {
                // fused BEV scatter (sparse2Dense.cu:201-206): channel c*D + z, pixel (y, x)
                const int4 c4 = __ldg(&a.out_coors[row]);
                const size_t plane = (size_t)a.D * a.H * a.W;
                T* d = static_cast<T*>(a.dense) + ((size_t)cur.frame * COUT + part) * plane + ((size_t)c4.y * a.H + c4.z) * a.W + c4.w;
#pragma unroll
                for (int c = 0; c < R::CH; ++c) d[c * plane] = static_cast<T>(v[c]);
            }
        }
    }
}

template <typename T, int CIN>
int launch_one(const ConvLaunch& c, cudaStream_t stream) {
    using R = Rows<T, CIN>;
    static const std::string name = std::string("conv_rows<") + (sizeof(T) == 4 ? "f32," : "f16,") + std::to_string(CIN) + ",16>";
    if (R::smem(ROWS_KVOL_MAX) > 48 * 1024) {
        // the attribute belongs to the device's context: set it once per device (repeating it is harmless)
        static std::atomic<uint64_t> configured{0};
        int dev = 0;
        SESSD_CUDA(cudaGetDevice(&dev));
        const uint64_t bit = 1ull << (dev & 63);
        if (!(configured.load(std::memory_order_acquire) & bit)) {
            SESSD_CUDA(cudaFuncSetAttribute(conv_rows_kernel<T, CIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            R::smem(ROWS_KVOL_MAX)));
            configured.fetch_or(bit, std::memory_order_release);
        }
    }
    const RowsArgs a{c.in, c.out, c.nbr, c.order, c.tile_mask, c.out_num, c.weights, c.scale, c.shift, c.relu, c.batch, c.max_voxels,
                     c.kvol, c.dense, reinterpret_cast<const int4*>(c.out_coors), c.D, c.H, c.W, c.maps_ready};
    const int64_t units = (int64_t)c.batch * ((c.max_voxels + R::RUN - 1) / R::RUN) * R::PARTS;
    const int64_t blocks = (units + R::WARPS - 1) / R::WARPS;
    const int most = persistent_grid(R::BLOCKS);
    SESSD_LAUNCH_NAMED(name.c_str(), (conv_rows_kernel<T, CIN>), (int)(blocks < most ? blocks : most), R::THREADS, R::smem(c.kvol),
                       stream, a);
    return SESSD_OK;
}

}  // namespace

// Where few rows are in use the narrow kernel's rows, a few threads each, are through sooner than a lane with all of a run's offsets;
// beyond that a run's weights, read once for 64 rows, pay. Row counts are on the device, so the line goes by what the host knows: the
// room, and in a front end the points, which level 0 has no more rows than.
//   - Room for 300,000 rows or less: narrow. The front end's first layer in us, narrow and here: fp16 1 x 20,000 points (room for 60,000)
//     11 and 16, 1 x 120,000 (200,000) 18.8 and 18.7, 4 x 20,000 (240,000) 18.9 and 18.9, 5 x 20,000 (300,000) 20.9 and 20.6.
//   - Room for 300,000 to 800,000: narrow up to 80,000 points in fp16 and 40,000 in fp32. Front ends in us, narrow and here: fp16 8 x 3,000
//     points (480,000) 304 and 310, 3 x 22,000 (600,000) 325 and 328, 8 x 9,000 436 and 438, 2 x 40,000 (400,000) 328 and 327, 4 x 22,000
//     (800,000) 398 and 394, 8 x 20,000 621 and 611; fp32, two layers, 6 x 3,000 (360,000) 1153 and 1161, 8 x 4,000 1869 and 1869, 2 x 22,000
//     1499 and 1495, 6 x 9,000 2373 and 2377, 2 x 30,000 1825 and 1808, 8 x 8,000 2963 and 2952.
//   - More room: here (narrow blocks look at every row there is room for). fp16 14 x 3,000 points (840,000) 427 and 427, 32 x 1,000 531
//     and 526; fp32 14 x 3,000 2556 and 2547.
// A plugin call's room is all there is: with a third of it in use calls are faster here (4 -> 16 fp16, 8 x 20,000 points 39 and 27, 2 x 30,000
// 23 and 21; fp32 16 -> 16 84 and 74, 46 and 35), with a tenth slower (fp16 8 x 3,000 15 and 17, 16 -> 16 21 and 29).
// fp32 16 -> 32 is no faster here at any size (4 x 120,000 236 and 246).
// A weight that is no finite number must not reach the rows without its neighbour, which multiply it by zero here. Rows are read in
// pieces of 8 (halves) or 16 bytes and written in pieces of 16.
bool conv_rows_takes(const ConvLaunch& c) {
    if (!c.weights_finite || !c.tile_mask || c.kvol > ROWS_KVOL_MAX) return false;
    const bool half = c.dtype == SESSD_F16;
    const int64_t room = (int64_t)c.batch * c.max_voxels;
    if (room <= kRunRows || (room < 800000 && c.most_rows < (half ? 80000 : 40000))) return false;
    if (c.cout != 16 || !(c.cin == 4 || (c.cin == 16 && !half))) return false;
    return reinterpret_cast<uintptr_t>(c.in) % (half ? 8 : 16) == 0 && reinterpret_cast<uintptr_t>(c.out) % 16 == 0;
}

int launch_conv_rows(const ConvLaunch& c, cudaStream_t stream) {
    if (c.dtype == SESSD_F16) return launch_one<__half, 4>(c, stream);
    return c.cin == 4 ? launch_one<float, 4>(c, stream) : launch_one<float, 16>(c, stream);
}

}  // namespace sessd
