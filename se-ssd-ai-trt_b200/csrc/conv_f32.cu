// Output-stationary sparse convolution in fp32 for the wide layers (32 and 64 channels).
//
// Same arithmetic as conv_simt.cu, bit for bit: per present neighbour a fused-multiply-add chain over ci (ascending)
// from zero, the neighbours' sums added in ascending kernel offset (submConv3dlayer.cu:503-515 with the order of its
// atomic additions fixed).
//
// What bounds it: the fp32 pipe (128 multiply-adds per clock and SM) and, close behind, the 128 bytes per clock that
// shared memory hands to registers. A thread that owns one output row and reads a weight vector per channel and row is
// bound by those reads (3 TFLOP/s). Hence this shape:
//   - a warp owns a strip of 16 (or 8) output rows and walks the kernel offsets alone, so that the order of a row's
//     additions needs no barrier. The strip is a register tile, 4 (2) rows x 8 or 4 channels per thread; an offset that
//     no row of the strip has is skipped, a row without the neighbour keeps its sum. (Compacting the present rows of a
//     larger strip saves a third of the multiply-adds, but its tiles' accumulators then live in shared memory and the
//     strips' serial chains get twice as long: slower on single frames.)
//   - the input rows of the strip's next offset are copied in while the current one is worked on;
//   - the lanes of a tile are (channel group = lane / 4, row group = lane % 4): two-channel weight loads then have
//     neighbouring lanes at the same address and cost one cycle for the warp instead of two (measured: 1.1 cycles when
//     lanes 4 i .. 4 i + 3 agree, 2.0 when the address depends on lane % 8);
//   - multiply-adds go two channels per instruction (each rounded like fmaf): a lone warp of a scheduler issues an fp32
//     instruction every second cycle only, and a single frame has one to three warps per scheduler;
//   - the strip warps of a block (one block per SM) share the weights: one more warp streams the offsets' blocks into a
//     ring with bulk copies, so that warps may be a few offsets apart.
// Strips are dealt out over the SMs first, so that a small frame uses all of them.
// Measured (events around the launch, 20,000-point frame): 64->64 at 1/4 resolution (26,400 rows, 417,000 pairs) 144 us,
// at 1/8 resolution (11,300 rows) 78 us, 32->32 at 1/2 resolution (38,200 rows) 95 us; one row per thread took 845, 495
// and 150 us.
#include <string>

#include "mbarrier.cuh"

namespace sessd {

namespace {

constexpr int F32_WARPS = 15;                // strip warps per block; one more streams the weights
constexpr int F32_THREADS = (F32_WARPS + 1) * 32;
constexpr int F32_KVOL_MAX = 27;

template <int CIN, int COUT>
struct F32Shared {
    static constexpr int STAGES = CIN * COUT > 2048 ? 4 : 8;     // weight ring (64 KB at most)
    float w[STAGES][CIN * COUT];
    struct Strip {
        float x[2][16 * CIN];                        // input rows of the current and the next offset
        int32_t idx[F32_KVOL_MAX][16];               // the strip's map entries
    } strip[F32_WARPS];
    unsigned long long full[STAGES], empty[STAGES];
    uint32_t mask[F32_WARPS];                        // offsets of every warp's tile, for the union
    int abort_flag, abort_where;                     // (mbar_wait expects them in this order)
    int stop;
};

struct F32Args {
    const float* in;
    float* out;
    const int32_t* nbr;
    const int32_t* order;
    const uint32_t* tile_mask;
    const int32_t* out_num;
    const float *weights, *scale, *shift;
    int relu, batch, max_voxels, kvol;
    float* dense;
    const int4* out_coors;
    int D, H, W;
    int32_t* status;
};

__device__ __forceinline__ void copy_16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ unsigned long long pair(float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 unpair(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ int f32_frame_rows(const F32Args& a, int f) {
    const int n = f < a.batch ? __ldg(a.out_num + f) : 0;
    return n > a.max_voxels ? a.max_voxels : (n < 0 ? 0 : n);
}

// RT rows per thread: a strip has 4 RT rows.
template <int CIN, int COUT, int RT>
__device__ __forceinline__ void f32_run(F32Shared<CIN, COUT>& s, const F32Args& a) {
    constexpr int STRIP = 4 * RT;
    constexpr int STAGES = F32Shared<CIN, COUT>::STAGES;
    constexpr int NP = COUT / 16;                    // channel pairs per thread: channels 16 p + 2 cg, + 1
    constexpr int CPR = CIN / 4;                     // 16-byte pieces of an input row
    constexpr uint32_t W_BYTES = CIN * COUT * 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rg = lane & 3, cg = lane >> 2;         // row group and channel group of the lane
    volatile int* abort_flag = &s.abort_flag;
    const int tiles_per_frame = (a.max_voxels + 127) / 128;
    uint32_t used = 0;                               // weight blocks of the rounds so far (the same for every warp)
    uint32_t issued = 0;                             // weight streamer: blocks whose copy has been started
    for (int round = 0;; ++round) {
        // strip of this warp: strips are numbered frame by frame and dealt out block by block
        const int64_t want = ((int64_t)round * F32_WARPS + (warp < F32_WARPS ? warp : 0)) * gridDim.x + blockIdx.x;
        int b = 0, row0 = 0, rows = 0;
        {
            int64_t before = 0;
            for (int f0 = 0; f0 < a.batch; f0 += 32) {
                int n = f32_frame_rows(a, f0 + lane);
                const int strips = (n + STRIP - 1) / STRIP;
                int incl = strips;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (lane >= d) incl += v;
                }
                const int64_t at = want - before;
                const uint32_t hit = __ballot_sync(0xFFFFFFFFu, at < incl && at >= incl - strips);
                if (hit) {
                    const int src = __ffs((int)hit) - 1;
                    b = f0 + src;
                    const int first = __shfl_sync(0xFFFFFFFFu, incl - strips, src);
                    n = __shfl_sync(0xFFFFFFFFu, n, src);
                    row0 = (int)(at - first) * STRIP;
                    rows = n - row0 < STRIP ? n - row0 : STRIP;
                    break;
                }
                before += __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
        }
        uint32_t mask = 0;                           // offsets that have a neighbour in this strip's tile
        if (rows > 0 && warp < F32_WARPS)
            mask = __ldg(a.tile_mask + (size_t)b * tiles_per_frame + (row0 >> 7)) & ((1u << a.kvol) - 1u);
        // the strip's rows under each of them: lane k keeps the row bits of offset k
        uint32_t have = 0, have_any = 0;
        if (mask) {
            typename F32Shared<CIN, COUT>::Strip& my = s.strip[warp];
            const int32_t* map = a.nbr + nbr_index(a.kvol, a.max_voxels, b, 0, row0) + lane;
            int idx[F32_KVOL_MAX];
#pragma unroll
            for (int k = 0; k < F32_KVOL_MAX; ++k) idx[k] = ((mask >> k) & 1u) && lane < rows ? __ldg(map + k * kNbrRun) : -1;
#pragma unroll
            for (int k = 0; k < F32_KVOL_MAX; ++k) {
                const uint32_t bits = __ballot_sync(0xFFFFFFFFu, idx[k] >= 0);
                if (lane < STRIP) my.idx[k][lane] = idx[k];
                if (lane == k) have = bits;
                have_any |= (bits ? 1u : 0u) << k;
            }
        }
        __syncthreads();                             // everybody is done with the previous round's union
        if (tid == 0) s.stop = *abort_flag;
        if (warp < F32_WARPS && lane == 0) s.mask[warp] = rows > 0 ? have_any | 0x80000000u : 0u;   // top bit: has a strip
        __syncthreads();
        uint32_t any = 0;
#pragma unroll
        for (int i = 0; i < F32_WARPS; ++i) any |= s.mask[i];
        if (any == 0u || s.stop) break;              // no strip left for any warp of the block
        any &= 0x7FFFFFFFu;

        if (warp == F32_WARPS) {
            // ---- weight streamer ----
            if (lane == 0) {
                uint32_t q = used;
                for (uint32_t m = any; m; m &= m - 1u, ++q) {
                    const uint32_t st = q % STAGES;
                    if (!mbar_wait(smem_u32(&s.empty[st]), ((q / STAGES) & 1u) ^ 1u, abort_flag, 9 | (int)(q << 4))) break;
                    mbar_arrive_expect_tx(smem_u32(&s.full[st]), W_BYTES);
                    bulk_load(smem_u32(s.w[st]), a.weights + (size_t)(__ffs((int)m) - 1) * CIN * COUT, W_BYTES,
                              smem_u32(&s.full[st]));
                    issued = q + 1u;
                }
            }
            __syncwarp();
            used += __popc(any);
            continue;
        }

        // ---- strip ----
        typename F32Shared<CIN, COUT>::Strip& my = s.strip[warp];
        const float* in_b = a.in + (size_t)b * a.max_voxels * CIN;
        // copy of the input rows of offset k: piece c of row r lands at piece c ^ (r / RT), so that the four row groups
        // read different banks; rows without the neighbour keep what an earlier copy left (their sums are not used)
        auto fetch = [&](int k, uint32_t bits, float* dst) {
#pragma unroll
            for (int r0 = 0; r0 < STRIP; r0 += 4) {
                const int r = r0 + (lane >> 3);
                if ((bits >> r) & 1u) {
                    const float* src = in_b + (size_t)my.idx[k][r] * CIN;
#pragma unroll
                    for (int c = 0; c < CPR; c += 8)
                        copy_16(dst + r * CIN + (((c + (lane & 7)) ^ (r / RT)) * 4), src + (c + (lane & 7)) * 4);
                }
            }
        };
        unsigned long long acc[RT][NP];
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int p = 0; p < NP; ++p) acc[i][p] = 0ull;
        int buf = 0;
        uint32_t ahead = have_any;                   // own offsets not begun yet
        uint32_t bits = 0;                           // rows of the strip under the next of them
        if (ahead) {
            const int k = __ffs((int)ahead) - 1;
            bits = __shfl_sync(0xFFFFFFFFu, have, k);
            fetch(k, bits, my.x[0]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        uint32_t q = used;
        bool ok = true;
        for (uint32_t m = any; m; m &= m - 1u, ++q) {
            const int k = __ffs((int)m) - 1;
            const uint32_t st = q % STAGES;
            ok = mbar_wait(smem_u32(&s.full[st]), (q / STAGES) & 1u, abort_flag, 10 | (int)(q << 4));
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            if ((have_any >> k) & 1u) {
                const uint32_t rows_k = bits;
                ahead &= ahead - 1u;
                if (ahead) {
                    const int k_next = __ffs((int)ahead) - 1;
                    bits = __shfl_sync(0xFFFFFFFFu, have, k_next);
                    fetch(k_next, bits, my.x[buf ^ 1]);
                }
                asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
                __syncwarp();
                const float* x = my.x[buf] + rg * RT * CIN;
                const float* w = s.w[st] + cg * 2;
                unsigned long long sum[RT][NP];
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int p = 0; p < NP; ++p) sum[i][p] = 0ull;
#pragma unroll 2
                for (int c4 = 0; c4 < CPR; ++c4) {
                    float4 xv[RT];
#pragma unroll
                    for (int i = 0; i < RT; ++i) xv[i] = *reinterpret_cast<const float4*>(x + i * CIN + ((c4 ^ rg) * 4));
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        unsigned long long wv[NP];
#pragma unroll
                        for (int p = 0; p < NP; ++p)
                            wv[p] = *reinterpret_cast<const unsigned long long*>(w + (c4 * 4 + j) * COUT + p * 16);
#pragma unroll
                        for (int i = 0; i < RT; ++i) {
                            const float v = j == 0 ? xv[i].x : (j == 1 ? xv[i].y : (j == 2 ? xv[i].z : xv[i].w));
                            const unsigned long long vv = pair(v, v);
#pragma unroll
                            for (int p = 0; p < NP; ++p) fma2(sum[i][p], vv, wv[p]);
                        }
                    }
                }
                __syncwarp();   // the buffer may be refilled
#pragma unroll
                for (int i = 0; i < RT; ++i)
                    if ((rows_k >> (rg * RT + i)) & 1u) {
#pragma unroll
                        for (int p = 0; p < NP; ++p) {
                            const float2 v = unpair(acc[i][p]), t = unpair(sum[i][p]);
                            acc[i][p] = pair(__fadd_rn(v.x, t.x), __fadd_rn(v.y, t.y));
                        }
                    }
                buf ^= 1;
            }
            if (lane == 0) mbar_arrive(smem_u32(&s.empty[st]));
        }
        used += __popc(any);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        if (!ok || rows <= 0) continue;
        // folded batch norm and ReLU; a store instruction writes 64 bytes of four rows
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const int r = rg * RT + i;
            if (r >= rows) continue;
            const size_t pos = (size_t)b * a.max_voxels + row0 + r;
            const size_t row = a.order ? (size_t)b * a.max_voxels + __ldg(a.order + pos) : pos;
            float* dst = a.out + row * COUT;
            float* d = nullptr;
            const size_t plane = (size_t)a.D * a.H * a.W;
            if (a.dense) {
                // fused BEV scatter (sparse2Dense.cu:201-206): channel c*D + z, pixel (y, x)
                const int4 c4 = __ldg(&a.out_coors[row]);
                d = a.dense + (size_t)b * COUT * plane + ((size_t)c4.y * a.H + c4.z) * a.W + c4.w;
            }
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const int c = p * 16 + cg * 2;
                float2 v = unpair(acc[i][p]);
                if (a.scale) {
                    const float2 sc = __ldg(reinterpret_cast<const float2*>(a.scale + c));
                    const float2 sh = a.shift ? __ldg(reinterpret_cast<const float2*>(a.shift + c)) : make_float2(0.f, 0.f);
                    v = make_float2(fmaf(v.x, sc.x, sh.x), fmaf(v.y, sc.y, sh.y));
                }
                if (a.relu) v = make_float2(v.x > 0.f ? v.x : 0.f, v.y > 0.f ? v.y : 0.f);
                *reinterpret_cast<float2*>(dst + c) = v;
                if (d) d[c * plane] = v.x, d[(c + 1) * plane] = v.y;
            }
        }
    }
    if (*abort_flag && warp == F32_WARPS && lane == 0) {
        // leave only when no bulk copy of this block is still on its way (bounded)
        for (uint32_t j = issued > STAGES ? issued - STAGES : 0u; j < issued; ++j) {
            const long long t0 = clock64();
            while (!mbar_try_wait(smem_u32(&s.full[j % STAGES]), (j / STAGES) & 1u) && clock64() - t0 < WAIT_LIMIT_CYCLES) {}
        }
        atomicOr(a.status, SESSD_STATUS_TIMEOUT);
        atomicCAS(a.status + 1, 0, s.abort_where);
    }
}

// Strips of 8 rows while a block has no more than one round of them (17,760 rows), of 16 rows otherwise: a short strip's chain
// is half as long and more warps share the schedulers, a high one loads a third fewer operands per multiply-add.
__device__ __forceinline__ bool f32_short_strips(const F32Args& a) {
    const int limit = F32_WARPS * (int)gridDim.x;
    int strips = 0;
    for (int f0 = 0; f0 < a.batch && strips <= limit; f0 += 32)
        strips += __reduce_add_sync(0xFFFFFFFFu, (f32_frame_rows(a, f0 + (threadIdx.x & 31)) + 7) / 8);
    return strips <= limit;
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(F32_THREADS, 1) conv_f32_kernel(const __grid_constant__ F32Args a) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t f32_smem[];
    F32Shared<CIN, COUT>& s = *reinterpret_cast<F32Shared<CIN, COUT>*>(f32_smem);
    if (threadIdx.x == 0) {
        for (int i = 0; i < F32Shared<CIN, COUT>::STAGES; ++i) {
            mbar_init(smem_u32(&s.full[i]), 1);              // the streamer's expect
            mbar_init(smem_u32(&s.empty[i]), F32_WARPS);     // every strip warp has read the block
        }
        s.abort_flag = s.abort_where = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (f32_short_strips(a)) f32_run<CIN, COUT, 2>(s, a);
    else f32_run<CIN, COUT, 4>(s, a);
}

template <int CIN, int COUT>
int launch_one(const ConvLaunch& c, cudaStream_t stream) {
    static const std::string name = "conv_f32<" + std::to_string(CIN) + "," + std::to_string(COUT) + ">";
    constexpr int smem = (int)sizeof(F32Shared<CIN, COUT>);
    static_assert(smem <= 227 * 1024, "the strips do not fit the shared memory of one SM");
    // the attribute belongs to the device's context: set it once per device (repeating it is harmless)
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    SESSD_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        SESSD_CUDA(cudaFuncSetAttribute(conv_f32_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured.fetch_or(bit, std::memory_order_release);
    }
    const F32Args a{static_cast<const float*>(c.in), static_cast<float*>(c.out), c.nbr, c.order, c.tile_mask, c.out_num,
                    static_cast<const float*>(c.weights), c.scale, c.shift, c.relu, c.batch, c.max_voxels, c.kvol,
                    static_cast<float*>(c.dense), reinterpret_cast<const int4*>(c.out_coors), c.D, c.H, c.W, c.status};
    SESSD_LAUNCH_NAMED(name.c_str(), (conv_f32_kernel<CIN, COUT>), persistent_grid(1), F32_THREADS, smem, stream, a);
    return SESSD_OK;
}

}  // namespace

// From 32 input channels on: below that a row's work per neighbour is a few hundred multiply-adds and the hand-overs
// would dominate (the 16-channel layers run in conv_simt.cu).
bool conv_f32_supported(int cin, int cout, int kvol) {
    return (cin == 32 || cin == 64) && (cout == 32 || cout == 64) && kvol <= F32_KVOL_MAX;
}

int launch_conv_f32(const ConvLaunch& c, cudaStream_t stream) {
    if (c.dtype != SESSD_F32 || !c.tile_mask) return SESSD_ERR_UNSUPPORTED;
    if (c.cin == 32 && c.cout == 32) return launch_one<32, 32>(c, stream);
    if (c.cin == 32 && c.cout == 64) return launch_one<32, 64>(c, stream);
    if (c.cin == 64 && c.cout == 32) return launch_one<64, 32>(c, stream);
    if (c.cin == 64 && c.cout == 64) return launch_one<64, 64>(c, stream);
    return SESSD_ERR_UNSUPPORTED;
}

}  // namespace sessd
