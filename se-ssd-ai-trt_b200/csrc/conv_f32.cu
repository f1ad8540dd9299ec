// Output-stationary sparse convolution in fp32 for the wide layers (32 and 64 channels).
//
// Same arithmetic as conv_simt.cu, bit for bit: per present neighbour a fused-multiply-add chain over ci (ascending)
// from zero, the neighbours' sums added in ascending kernel offset (submConv3dlayer.cu:503-515 with the order of its
// atomic additions fixed).
//
// What bounds it: the fp32 pipe (128 multiply-adds per clock and SM) and, close behind, the 128 bytes per clock that
// shared memory hands to registers. A thread that owns one output row and reads a weight vector per channel and row is
// bound by those reads (3 TFLOP/s). Hence this shape:
//   - a block (one per SM) owns up to ROWS output rows, eight by eight from all over the map, so that blocks get alike shares
//     although the map's rows are ordered by their neighbours. Per offset it lists the rows that have the neighbour, and sixteen of a
//     list at a time, offset by offset, go to its warps in turn: rows without the neighbour cost nothing, and a warp that is early
//     waits to add its sums until the offset before has all of its own;
//   - sixteen rows are a register tile, 4 rows x 8 (or 4) channels per thread; their sums under the offset are added to the rows'
//     sums in shared memory once all of the offset before have been: ascending offsets, whichever warps they fall to;
//   - the input rows of a warp's next sixteen are copied in while the current ones are worked on;
//   - the lanes of a tile are (channel group = lane / 4, row group = lane % 4): two-channel weight loads then have
//     neighbouring lanes at the same address and cost one cycle for the warp instead of two (measured: 1.1 cycles when
//     lanes 4 i .. 4 i + 3 agree, 2.0 when the address depends on lane % 8);
//   - multiply-adds go two channels per instruction (each rounded like fmaf): a lone warp of a scheduler issues an fp32
//     instruction every second cycle only, and a single frame has a few warps per scheduler;
//   - the block's warps share the weights: one more warp streams the offsets' blocks into a ring with bulk copies.
// Waits are barriers, which park a warp: with counters in shared memory that a lane polls, the waiting warps took so many
// issue slots that the same kernel was no faster than one strip of rows per warp.
// Measured against that (a warp took sixteen rows through all offsets, rows without the neighbour included): front end of a
// 20,000-point frame 1003 us, now 809 (64->64 at 1/4 resolution, 26,400 rows, 125 us a layer, now 112; at 1/8, 11,300 rows, 67 and 57;
// 32->64 between 1/2 and 1/4 71 and 38), of 3,000 points 531 and 420, of 2 x 40,000 2551 and 2238; calls of 4 x 120,000 points,
// 32->32 1157 and 1073, 64->64 1471 and 1450. Dense maps have few rows to leave out: 4 x 30,000 rows with 18 of 27 neighbours, 32->32
// 227 and 237, 64->64 580 and 486. On one 120,000-point frame the 64->64 kernel keeps the fp32 pipe active 53 % of the time and the
// shared-memory data path 68 %; about a fifth of the pipe's 111 M instructions are no multiply-adds (they make operand pairs,
// among other things), but scalar multiply-adds are slower still (issue slots).
#include <string>

#include "mbarrier.cuh"

namespace sessd {

namespace {

constexpr int F32_WARPS = 12;                // warps that multiply; the next one streams the weights
constexpr int F32_THREADS = 512;             // all of them make the lists and write the rows
constexpr int F32_KVOL_MAX = 27;
constexpr int F32_UNIT = 16;                 // rows of a register tile
constexpr int F32_RT = F32_UNIT / 4;         // rows per thread
constexpr int F32_STRIP = 8;                 // rows that are dealt out together (of one tile)
constexpr int F32_FEW_FRAMES = 8;            // up to here a strip's frame is looked for frame by frame

template <int CIN, int COUT>
struct F32Shared {
    static constexpr int STAGES = CIN * COUT > 2048 ? 3 : (CIN * COUT > 1024 ? 4 : 8);   // weight ring
    static constexpr int ROWS = COUT == 64 ? (CIN == 64 ? 192 : 256) : (CIN == 64 ? 256 : 384);
    static constexpr int STRIPS = ROWS / F32_STRIP;
    float w[STAGES][CIN * COUT];
    float x[F32_WARPS][2][F32_UNIT * CIN];           // input rows of a warp's current and next unit
    float sum[ROWS * COUT];                          // channel c of row r at c ^ swizzle(r)
    uint32_t idx[F32_KVOL_MAX][ROWS];                // per offset: the input rows (of the whole batch) ..
    uint16_t row[F32_KVOL_MAX][ROWS];                // .. and the block's rows that have them
    int strip_frame[STRIPS], strip_row[STRIPS], strip_rows[STRIPS];   // of the present round
    uint32_t strip_mask[STRIPS];                     // offsets of the strip's tile
    int count[F32_KVOL_MAX + 1];                     // entries of an offset's list
    unsigned long long full[STAGES];
    int added[F32_KVOL_MAX + 1];                     // its units that have been added
    unsigned long long done[F32_KVOL_MAX];           // all of them have been: a phase per round
    int strips;                                      // of the whole call
    int abort_flag, abort_where;                     // (mbar_wait expects them in this order)
    static __device__ __forceinline__ int swizzle(int r) { return (r & (COUT / 16 - 1)) << 4; }
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
    int maps_ready, withhold_weights;   // withhold_weights: tests of the time-out path only
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
    const int n = f < a.batch ? load_late(a.out_num + f) : 0;
    return n > a.max_voxels ? a.max_voxels : (n < 0 ? 0 : n);
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(F32_THREADS, 1) conv_f32_kernel(const __grid_constant__ F32Args a) {
    using S = F32Shared<CIN, COUT>;
    constexpr int STAGES = S::STAGES, ROWS = S::ROWS, RT = F32_RT;
    constexpr int NP = COUT / 16;                    // channel pairs per thread: channels 16 p + 2 cg, + 1
    constexpr int CPR = CIN / 4;                     // 16-byte pieces of an input row
    constexpr uint32_t W_BYTES = CIN * COUT * 4;
    extern __shared__ __align__(128) uint8_t f32_smem[];
    S& s = *reinterpret_cast<S*>(f32_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rg = lane & 3, cg = lane >> 2;         // row group and channel group of the lane
    volatile int* abort_flag = &s.abort_flag;
    // maps, masks and row counts are older than the preceding kernel where maps_ready says so
    bool waited = false;
    if (!a.maps_ready) {
        pdl_enter();
        waited = true;
    }
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) mbar_init(smem_u32(&s.full[i]), 1);              // the streamer's expect
        for (int k = 0; k < F32_KVOL_MAX; ++k) mbar_init(smem_u32(&s.done[k]), 1);        // whoever adds the last unit
        s.abort_flag = s.abort_where = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        int strips = 0;
#pragma unroll 8
        for (int f = lane; f < a.batch; f += 32) strips += (f32_frame_rows(a, f) + F32_STRIP - 1) / F32_STRIP;
        strips = __reduce_add_sync(0xFFFFFFFFu, strips);
        if (lane == 0) s.strips = strips;
    }
    __syncthreads();
    // rounds of equal size, none larger than ROWS rows
    const int strips = s.strips, grid = (int)gridDim.x;
    const int rounds = (strips + grid * S::STRIPS - 1) / (grid * S::STRIPS);
    const int per_round = rounds > 0 ? (strips + grid * rounds - 1) / (grid * rounds) : 0;   // strips of a block
    const int rows_here = per_round * F32_STRIP;
    const int tiles_per_frame = (a.max_voxels + 127) / 128;
    int at_frame = 0, at_strip = 0;                  // where the look-up of the present round's strips starts, and the strips before
    uint32_t used = 0;                               // weight blocks of the rounds so far
    uint32_t issued = 0;                             // weight streamer: blocks whose copy has been started
    for (int round = 0; round < rounds; ++round) {
        __syncthreads();                             // the previous round has been written out
        if (*abort_flag) break;
        // the block's strips: numbered frame by frame, dealt out block by block
        if (warp < S::STRIPS / 32 + (S::STRIPS % 32 ? 1 : 0)) {
            const int i = warp * 32 + lane;
            const int want = i < per_round ? (round * per_round + i) * grid + (int)blockIdx.x : INT32_MAX;
            int frame = 0, row0 = 0, rows = 0;
            if (a.batch <= F32_FEW_FRAMES) {
                const int n = f32_frame_rows(a, lane);
                int before = 0;
                for (int f = 0; f < a.batch; ++f) {
                    const int nf = __shfl_sync(0xFFFFFFFFu, n, f), mine = (nf + F32_STRIP - 1) / F32_STRIP;
                    if (want >= before && want - before < mine)
                        frame = f, row0 = (want - before) * F32_STRIP, rows = min(nf - row0, F32_STRIP);
                    before += mine;
                }
            } else if (warp * 32 < per_round) {
                // 32 frames at a time, from where the round before found its last strip. (All frames one after the other, in every
                // round: calls of 4,096 frames of 200 rows 4427 us, now 1381 (32 -> 32), and 8811 and 2697 (64 -> 64).)
                const int last = __shfl_sync(0xFFFFFFFFu, want, min(per_round - warp * 32, 32) - 1);
                int ahead = f32_frame_rows(a, at_frame + lane);
                for (;;) {
                    const int n = ahead, mine = (n + F32_STRIP - 1) / F32_STRIP;
                    ahead = f32_frame_rows(a, at_frame + 32 + lane);
                    int start = mine;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int v = __shfl_up_sync(0xFFFFFFFFu, start, d);
                        if (lane >= d) start += v;
                    }
                    const int end = at_strip + __shfl_sync(0xFFFFFFFFu, start, 31);
                    start += at_strip - mine;
                    int src = 0;                     // the last of the frames that starts at or before the strip
#pragma unroll
                    for (int d = 16; d; d >>= 1)
                        if (__shfl_sync(0xFFFFFFFFu, start, src + d) <= want) src += d;
                    const int from = __shfl_sync(0xFFFFFFFFu, start, src), nf = __shfl_sync(0xFFFFFFFFu, n, src);
                    if (want >= at_strip && want < end)
                        frame = at_frame + src, row0 = (want - from) * F32_STRIP, rows = min(nf - row0, F32_STRIP);
                    if (last < end || at_frame + 32 >= a.batch) break;
                    at_frame += 32, at_strip = end;
                }
            }
            if (i < S::STRIPS) {
                s.strip_frame[i] = frame, s.strip_row[i] = row0, s.strip_rows[i] = rows;
                s.strip_mask[i] = rows > 0 ? __ldg(a.tile_mask + (size_t)frame * tiles_per_frame + (row0 >> 7)) : 0u;
            }
        }
        for (int e = tid; e < per_round * F32_STRIP * COUT / 4; e += F32_THREADS)
            reinterpret_cast<float4*>(s.sum)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        // lists: a warp per offset, all of its reads in flight
        for (int k = warp; k < F32_KVOL_MAX; k += F32_THREADS / 32) {
            int v[ROWS / 32];
#pragma unroll
            for (int j = 0; j < ROWS / 32; ++j) {
                const int r = j * 32 + lane, i = r / F32_STRIP, o = r % F32_STRIP;
                v[j] = -1;
                if (k < a.kvol && r < rows_here && o < s.strip_rows[i] && ((s.strip_mask[i] >> k) & 1u)) {
                    const int e = __ldg(a.nbr + nbr_index(a.kvol, a.max_voxels, s.strip_frame[i], k, s.strip_row[i] + o));
                    if (e >= 0) v[j] = s.strip_frame[i] * a.max_voxels + e;
                }
            }
            int n = 0;
#pragma unroll
            for (int j = 0; j < ROWS / 32; ++j) {
                const uint32_t votes = __ballot_sync(0xFFFFFFFFu, v[j] >= 0);
                if (v[j] >= 0) {
                    const int at = n + __popc(votes & ((1u << lane) - 1u));
                    s.idx[k][at] = (uint32_t)v[j];
                    s.row[k][at] = (uint16_t)(j * 32 + lane);
                }
                n += __popc(votes);
            }
            if (lane == 0) {
                s.count[k] = n;
                s.added[k] = 0;
                if (n == 0) mbar_arrive(smem_u32(&s.done[k]));
            }
        }
        if (!waited) {
            pdl_enter();
            waited = true;
        }
        __syncthreads();
        // lane k: units of offset k and of those before it
        const int units = lane < F32_KVOL_MAX ? (s.count[lane] + F32_UNIT - 1) / F32_UNIT : 0;
        const uint32_t present = __ballot_sync(0xFFFFFFFFu, units > 0);
        int first = units;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(0xFFFFFFFFu, first, d);
            if (lane >= d) first += v;
        }
        const int total = __shfl_sync(0xFFFFFFFFu, first, 31);
        first -= units;
        auto nth = [&](int q) {                      // the q-th present offset
            uint32_t m = present;
            for (int i = 0; i < q; ++i) m &= m - 1u;
            return __ffs((int)m) - 1;
        };

        if (warp == F32_WARPS) {
            // ---- weight streamer ----
            uint32_t m = a.withhold_weights ? 0u : present, old = present;   // old: the offset whose block a stage held
            for (int q = 0; m; m &= m - 1u, ++q) {
                const uint32_t at = used + (uint32_t)q, st = at % STAGES;
                if (q >= STAGES) {
                    const int k = __ffs((int)old) - 1;
                    old &= old - 1u;
                    const bool ok = mbar_wait(smem_u32(&s.done[k]), (uint32_t)round & 1u, abort_flag, 9 | (int)(at << 4));
                    if (!__all_sync(0xFFFFFFFFu, ok)) break;
                }
                if (lane == 0) {
                    mbar_arrive_expect_tx(smem_u32(&s.full[st]), W_BYTES);
                    bulk_load(smem_u32(s.w[st]), a.weights + (size_t)(__ffs((int)m) - 1) * CIN * COUT, W_BYTES, smem_u32(&s.full[st]));
                }
                issued = at + 1u;
            }
        } else if (warp < F32_WARPS) {
            // ---- units ----
            // copy of a unit's input rows: piece c of row r lands at piece c ^ (r / RT), so that the four row groups read different
            // banks; rows past the list's end keep what an earlier copy left (their sums are not used)
            auto fetch = [&](int u, float* dst) {
                const int k = __popc(__ballot_sync(0xFFFFFFFFu, lane < F32_KVOL_MAX && u >= first)) - 1;
                const int at = (u - __shfl_sync(0xFFFFFFFFu, first, k)) * F32_UNIT, n = s.count[k] - at;
#pragma unroll
                for (int r0 = 0; r0 < F32_UNIT; r0 += 4) {
                    const int r = r0 + (lane >> 3);
                    if (r < n) {
                        const float* src = a.in + (size_t)s.idx[k][at + r] * CIN;
#pragma unroll
                        for (int c = 0; c < CPR; c += 8)
                            copy_16(dst + r * CIN + (((c + (lane & 7)) ^ (r / RT)) * 4), src + (c + (lane & 7)) * 4);
                    }
                }
            };
            int buf = 0;
            if (warp < total) fetch(warp, s.x[warp][0]);
            asm volatile("cp.async.commit_group;" ::: "memory");
            bool ok = true;
            for (int u = warp; u < total; u += F32_WARPS, buf ^= 1) {
                const int k = __popc(__ballot_sync(0xFFFFFFFFu, lane < F32_KVOL_MAX && u >= first)) - 1;
                const int at = (u - __shfl_sync(0xFFFFFFFFu, first, k)) * F32_UNIT;
                const int q = __popc(present & ((1u << k) - 1u));
                if (u + F32_WARPS < total) fetch(u + F32_WARPS, s.x[warp][buf ^ 1]);
                asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
                __syncwarp();
                const uint32_t st = (used + (uint32_t)q) % STAGES;
                // a stage's barrier may be asked for its phase once the phase before is over, whoever saw that
                if (q >= STAGES) {
                    ok = mbar_wait(smem_u32(&s.done[nth(q - STAGES)]), (uint32_t)round & 1u, abort_flag, 10 | (int)(u << 4));
                    ok = __all_sync(0xFFFFFFFFu, ok);
                    if (!ok) break;
                }
                ok = mbar_wait(smem_u32(&s.full[st]), ((used + (uint32_t)q) / STAGES) & 1u, abort_flag, 10 | (int)(u << 4));
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) break;
                const float* x = s.x[warp][buf] + rg * RT * CIN;
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
                // all sums under the offset before have been added (which waited for the one before that)
                if (q > 0) {
                    const int kp = 31 - __clz((int)(present & ((1u << k) - 1u)));
                    ok = mbar_wait(smem_u32(&s.done[kp]), (uint32_t)round & 1u, abort_flag, 11 | (int)(u << 4));
                    ok = __all_sync(0xFFFFFFFFu, ok);
                    if (!ok) break;
                }
                const int n = s.count[k] - at;
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    if (rg * RT + i >= n) continue;
                    const int r = s.row[k][at + rg * RT + i];
                    float* acc = s.sum + r * COUT;
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        float2* to = reinterpret_cast<float2*>(acc + ((p * 16 + cg * 2) ^ S::swizzle(r)));
                        const float2 v = *to, t = unpair(sum[i][p]);
                        *to = make_float2(__fadd_rn(v.x, t.x), __fadd_rn(v.y, t.y));
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    __threadfence_block();
                    if (atomicAdd(&s.added[k], 1) == (s.count[k] + F32_UNIT - 1) / F32_UNIT - 1) {
                        __threadfence_block();
                        mbar_arrive(smem_u32(&s.done[k]));
                    }
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        used += (uint32_t)__popc(present);
        __syncthreads();
        if (*abort_flag) break;
        // folded batch norm and ReLU
        for (int e = tid; e < rows_here * (COUT / 4); e += F32_THREADS) {
            const int r = e / (COUT / 4), c = e % (COUT / 4) * 4, i = r / F32_STRIP, o = r % F32_STRIP;
            if (o >= s.strip_rows[i]) continue;
            const int b = s.strip_frame[i];
            const size_t pos = (size_t)b * a.max_voxels + s.strip_row[i] + o;
            const size_t row = a.order ? (size_t)b * a.max_voxels + __ldg(a.order + pos) : pos;
            float4 v = *reinterpret_cast<const float4*>(s.sum + r * COUT + (c ^ S::swizzle(r)));
            if (a.scale) {
                const float4 sc = __ldg(reinterpret_cast<const float4*>(a.scale + c));
                const float4 sh = a.shift ? __ldg(reinterpret_cast<const float4*>(a.shift + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
                v = make_float4(fmaf(v.x, sc.x, sh.x), fmaf(v.y, sc.y, sh.y), fmaf(v.z, sc.z, sh.z), fmaf(v.w, sc.w, sh.w));
            }
            if (a.relu) v = make_float4(v.x > 0.f ? v.x : 0.f, v.y > 0.f ? v.y : 0.f, v.z > 0.f ? v.z : 0.f, v.w > 0.f ? v.w : 0.f);
            *reinterpret_cast<float4*>(a.out + row * COUT + c) = v;
            if (a.dense) {
                // fused BEV scatter (sparse2Dense.cu:201-206): channel c*D + z, pixel (y, x)
                const int4 c4 = __ldg(&a.out_coors[row]);
                const size_t plane = (size_t)a.D * a.H * a.W;
                float* d = a.dense + (size_t)b * COUT * plane + ((size_t)c4.y * a.H + c4.z) * a.W + c4.w + c * plane;
                d[0] = v.x, d[plane] = v.y, d[2 * plane] = v.z, d[3 * plane] = v.w;
            }
        }
    }
    if (!waited) pdl_enter();                        // every block waits: the next kernel counts on what came before this one
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

template <int CIN, int COUT>
int launch_one(const ConvLaunch& c, cudaStream_t stream) {
    static const std::string name = "conv_f32<" + std::to_string(CIN) + "," + std::to_string(COUT) + ">";
    constexpr int smem = (int)sizeof(F32Shared<CIN, COUT>);
    static_assert(smem <= 227 * 1024, "a block does not fit the shared memory of one SM");
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
                    static_cast<float*>(c.dense), reinterpret_cast<const int4*>(c.out_coors), c.D, c.H, c.W, c.status, c.maps_ready,
                    c.debug_withhold_weights};
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
