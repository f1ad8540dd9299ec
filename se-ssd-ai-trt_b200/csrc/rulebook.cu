// Rulebook construction for submanifold and strided sparse convolutions.
//
// The reference builds, in every plugin call, a dense index grid (up to 369 MB, reset with
// cudaMemset), a candidate list per voxel and an input-stationary pair list per kernel offset
// (submConv3dlayer.cu:271-459, sparseConv3dlayer.cu:310-555). Here the rulebook is kept in
// output-stationary form: nbr[b][k][o] = input row that feeds output row o through kernel offset k,
// or -1. Pair (k, i, o) of the reference exists exactly when nbr[b][k][o] == i, because
// k = in - out*stride + pad per axis (submConv3dlayer.cu:328-329) and input rows are unique.
// nbr[b][k][o] names the entry; in memory the map is tile-major (nbr_index in common.cuh: the offsets of a
// 128-row tile side by side), so that the tensor-core kernel fetches a tile's offsets with one copy.
//
// Where the rows of a frame come from decides how a coordinate is turned back into its row:
//   - the voxeliser's rows (full resolution, 92 M cells, 80 K of them active) sit in an x-grouped
//     open-addressing table (32-byte buckets of four x-neighbours);
//   - the rows a strided layer produces are numbered through an occupancy grid of the output level: one
//     bit per cell, 64 x-neighbours per word, each word followed by the number of rows before it. Every
//     candidate output of every input row sets its bit (sparseConv3dlayer.cu:310-386 with the truncating
//     divisions kept); a count and a scan/emit pass then number the set bits in (z, y, x) order and write
//     the output coordinates. A cell's row is prefix + popcount(bits below), one 16-byte read, and the
//     three x-neighbours of a 3x3x3 kernel share that read. The grids are small (3 MB per frame at half
//     resolution, 0.4 MB at quarter resolution) and stay in L2. The reference numbers outputs in the
//     arrival order of an atomic over a dense scan (sparseConv3dlayer.cu:529-541); (z, y, x) order is
//     deterministic and keeps the rows of a 128-row tile close together in space;
//   - coordinates handed in by a caller (the stand-alone plugin entry points) go into a flat table.
#include "fill.cuh"
#include "rulebook.cuh"
#include "scan.cuh"

namespace sessd {

namespace {

__global__ void __launch_bounds__(kThreads)
table_build_kernel(const int4* __restrict__ coors, const int32_t* __restrict__ voxel_num, int batch, int max_voxels,
                   int Z, int Y, int X, Table t, int32_t* status) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int i = (it - b * chunks) * kThreads + threadIdx.x;
        int n = voxel_num[b];
        n = n > max_voxels ? max_voxels : n;
        if (i >= n) continue;
        const int4 c = __ldg(&coors[(size_t)b * max_voxels + i]);  // (b, z, y, x)
        if (c.y < 0 || c.y >= Z || c.z < 0 || c.z >= Y || c.w < 0 || c.w >= X) {
            atomicOr(status, SESSD_STATUS_BAD_COORD);
            continue;
        }
        const uint32_t key = ((uint32_t)c.y * Y + c.z) * X + c.w;
        const int slot = table_insert(t.keys + (size_t)b * t.cap, t.cap, t.shift, key);
        if (slot < 0) {
            atomicOr(status, SESSD_STATUS_HASH_FULL);
            continue;
        }
        // Duplicate coordinates (the reference's grid keeps whichever write lands last,
        // submConv3dlayer.cu:457) resolve to the highest row here.
        atomicMax(&t.vals[(size_t)b * t.cap + slot], i);
    }
}

// One thread per (offset k, output row o); threads of a warp share k and walk consecutive rows, so
// the writes to nbr[b][k][*] are coalesced.
__global__ void __launch_bounds__(kThreads)
nbr_build_kernel(const int4* __restrict__ out_coors, const int32_t* __restrict__ out_num, int batch, int max_voxels,
                 ConvGeom g, Table in_table, int32_t* __restrict__ nbr) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * g.kvol * chunks;
    const int k12 = g.K[1] * g.K[2];
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / (g.kvol * chunks);
        const int r = it - b * (g.kvol * chunks);
        const int k = r / chunks;
        const int o = (r - k * chunks) * kThreads + threadIdx.x;
        int n = out_num[b];
        n = n > max_voxels ? max_voxels : n;
        if (o >= n) continue;
        const int4 c = __ldg(&out_coors[(size_t)b * max_voxels + o]);
        const int kz = k / k12, ky = (k - kz * k12) / g.K[2], kx = k - kz * k12 - ky * g.K[2];
        // in = out*stride - pad + k*dilation (inverse of the offset formula at submConv3dlayer.cu:328)
        const int iz = c.y * g.S[0] - g.P[0] + kz * g.dil;
        const int iy = c.z * g.S[1] - g.P[1] + ky * g.dil;
        const int ix = c.w * g.S[2] - g.P[2] + kx * g.dil;
        int row = -1;
        if (iz >= 0 && iz < g.in_shape[0] && iy >= 0 && iy < g.in_shape[1] && ix >= 0 && ix < g.in_shape[2]) {
            const uint32_t key = ((uint32_t)iz * g.in_shape[1] + iy) * g.in_shape[2] + ix;
            const int slot = table_find(in_table.keys + (size_t)b * in_table.cap, in_table.cap, in_table.shift, key);
            if (slot >= 0) row = in_table.vals[(size_t)b * in_table.cap + slot];
        }
        nbr[nbr_index(g.kvol, max_voxels, b, k, o)] = row;
    }
}

// One block per kernel offset: compacts nbr[frame][k][*] into the reference's pair columns.
__global__ void __launch_bounds__(kThreads)
rulebook_export_kernel(const int32_t* __restrict__ nbr, const int32_t* __restrict__ out_num, int frame, int kvol,
                       int max_voxels, int32_t* __restrict__ pairs, uint32_t* __restrict__ pair_num) {
    pdl_enter();
    const int k = blockIdx.x;
    int n = out_num[frame];
    n = n > max_voxels ? max_voxels : n;
    const int32_t* col = nbr + nbr_index(kvol, max_voxels, frame, k, 0);   // entry o of the column: col[(o >> 7) * kvol * kNbrRun + (o & 127)]
    int32_t* pin = pairs + ((size_t)k * 2 + 0) * max_voxels;
    int32_t* pout = pairs + ((size_t)k * 2 + 1) * max_voxels;
    int base = 0;
    for (int o0 = 0; o0 < n; o0 += kThreads) {
        const int o = o0 + threadIdx.x;
        const int v = o < n ? col[(size_t)(o >> 7) * kvol * kNbrRun + (o & 127)] : -1;
        int total;
        const int pos = base + block_exclusive_scan(v >= 0 ? 1 : 0, &total);
        if (v >= 0) {
            pin[pos] = v;
            pout[pos] = o;
        }
        base += total;
    }
    if (threadIdx.x == 0) pair_num[k] = (uint32_t)base;
}

// Number of present neighbours (= rulebook pairs) of one layer, added to *total.
__global__ void __launch_bounds__(kThreads)
count_pairs_kernel(const int32_t* __restrict__ nbr, const int32_t* __restrict__ out_num, int batch, int max_voxels,
                   int kvol, unsigned long long* total) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * kvol * chunks;
    int local = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / (kvol * chunks);
        const int r = it - b * (kvol * chunks);
        const int k = r / chunks;
        const int o = (r - k * chunks) * kThreads + threadIdx.x;
        int n = out_num[b];
        n = n > max_voxels ? max_voxels : n;
        if (o < n && nbr[nbr_index(kvol, max_voxels, b, k, o)] >= 0) ++local;
    }
    const int sum = block_sum(local);
    if (threadIdx.x == 0 && sum) atomicAdd(total, (unsigned long long)sum);
}

// ---- x-grouped coordinate table ---------------------------------------------------------------
// A bucket is one 32-byte sector: the rows of the 4 cells that share (z, y, x >> 2), then the group
// key. The three x-neighbours of a cell lie in at most two buckets, so a 3x3x3 neighbourhood costs 9-18
// sector reads instead of 27 probes of a flat table.

__global__ void __launch_bounds__(kThreads)
bucket_build_kernel(const int4* __restrict__ coors, const int32_t* __restrict__ voxel_num, int batch, int max_voxels,
                    int Z, int Y, int X, Buckets t, int32_t* status) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int i = (it - b * chunks) * kThreads + threadIdx.x;
        int n = voxel_num[b];
        n = n > max_voxels ? max_voxels : n;
        if (i >= n) continue;
        const int4 c = __ldg(&coors[(size_t)b * max_voxels + i]);
        if (c.y < 0 || c.y >= Z || c.z < 0 || c.z >= Y || c.w < 0 || c.w >= X) {
            atomicOr(status, SESSD_STATUS_BAD_COORD);
            continue;
        }
        const uint32_t key = ((uint32_t)c.y * Y + c.z) * X + c.w;
        if (!bucket_insert(t.data + (size_t)b * t.cap * 8, t.cap, t.shift, key, i)) atomicOr(status, SESSD_STATUS_HASH_FULL);
    }
}

__device__ __forceinline__ int pick4(const int4& v, uint32_t i) {
    return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

// First probe of a bucket lookup, kept apart from its evaluation so that a thread can have the probes of
// several lookups in flight at once (the kernel below is bound by dependent round trips to L2, not by bytes).
struct BucketProbe {
    uint4 lo, hi;
    uint32_t h;
};
__device__ __forceinline__ void bucket_probe(const uint32_t* __restrict__ base, int shift, uint32_t gkey, bool on,
                                             BucketProbe* p) {
    p->h = hash_slot(gkey, shift);
    p->hi = make_uint4(kEmpty, 0u, 0u, 0u);
    p->lo = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (on) {
        // the whole 32-byte bucket with one 256-bit load (one request to L1 instead of two)
        const uint32_t* bk = base + (size_t)p->h * 8;
        asm volatile("ld.global.nc.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(p->lo.x), "=r"(p->lo.y), "=r"(p->lo.z), "=r"(p->lo.w), "=r"(p->hi.x), "=r"(p->hi.y),
                       "=r"(p->hi.z), "=r"(p->hi.w)
                     : "l"(bk));
    }
}
__device__ __forceinline__ int4 bucket_finish(const uint32_t* __restrict__ base, uint32_t cap, uint32_t gkey,
                                              const BucketProbe& p) {
    if (p.hi.x == gkey) return make_int4((int)p.lo.x, (int)p.lo.y, (int)p.lo.z, (int)p.lo.w);
    int4 none = make_int4(-1, -1, -1, -1);
    if (p.hi.x == kEmpty) return none;
    uint32_t h = (p.h + 1) & (cap - 1);   // first slot taken by another group: keep probing
    for (uint32_t probe = 1; probe < cap; ++probe) {
        const uint4* bk = reinterpret_cast<const uint4*>(base + (size_t)h * 8);
        const uint4 hi = __ldg(bk + 1);
        const uint4 lo = __ldg(bk);
        if (hi.x == gkey) return make_int4((int)lo.x, (int)lo.y, (int)lo.z, (int)lo.w);
        if (hi.x == kEmpty) return none;
        h = (h + 1) & (cap - 1);
    }
    return none;
}

// Submanifold 3x3x3 neighbour map. One thread per output row: it reads its coordinates once and, for each
// kz, has the bucket probes of the three ky rows (one or two 32-byte buckets each) in flight together,
// then writes nbr[b][k][o] for the nine offsets of that kz. Threads of a warp cover 32 consecutive rows of
// one 128-row tile, so the writes are coalesced and the per-tile offset mask (which offsets have any
// neighbour) costs one ballot per offset and one atomic per warp.
__global__ void __launch_bounds__(kThreads, 4)
nbr_build_subm_kernel(const int4* __restrict__ coors, const int32_t* __restrict__ voxel_num, int batch,
                      int max_voxels, int Z, int Y, int X, Buckets t, int32_t* __restrict__ nbr,
                      uint32_t* __restrict__ tile_mask, int tiles_per_frame) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int o0 = (it - b * chunks) * kThreads;
        int n = voxel_num[b];
        n = n > max_voxels ? max_voxels : n;
        if (o0 >= n) continue;
        const int o = o0 + threadIdx.x;
        const bool live = o < n;
        int4 c = make_int4(0, -4, -4, -4);
        if (live) c = __ldg(&coors[(size_t)b * max_voxels + o]);
        const int x = c.w;
        const bool x_ok = live && x >= 0 && x < X;
        const uint32_t* base = t.data + (size_t)b * t.cap * 8;
        int32_t* out = nbr + nbr_index(27, max_voxels, b, 0, o);
        uint32_t bits = 0;
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
            const int z = c.y + kz - 1;
            BucketProbe pa[3], pb[3];
            uint32_t center[3], g_lo[3], g_hi[3];
            bool on[3];
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                const int y = c.z + ky - 1;
                on[ky] = x_ok && z >= 0 && z < Z && y >= 0 && y < Y;
                center[ky] = on[ky] ? ((uint32_t)z * Y + y) * X + x : 0u;
                g_lo[ky] = (x > 0 ? center[ky] - 1 : center[ky]) >> 2;
                g_hi[ky] = (x + 1 < X ? center[ky] + 1 : center[ky]) >> 2;
                bucket_probe(base, t.shift, g_lo[ky], on[ky], &pa[ky]);
                bucket_probe(base, t.shift, g_hi[ky], on[ky] && g_hi[ky] != g_lo[ky], &pb[ky]);
            }
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                int res[3] = {-1, -1, -1};
                if (on[ky]) {
                    const int4 va = bucket_finish(base, t.cap, g_lo[ky], pa[ky]);
                    const int4 vb = g_hi[ky] != g_lo[ky] ? bucket_finish(base, t.cap, g_hi[ky], pb[ky]) : va;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const int xx = x + d - 1;
                        if (xx < 0 || xx >= X) continue;
                        const uint32_t key = center[ky] + d - 1;
                        res[d] = pick4((key >> 2) == g_lo[ky] ? va : vb, key & 3u);
                    }
                }
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int k = (kz * 3 + ky) * 3 + d;
                    if (live) out[k * kNbrRun] = res[d];
                    if (__ballot_sync(0xFFFFFFFFu, res[d] >= 0)) bits |= 1u << k;
                }
            }
        }
        if ((threadIdx.x & 31) == 0 && bits && live)
            atomicOr(&tile_mask[(size_t)b * tiles_per_frame + (o >> 7)], bits);
    }
}

// ---- occupancy grids -----------------------------------------------------------------------------

// Marks the candidate outputs of every input row, one thread per row.
__global__ void __launch_bounds__(kThreads)
mark_outputs_kernel(const int4* __restrict__ in_coors, const int32_t* __restrict__ in_num, int batch, int max_voxels,
                    ConvGeom g, BitGrid out) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int i = (it - b * chunks) * kThreads + threadIdx.x;
        int n = in_num[b];
        n = n > max_voxels ? max_voxels : n;
        if (i >= n) continue;
        mark_row(__ldg(&in_coors[(size_t)b * max_voxels + i]), b, g, out);
    }
}

// The even bits of v, packed into the low half.
__device__ __forceinline__ uint32_t even_bits(unsigned long long v) {
    v &= 0x5555555555555555ull;
    v = (v | (v >> 1)) & 0x3333333333333333ull;
    v = (v | (v >> 2)) & 0x0F0F0F0F0F0F0F0Full;
    v = (v | (v >> 4)) & 0x00FF00FF00FF00FFull;
    v = (v | (v >> 8)) & 0x0000FFFF0000FFFFull;
    return (uint32_t)(v | (v >> 16));
}

// Output cells of word w of an output level from the occupancy of its input level: a cell is an output when any cell of
// its receptive field is occupied, which is the set that marking every input row's candidates gives (the truncating
// divisions of sparseConv3dlayer.cu:339-348 drop no valid candidate). In x the two cases of derivable_in_x; z and y are
// free. The input words of all lines are read side by side and ORed before the bits are spread.
__device__ __forceinline__ unsigned long long derive_word(const BitGrid& in, const BitGrid& out, const ConvGeom& g, int b, int w) {
    const int row = w / out.xw, wx = w - row * out.xw;
    const int z = row / out.Y, y = row - z * out.Y;
    const bool same = g.K[2] == 1;                  // kernel 1, stride 1: the word itself; else kernel 3, stride 2, padding 1
    const int first = same ? wx : 2 * wx;
    unsigned long long before = 0ull, lo = 0ull, hi = 0ull;
#pragma unroll
    for (int kz = 0; kz < 3; ++kz) {
        const int iz = z * g.S[0] - g.P[0] + kz;
        if (kz >= g.K[0] || iz < 0 || iz >= in.Z) continue;
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            const int iy = y * g.S[1] - g.P[1] + ky;
            if (ky >= g.K[1] || iy < 0 || iy >= in.Y) continue;
            const int line = (iz * in.Y + iy) * in.xw;
            if (in.top) {
                // the three words' occupancy first: they are nearly always empty
                const int w0 = same ? line + first : (first > 0 ? line + first - 1 : line + first);
                const int w1 = same ? w0 : (first + 1 < in.xw ? line + first + 1 : line + first);
                const uint4* top = in.top + (size_t)b * in.top_words;
                const uint4 t0 = __ldg(top + (w0 >> 6));
                const uint4 t1 = (w1 >> 6) != (w0 >> 6) ? __ldg(top + (w1 >> 6)) : t0;
                for (int v = w0; v <= w1; ++v) {
                    const uint4& t = (v >> 6) == (w0 >> 6) ? t0 : t1;
                    const unsigned long long tb = rec_bits(t), bit = 1ull << (v & 63);
                    if (!(tb & bit)) continue;
                    const unsigned long long word =
                        rec_bits(__ldg(in.rec + (size_t)b * in.words + (int)t.z + __popcll(tb & (bit - 1ull))));
                    if (v == line + first) lo |= word;
                    else if (v < line + first) before |= word;
                    else hi |= word;
                }
                continue;
            }
            // a record is 16 bytes: bits first
            const unsigned long long* at =
                reinterpret_cast<const unsigned long long*>(in.rec + (size_t)b * in.words) + 2 * (size_t)line;
            if (first < in.xw) lo |= __ldg(at + 2 * first);
            if (!same) {
                if (first > 0) before |= __ldg(at + 2 * (first - 1));
                if (first + 1 < in.xw) hi |= __ldg(at + 2 * (first + 1));
            }
        }
    }
    unsigned long long bits = lo;
    if (!same) {
        // output x has the inputs 2x - 1, 2x, 2x + 1
        const unsigned long long even = (unsigned long long)even_bits(lo) | (unsigned long long)even_bits(hi) << 32;
        const unsigned long long odd = (unsigned long long)even_bits(lo >> 1) | (unsigned long long)even_bits(hi >> 1) << 32;
        bits = even | odd | (odd << 1) | (before >> 63);
    }
    const int x0 = wx << 6;
    if (x0 + 64 > out.X) bits &= x0 < out.X ? (1ull << (out.X - x0)) - 1ull : 0ull;   // cells past the line's end
    return bits;
}

// Numbers the occupied cells of every frame's output level in word order (= (z, y, x) order): completes the records
// (bits, rows before the word), writes the output coordinates (sparseConv3dlayer.cu:436-441 writes them per pair) and the
// frame's row count. The bits come from the records (marked by an earlier kernel) or, with DERIVE, from the input
// level's records; then the grid needs no reset either. Rows past max_voxels are dropped (their bits too, so that the
// next level does not see them) and reported. One thread per word; a warp then writes its words' coordinates one word
// at a time, a lane per cell. Two kernels (count, then prefix and emit with a serial loop over a thread's bits) took 3.5 +
// 18 us per level of a 20,000-point frame.
template <bool DERIVE>
__global__ void __launch_bounds__(kThreads)
number_outputs_kernel(BitGrid g, BitGrid in, ConvGeom geom, int batch, int max_voxels, ScanState scan,
                      int4* __restrict__ out_coors, int32_t* __restrict__ out_num, int32_t* status) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int chunks = scan_chunks(g.words), items = batch * chunks;
    for (int t = scan_ticket(scan.ticket, items); t >= 0; t = scan_ticket(scan.ticket, items)) {
        const int c = t / batch, b = t - c * batch;
        const int w = c * kThreads + threadIdx.x;
        uint4* rec = g.rec + (size_t)b * g.words;
        unsigned long long bits = 0ull;
        if (w < g.words) bits = DERIVE ? derive_word(in, g, geom, b, w) : rec_bits(rec[w]);
        int end;
        const int id = scan_position(scan.state + (size_t)b * chunks, c, __popcll(bits), &end, status);
        if (c == chunks - 1 && threadIdx.x == 0) {
            out_num[b] = end > max_voxels ? max_voxels : end;
            if (end > max_voxels) atomicOr(status, SESSD_STATUS_VOXEL_OVERFLOW);
        }
        if (id + __popcll(bits) > max_voxels) {          // keep the first max_voxels - id cells
            int keep = max_voxels - id > 0 ? max_voxels - id : 0;
            unsigned long long kept = 0ull;
            for (unsigned long long rem = bits; rem && keep; --keep) {
                kept |= rem & (0ull - rem);
                rem &= rem - 1ull;
            }
            bits = kept;
        }
        if (w < g.words) rec[w] = make_uint4((uint32_t)bits, (uint32_t)(bits >> 32), (uint32_t)id, 0u);
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, bits != 0ull); todo; todo &= todo - 1u) {
            const int src = __ffs((int)todo) - 1;
            const unsigned long long v = __shfl_sync(0xFFFFFFFFu, bits, src);
            const int id0 = __shfl_sync(0xFFFFFFFFu, id, src);
            const int word = w - lane + src;
            const int row = word / g.xw;                 // z * Y + y
            const int x0 = (word - row * g.xw) << 6;
            const int z = row / g.Y, y = row - z * g.Y;
            int4* dst = out_coors + (size_t)b * max_voxels + id0;
            const uint32_t v_lo = (uint32_t)v, v_hi = (uint32_t)(v >> 32), below = (1u << lane) - 1u;
            if ((v_lo >> lane) & 1u) dst[__popc(v_lo & below)] = make_int4(b, z, y, x0 + lane);
            if ((v_hi >> lane) & 1u) dst[__popc(v_lo) + __popc(v_hi & below)] = make_int4(b, z, y, x0 + 32 + lane);
        }
    }
}

// Rows of up to three x-neighbours (x0, x0+1, x0+2; `count` of them) of one (z, y) line of the input level.
struct BitsIndex {
    BitGrid g;
    int max_rows;
    struct Probe { uint4 a, b; int w; bool two; };
    // Record of word `line + w` of a two-level grid, given its top record; empty (with the right number of rows before
    // it left open) when the word is.
    __device__ __forceinline__ uint4 word_record(int b, int word, const uint4& t) const {
        const unsigned long long tb = rec_bits(t), bit = 1ull << (word & 63);
        if (!(tb & bit)) return make_uint4(0u, 0u, 0u, 0u);
        return __ldg(g.rec + (size_t)b * g.words + (int)t.z + __popcll(tb & (bit - 1ull)));
    }
    // First reads of a line's probe (the top records of a two-level grid), then the records themselves: kept apart so
    // that a thread has the reads of several lines in flight.
    __device__ __forceinline__ void probe_top(int b, int z, int y, int x0, int count, bool on, Probe* p) const {
        p->a = p->b = make_uint4(0u, 0u, 0u, 0u);
        p->two = false;
        p->w = -1;
        if (!on) return;
        const int lo = x0 < 0 ? 0 : x0, hi = x0 + count - 1 >= g.X ? g.X - 1 : x0 + count - 1;
        if (lo > hi) return;
        p->w = lo >> 6;
        p->two = (hi >> 6) != p->w;
        if (!g.top) return;
        const int word = (z * g.Y + y) * g.xw + p->w;
        p->a = __ldg(g.top + (size_t)b * g.top_words + (word >> 6));
        if (p->two) p->b = __ldg(g.top + (size_t)b * g.top_words + ((word + 1) >> 6));
    }
    __device__ __forceinline__ void probe_rec(int b, int z, int y, Probe* p) const {
        if (p->w < 0) return;
        const int word = (z * g.Y + y) * g.xw + p->w;
        if (g.top) {
            p->a = word_record(b, word, p->a);
            if (p->two) p->b = word_record(b, word + 1, p->b);
            if (rec_bits(p->a) == 0ull) p->a.z = p->b.z;   // the rows of the window are then all of the second word
        } else {
            const uint4* rec = g.rec + (size_t)b * g.words + word;
            p->a = __ldg(rec);
            if (p->two) p->b = __ldg(rec + 1);
        }
    }
    __device__ __forceinline__ void probe(int b, int z, int y, int x0, int count, bool on, Probe* p) const {
        probe_top(b, z, y, x0, count, on, p);
        probe_rec(b, z, y, p);
    }
    __device__ __forceinline__ int finish(const Probe& p, int x) const {
        if (x < 0 || x >= g.X) return -1;
        const uint4& r = (x >> 6) == p.w ? p.a : p.b;
        if ((x >> 6) != p.w && !p.two) return -1;
        const unsigned long long bits = rec_bits(r);
        const int bit = x & 63;
        if (!((bits >> bit) & 1ull)) return -1;
        const int id = (int)r.z + __popcll(bits & ((1ull << bit) - 1ull));
        return id < max_rows ? id : -1;
    }
    // The rows of the cells x0 .. x0 + count - 1 (count <= 3) of a probed line at once: the cells are neighbouring
    // bits of a window that may straddle two records, and rows are numbered along the line, so the row of a set
    // cell is the row of the window's first cell plus the set cells before it.
    __device__ __forceinline__ void finish_line(const Probe& p, int x0, int count, int (&rows)[3]) const {
        const int lo = x0 < 0 ? 0 : x0;
        const int sh = lo & 63;
        const unsigned long long a = rec_bits(p.a), b = p.two ? rec_bits(p.b) : 0ull;
        const unsigned long long window = sh ? (a >> sh) | (b << (64 - sh)) : a;
        const int base = (int)p.a.z + __popcll(a & ((1ull << sh) - 1ull));
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int x = x0 + e, pos = x - lo;
            int row = -1;
            if (e < count && x >= 0 && x < g.X && ((window >> pos) & 1ull)) {
                const int id = base + __popcll(window & ((1ull << pos) - 1ull));
                row = id < max_rows ? id : -1;
            }
            rows[e] = row;
        }
    }
};

// Neighbour maps of layers whose input level has an occupancy grid: one thread per output row walks the
// K0 x K1 lines of its receptive field, has the grid reads of a kz plane in flight together, and writes
// nbr[b][k][o] (coalesced over o) plus the per-128-row-tile offset mask (one ballot per offset, one atomic
// per warp). in = out*stride - pad + k, the inverse of the offset formula at submConv3dlayer.cu:328.
// All layers of a call go in one launch (the maps depend on coordinates only): on a 20,000-point frame six launches of
// 6 to 10 us each kept a fraction of the SMs busy.
__global__ void __launch_bounds__(kThreads, 4)
map_rows_kernel(const __grid_constant__ MapJobs jobs, int batch, int max_voxels, int tiles_per_frame) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int per_job = batch * chunks, items = per_job * jobs.count;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int j = it / per_job;
        const MapJob& job = jobs.job[j];
        const ConvGeom& g = job.g;
        const BitsIndex in{job.in, max_voxels};
        const int K0 = g.K[0], K1 = g.K[1], K2 = g.K[2];
        const int4* out_coors = reinterpret_cast<const int4*>(job.out_coors);
        int32_t* nbr = job.nbr;
        const int b = (it - j * per_job) / chunks;
        const int o0 = (it - j * per_job - b * chunks) * kThreads;
        int n = __ldg(job.out_num + b);
        n = n > max_voxels ? max_voxels : n;
        if (o0 >= n) continue;
        const int o = o0 + threadIdx.x;
        const bool live = o < n;
        int4 c = make_int4(0, 0, 0, 0);
        if (live) c = __ldg(&out_coors[(size_t)b * max_voxels + o]);
        const int bz = c.y * g.S[0] - g.P[0], by = c.z * g.S[1] - g.P[1], bx = c.w * g.S[2] - g.P[2];
        int32_t* out = nbr + nbr_index(g.kvol, max_voxels, b, 0, o);
        uint32_t bits = 0;
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
            if (kz >= K0) break;
            const int z = bz + kz;
            const bool z_ok = live && z >= 0 && z < g.in_shape[0];
            BitsIndex::Probe pb[3];
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                if (ky >= K1) break;
                const int y = by + ky;
                in.probe_top(b, z, y, bx, K2, z_ok && y >= 0 && y < g.in_shape[1], &pb[ky]);
            }
#pragma unroll
            for (int ky = 0; ky < 3; ++ky)
                if (ky < K1) in.probe_rec(b, z, by + ky, &pb[ky]);
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                if (ky >= K1) break;
                const int y = by + ky;
                const bool on = z_ok && y >= 0 && y < g.in_shape[1];
                int rows3[3] = {-1, -1, -1};
                if (on) in.finish_line(pb[ky], bx, K2, rows3);
#pragma unroll
                for (int kx = 0; kx < 3; ++kx) {
                    if (kx >= K2) break;
                    const int row = rows3[kx];
                    const int k = (kz * K1 + ky) * K2 + kx;
                    if (live) out[k * kNbrRun] = row;
                    if (__ballot_sync(0xFFFFFFFFu, row >= 0)) bits |= 1u << k;
                }
            }
        }
        if ((threadIdx.x & 31) == 0 && bits && live)
            atomicOr(&job.tile_mask[(size_t)b * tiles_per_frame + (o >> 7)], bits);
    }
}

// Fills the map entries of the tiles that hold rows 0 .. out_num[b] with -1, one int4 per thread (a tile's block of
// kvol x kNbrRun words is contiguous and 16-byte aligned; the padding words are written too), and zeroes the tails of
// the call's outputs, whose row counts are known by now.
__global__ void __launch_bounds__(kThreads)
nbr_clear_kernel(int32_t* __restrict__ nbr, const int32_t* __restrict__ out_num, int batch, int max_voxels, int kvol,
                 TailRows tails) {
    pdl_enter();
    zero_tails(tails);
    const size_t frame_words = nbr_frame_words(kvol, max_voxels);
    const int chunks = (int)((frame_words / 4 + kThreads - 1) / kThreads);
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        int n = out_num[b];
        n = n > max_voxels ? max_voxels : n;
        const size_t used_words = (size_t)((n + 127) / 128) * kvol * kNbrRun;   // a multiple of 4
        const size_t w = ((size_t)(it - b * chunks) * kThreads + threadIdx.x) * 4;
        if (w >= used_words) continue;
        *reinterpret_cast<int4*>(nbr + (size_t)b * frame_words + w) = make_int4(-1, -1, -1, -1);
    }
}

// Neighbour map of a strided layer whose input rows have no occupancy grid (the voxeliser's rows, or rows handed
// in by a caller): input-stationary. Thread = (input row i, candidate e) as in mark_outputs_kernel; the candidate's
// row in the numbered output grid is one read, and the pair lands as nbr[b][k][out] = i with
// k = in - out*stride + pad per axis (sparseConv3dlayer.cu:366). Each (k, out) has at most one input, so the
// writes never collide. The map must hold -1 for rows < out_num beforehand.
__global__ void __launch_bounds__(kThreads)
scatter_rows_kernel(const int4* __restrict__ in_coors, const int32_t* __restrict__ in_num, int batch, int max_voxels,
                    ConvGeom g, BitsIndex out, int32_t* __restrict__ nbr, uint32_t* __restrict__ tile_mask,
                    int tiles_per_frame) {
    pdl_enter();
    const int64_t per_frame = (int64_t)max_voxels * g.ncand;
    const int chunks = (int)((per_frame + kThreads - 1) / kThreads);
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int t = (it - b * chunks) * kThreads + threadIdx.x;
        int n = in_num[b];
        n = n > max_voxels ? max_voxels : n;
        if ((it - b * chunks) * kThreads >= n * g.ncand) continue;   // uniform over the block
        if (t >= n * g.ncand) continue;
        const int i = g.cand_shift >= 0 ? (t >> g.cand_shift) : t / g.ncand;
        const int e = t - i * g.ncand;
        int cz, cy, cx, rest;
        split_small(e, g.span_max[2], &rest, &cx);
        split_small(rest, g.span_max[1], &cz, &cy);
        const int4 c4 = __ldg(&in_coors[(size_t)b * max_voxels + i]);
        const int c[3] = {c4.y, c4.z, c4.w};
        const int cj[3] = {cz, cy, cx};
        int o[3];
        bool ok = true;
        int k = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int lo = div_trunc(c[j] - (g.K[j] - 1) - 1 + g.S[j] + g.P[j], g.S[j]);
            const int hi = div_trunc(c[j] + g.P[j], g.S[j]);
            o[j] = hi - cj[j];
            const int kj = c[j] - o[j] * g.S[j] + g.P[j];
            ok = ok && cj[j] <= hi - lo && o[j] >= 0 && o[j] < g.out_shape[j] && kj >= 0 && kj < g.K[j] &&
                 c[j] >= 0 && c[j] < g.in_shape[j];
            k = k * g.K[j] + kj;
        }
        if (!ok) continue;
        BitsIndex::Probe p;
        out.probe(b, o[0], o[1], o[2], 1, true, &p);
        const int id = out.finish(p, o[2]);
        if (id < 0) continue;   // output dropped by the max_voxels cap
        nbr[nbr_index(g.kvol, max_voxels, b, k, id)] = i;
        uint32_t* m = &tile_mask[(size_t)b * tiles_per_frame + (id >> 7)];
        if (!((*reinterpret_cast<volatile uint32_t*>(m) >> k) & 1u)) atomicOr(m, 1u << k);
    }
}

// Generic variant of the tile mask for maps built by nbr_build_kernel: one warp per (tile, k).
__global__ void __launch_bounds__(kThreads)
tile_mask_kernel(const int32_t* __restrict__ nbr, const int32_t* __restrict__ out_num, int batch, int max_voxels,
                 int kvol, uint32_t* __restrict__ tile_mask, int tiles_per_frame) {
    pdl_enter();
    const int warps_per_block = kThreads / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t items = (int64_t)batch * tiles_per_frame * kvol;
    for (int64_t it = (int64_t)blockIdx.x * warps_per_block + w; it < items; it += (int64_t)gridDim.x * warps_per_block) {
        const int k = (int)(it % kvol);
        const int64_t bt = it / kvol;
        const int tile = (int)(bt % tiles_per_frame), b = (int)(bt / tiles_per_frame);
        int n = out_num[b];
        n = n > max_voxels ? max_voxels : n;
        bool any = false;
        for (int q = 0; q < 4; ++q) {
            const int o = tile * 128 + q * 32 + lane;
            if (o < n && nbr[nbr_index(kvol, max_voxels, b, k, o)] >= 0) any = true;
        }
        if (__ballot_sync(0xFFFFFFFFu, any) && lane == 0) atomicOr(&tile_mask[(size_t)b * tiles_per_frame + tile], 1u << k);
    }
}

}  // namespace

int launch_bucket_build(const int32_t* coors, const int32_t* voxel_num, int batch, int max_voxels, const int shape[3],
                        const Buckets& t, int32_t* status, cudaStream_t stream) {
    SESSD_LAUNCH(bucket_build_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(coors),
                 voxel_num, batch, max_voxels, shape[0], shape[1], shape[2], t, status);
    return SESSD_OK;
}

int launch_nbr_build_subm(const int32_t* coors, const int32_t* voxel_num, int batch, int max_voxels, const int shape[3],
                          const Buckets& t, int32_t* nbr, uint32_t* tile_mask, cudaStream_t stream) {
    SESSD_LAUNCH(nbr_build_subm_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(coors),
                 voxel_num, batch, max_voxels, shape[0], shape[1], shape[2], t, nbr, tile_mask,
                 (max_voxels + 127) / 128);
    return SESSD_OK;
}

int launch_tile_mask(const int32_t* nbr, const int32_t* out_num, int batch, int max_voxels, int kvol,
                     uint32_t* tile_mask, cudaStream_t stream) {
    SESSD_LAUNCH(tile_mask_kernel, persistent_grid(8), kThreads, 0, stream, nbr, out_num, batch, max_voxels, kvol,
                 tile_mask, (max_voxels + 127) / 128);
    return SESSD_OK;
}

int launch_count_pairs(const int32_t* nbr, const int32_t* out_num, int batch, int max_voxels, int kvol,
                       unsigned long long* total, cudaStream_t stream) {
    SESSD_LAUNCH(count_pairs_kernel, persistent_grid(8), kThreads, 0, stream, nbr, out_num, batch, max_voxels, kvol,
                 total);
    return SESSD_OK;
}

int conv_geom_from_params(const sessd_conv_params* p, ConvGeom* g) {
    for (int j = 0; j < 3; ++j) {
        g->K[j] = p->ksize[j];
        g->S[j] = p->subm ? 1 : p->stride[j];
        g->P[j] = p->padding[j];
        if (g->K[j] < 1 || g->K[j] > 3 || g->S[j] < 1 || g->S[j] > 3 || g->P[j] < 0 || g->P[j] > 2) return SESSD_ERR_PARAM;
    }
    g->dil = p->dilation < 1 ? 1 : p->dilation;
    if (g->dil != 1) return SESSD_ERR_UNSUPPORTED;  // the reference only ever passes 1 (se-ssd-ai-trt.cpp:704)
    g->out_shape[0] = p->out_shape_z; g->out_shape[1] = p->out_shape_y; g->out_shape[2] = p->out_shape_x;
    if (p->subm) {
        // SubM layers carry only out_shape in the reference (submConv3dlayer.cu:596-603).
        for (int j = 0; j < 3; ++j) g->in_shape[j] = g->out_shape[j];
    } else {
        g->in_shape[0] = p->spatial_shape_z; g->in_shape[1] = p->spatial_shape_y; g->in_shape[2] = p->spatial_shape_x;
    }
    g->kvol = g->K[0] * g->K[1] * g->K[2];
    g->ncand = 1;
    for (int j = 0; j < 3; ++j) {
        if (g->in_shape[j] < 1 || g->out_shape[j] < 1) return SESSD_ERR_PARAM;
        g->span_max[j] = (g->K[j] - 1) / g->S[j] + 1;
        g->ncand *= g->span_max[j];
    }
    g->cand_shift = -1;
    for (int sh = 0; sh < 6; ++sh)
        if (g->ncand == (1 << sh)) g->cand_shift = sh;
    const uint64_t vin = (uint64_t)g->in_shape[0] * g->in_shape[1] * g->in_shape[2];
    const uint64_t vout = (uint64_t)g->out_shape[0] * g->out_shape[1] * g->out_shape[2];
    if (vin >= 0xFFFFFFFFull || vout >= 0xFFFFFFFFull) return SESSD_ERR_PARAM;  // keys are 32-bit cell indices
    return SESSD_OK;
}

int launch_table_build(const int32_t* coors, const int32_t* voxel_num, int batch, int max_voxels, const int shape[3],
                       const Table& t, int32_t* status, cudaStream_t stream) {
    SESSD_LAUNCH(table_build_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(coors),
                 voxel_num, batch, max_voxels, shape[0], shape[1], shape[2], t, status);
    return SESSD_OK;
}

int launch_nbr_build(const int32_t* out_coors, const int32_t* out_num, int batch, int max_voxels, const ConvGeom& g,
                     const Table& in_table, int32_t* nbr, cudaStream_t stream) {
    SESSD_LAUNCH(nbr_build_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(out_coors),
                 out_num, batch, max_voxels, g, in_table, nbr);
    return SESSD_OK;
}

int launch_mark_outputs(const int32_t* in_coors, const int32_t* in_num, int batch, int max_voxels, const ConvGeom& g,
                        const BitGrid& out, cudaStream_t stream) {
    SESSD_LAUNCH(mark_outputs_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(in_coors),
                 in_num, batch, max_voxels, g, out);
    return SESSD_OK;
}

// Whether an output level's occupancy can be taken from its input level's grid word by word.
bool derivable_in_x(const ConvGeom& g) {
    return (g.K[2] == 3 && g.S[2] == 2 && g.P[2] == 1) || (g.K[2] == 1 && g.S[2] == 1 && g.P[2] == 0);
}

int launch_number_outputs(const BitGrid& out, const BitGrid* derive_from, const ConvGeom& g, int batch, int max_voxels,
                          const ScanState& scan, int32_t* out_coors, int32_t* out_num, int32_t* status,
                          cudaStream_t stream) {
    const int64_t items = (int64_t)batch * scan_chunks(out.words);
    const int grid = (int)(items < persistent_grid(8) ? items : persistent_grid(8));
    if (derive_from)
        SESSD_LAUNCH(number_outputs_kernel<true>, grid, kThreads, 0, stream, out, *derive_from, g, batch, max_voxels, scan,
                     reinterpret_cast<int4*>(out_coors), out_num, status);
    else
        SESSD_LAUNCH(number_outputs_kernel<false>, grid, kThreads, 0, stream, out, BitGrid{}, g, batch, max_voxels, scan,
                     reinterpret_cast<int4*>(out_coors), out_num, status);
    return SESSD_OK;
}

int launch_map_rows(const MapJobs& jobs, int batch, int max_voxels, cudaStream_t stream) {
    if (jobs.count == 0) return SESSD_OK;
    SESSD_LAUNCH(map_rows_kernel, persistent_grid(8), kThreads, 0, stream, jobs, batch, max_voxels, (max_voxels + 127) / 128);
    return SESSD_OK;
}

int launch_scatter_rows(const int32_t* in_coors, const int32_t* in_num, const int32_t* out_num, int batch,
                        int max_voxels, const ConvGeom& g, const BitGrid& out, int32_t* nbr, uint32_t* tile_mask,
                        const TailRows& tails, cudaStream_t stream) {
    SESSD_LAUNCH(nbr_clear_kernel, persistent_grid(8), kThreads, 0, stream, nbr, out_num, batch, max_voxels, g.kvol, tails);
    SESSD_LAUNCH(scatter_rows_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(in_coors),
                 in_num, batch, max_voxels, g, BitsIndex{out, max_voxels}, nbr, tile_mask, (max_voxels + 127) / 128);
    return SESSD_OK;
}

int launch_rulebook_export(const int32_t* nbr, const int32_t* out_num, int frame, int kvol, int max_voxels,
                           int32_t* pairs, uint32_t* pair_num, cudaStream_t stream) {
    SESSD_CUDA(cudaMemsetAsync(pairs, 0xFF, sizeof(int32_t) * 2 * (size_t)kvol * max_voxels, stream));
    SESSD_LAUNCH(rulebook_export_kernel, kvol, kThreads, 0, stream, nbr, out_num, frame, kvol, max_voxels, pairs,
                 pair_num);
    return SESSD_OK;
}

}  // namespace sessd
