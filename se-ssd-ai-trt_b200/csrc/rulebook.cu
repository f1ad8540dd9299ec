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
//   - the front end's own rows are numbered through an occupancy grid of their level, 64 x-neighbouring cells to a word, each
//     word followed by the number of rows before it: a cell's row is prefix + popcount(bits below), one 16-byte read that the
//     three x-neighbours of a 3x3x3 kernel share. The voxeliser's level (92 M cells, 80 K of them active) has a grid of two levels
//     (voxel_grid.cu), the derived ones (3 MB per frame at half resolution, 0.4 MB at quarter) one. A strided layer's
//     candidate outputs (sparseConv3dlayer.cu:310-386, truncating divisions kept) are set as bits; a one-pass scan (scan.cuh)
//     numbers them in (z, y, x) order and writes the output coordinates. The reference numbers outputs in the arrival
//     order of an atomic over a dense scan (sparseConv3dlayer.cu:529-541); (z, y, x) order is deterministic and keeps the
//     rows of a 128-row tile close together in space;
//   - rows in an order of their own (a caller's, or the voxeliser's where rows may have to be dropped) sit in an x-grouped
//     open-addressing table (32-byte buckets of four x-neighbours). Large strided calls on fine grids go without: their input rows
//     look up their outputs in the numbered grid (scatter_rows_kernel);
//   - submanifold kernels other than 3x3x3 use a flat table.
#include "fill.cuh"
#include "rulebook.cuh"
#include "scan.cuh"
#include "voxel.cuh"

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
        int n = load_late(voxel_num + b);
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
        int n = load_late(out_num + b);
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
        if (k == 0 && (o & 31) == 0) nbr[nbr_runs_index(g.kvol, max_voxels, b, o)] = -1;
    }
}

// One block per kernel offset: compacts nbr[frame][k][*] of a map in row order into the reference's pair columns, in ascending
// output row.
__global__ void __launch_bounds__(kThreads)
rulebook_export_kernel(const int32_t* __restrict__ nbr, const uint32_t* __restrict__ tile_mask,
                       const int32_t* __restrict__ out_num, int frame, int kvol, int max_voxels, int32_t* __restrict__ pairs,
                       uint32_t* __restrict__ pair_num) {
    pdl_enter();
    const int k = blockIdx.x;
    int n = load_late(out_num + frame);
    n = n > max_voxels ? max_voxels : n;
    const int32_t* col = nbr + nbr_index(kvol, max_voxels, frame, k, 0);   // entry o of the column: col[(o >> 7) * kvol * kNbrRun + (o & 127)]
    const uint32_t* mask = tile_mask + (size_t)frame * ((max_voxels + 127) / 128);
    int32_t* pin = pairs + ((size_t)k * 2 + 0) * max_voxels;
    int32_t* pout = pairs + ((size_t)k * 2 + 1) * max_voxels;
    int base = 0;
    for (int o0 = 0; o0 < n; o0 += kThreads) {
        const int o = o0 + threadIdx.x;
        const int v = o < n && (mask[o >> 7] >> k) & 1u ? col[(size_t)(o >> 7) * kvol * kNbrRun + (o & 127)] : -1;
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
count_pairs_kernel(const int32_t* __restrict__ nbr, const uint32_t* __restrict__ tile_mask,
                   const int32_t* __restrict__ out_num, int batch, int max_voxels, int kvol, unsigned long long* total) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads, tiles = (max_voxels + 127) / 128;
    const int items = batch * kvol * chunks;
    int local = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / (kvol * chunks);
        const int r = it - b * (kvol * chunks);
        const int k = r / chunks;
        const int p = (r - k * chunks) * kThreads + threadIdx.x;
        int n = load_late(out_num + b);
        n = n > max_voxels ? max_voxels : n;
        if (p < n && ((tile_mask[(size_t)b * tiles + (p >> 7)] >> k) & 1u) && nbr[nbr_index(kvol, max_voxels, b, k, p)] >= 0)
            ++local;
    }
    const int sum = block_sum(local);
    if (threadIdx.x == 0 && sum) atomicAdd(total, (unsigned long long)sum);
}

// ---- x-grouped coordinate table ---------------------------------------------------------------
// A bucket is one 32-byte sector: the rows of the 4 cells that share (z, y, x >> 2), then the group
// key. The three x-neighbours of a cell lie in at most two buckets, so a 3x3x3 neighbourhood costs 9-18
// sector reads instead of 27 probes of a flat table.

// Enters every row into the table. MARK (strided layers): also marks its candidate outputs; rows outside the grid are
// then skipped silently, as the reference's candidate enumeration does.
template <bool MARK>
__global__ void __launch_bounds__(kThreads)
bucket_build_kernel(const int4* __restrict__ coors, const int32_t* __restrict__ voxel_num, int batch, int max_voxels,
                    int Z, int Y, int X, Buckets t, ConvGeom g, BitGrid out, int32_t* status) {
    pdl_enter();
    const int chunks = (max_voxels + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int i = (it - b * chunks) * kThreads + threadIdx.x;
        int n = load_late(voxel_num + b);
        n = n > max_voxels ? max_voxels : n;
        if (i >= n) continue;
        const int4 c = __ldg(&coors[(size_t)b * max_voxels + i]);
        if (c.y < 0 || c.y >= Z || c.z < 0 || c.z >= Y || c.w < 0 || c.w >= X) {
            if (!MARK) atomicOr(status, SESSD_STATUS_BAD_COORD);
            continue;
        }
        if (MARK) mark_row(c, b, g, out);
        const uint32_t key = ((uint32_t)c.y * Y + c.z) * X + c.w;
        if (!bucket_insert(t.data + (size_t)b * t.cap * 8, t.cap, t.shift, key, i)) atomicOr(status, SESSD_STATUS_HASH_FULL);
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
        int n = load_late(in_num + b);
        n = n > max_voxels ? max_voxels : n;
        if (i >= n) continue;
        mark_row(__ldg(&in_coors[(size_t)b * max_voxels + i]), b, g, out);
    }
}

// ---- maps of strided layers by input rows ----------------------------------------------------------
// No table: every candidate output of an input row is looked up in the numbered output grid, and the pair lands as
// nbr[b][k][out] = row. Pays for large calls where the grid is fine (scatter_rows_usable): rows then have few neighbours and there are
// more outputs than inputs.

// Fills the map entries of the tiles that hold rows 0 .. out_num[b] with -1, 16 bytes per thread (a tile's kvol x kNbrRun words
// are contiguous; the padding is written too: any offset for every 32 rows), and zeroes the tails of the call's outputs.
__global__ void __launch_bounds__(kThreads)
nbr_clear_kernel(int32_t* __restrict__ nbr, const int32_t* __restrict__ out_num, int batch, int max_voxels, int kvol,
                 TailRows tails) {
    pdl_enter();
    zero_tails(tails);
    const size_t frame_words = nbr_frame_words(kvol, max_voxels);
    const int chunks = (int)((frame_words / 4 + kThreads - 1) / kThreads);
    const int64_t items = (int64_t)batch * chunks;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = (int)(it / chunks);
        const int n = min(load_late(out_num + b), max_voxels);
        const size_t w = ((size_t)(it - (int64_t)b * chunks) * kThreads + threadIdx.x) * 4;
        if (w < (size_t)((n + 127) / 128) * kvol * kNbrRun)
            *reinterpret_cast<int4*>(nbr + (size_t)b * frame_words + w) = make_int4(-1, -1, -1, -1);
    }
}

// Thread = (input row, candidate output) as in mark_row, k = in - out*stride + pad per axis (sparseConv3dlayer.cu:366). Rows of
// the same cell: the highest wins, as in a table.
__global__ void __launch_bounds__(kThreads)
scatter_rows_kernel(const int4* __restrict__ in_coors, const int32_t* __restrict__ in_num, int batch, int max_voxels,
                    ConvGeom g, BitGrid out, int32_t* __restrict__ nbr, uint32_t* __restrict__ tile_mask) {
    pdl_enter();
    const int tiles = (max_voxels + 127) / 128;
    const int chunks = (int)(((int64_t)max_voxels * g.ncand + kThreads - 1) / kThreads);
    const int64_t items = (int64_t)batch * chunks;
    for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = (int)(it / chunks);
        const int t = (int)(it - (int64_t)b * chunks) * kThreads + threadIdx.x;
        const int n = min(load_late(in_num + b), max_voxels);
        if (t >= n * g.ncand) continue;
        int i, e[3], rest;
        split_small(t, g.span_max[2], &rest, &e[2]);
        split_small(rest, g.span_max[1], &rest, &e[1]);
        split_small(rest, g.span_max[0], &i, &e[0]);
        const int4 c4 = __ldg(&in_coors[(size_t)b * max_voxels + i]);
        const int c[3] = {c4.y, c4.z, c4.w};
        int o[3], k = 0;
        bool ok = true;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int lo = div_trunc(c[j] - (g.K[j] - 1) - 1 + g.S[j] + g.P[j], g.S[j]);
            const int hi = div_trunc(c[j] + g.P[j], g.S[j]);
            o[j] = hi - e[j];
            const int kj = c[j] - o[j] * g.S[j] + g.P[j];
            ok = ok && e[j] <= hi - lo && o[j] >= 0 && o[j] < g.out_shape[j] && kj >= 0 && kj < g.K[j] && c[j] >= 0 &&
                 c[j] < g.in_shape[j];
            k = k * g.K[j] + kj;
        }
        if (!ok) continue;
        const uint4 r = __ldg(out.rec + (size_t)b * out.words + ((size_t)o[0] * out.Y + o[1]) * out.xw + (o[2] >> 6));
        const unsigned long long bits = rec_bits(r), bit = 1ull << (o[2] & 63);
        if (!(bits & bit)) continue;                     // dropped: past max_voxels
        const int row = (int)r.z + __popcll(bits & (bit - 1ull));
        atomicMax(nbr + nbr_index(g.kvol, max_voxels, b, k, row), i);
        uint32_t* m = tile_mask + (size_t)b * tiles + (row >> 7);
        if (!((*reinterpret_cast<volatile uint32_t*>(m) >> k) & 1u)) atomicOr(m, 1u << k);
    }
}

// Numbers one chunk (kThreads x WORDS words) of one frame of a level whose bits are set, in word order (= (z, y, x)
// order): completes the records (rows before the word), writes the output coordinates (sparseConv3dlayer.cu:436-441 writes
// them per pair) and, with the last chunk, the row count. Rows past max_voxels are dropped (their bits too, so that the
// next level does not see them; the record of a word that lost all of them gets kLostCells in its third word) and
// reported. before_chunk(total): rows before the chunk, which has `total`. Returns the running total with the chunk.
constexpr uint32_t kLostCells = 0x80000000u;
template <int WORDS, bool WRITE = true, class Before>
__device__ __forceinline__ int number_chunk(const BitGrid& g, int b, int c, int chunks, int max_voxels, int4* __restrict__ out_coors,
                                            int32_t* __restrict__ out_num, int32_t* status, Before before_chunk) {
    // word i of a thread: c * kThreads * WORDS + i * kThreads + threadIdx.x, so that a warp's words of a step are neighbours.
    // Counts of the steps travel through one block scan, 16 bits each (a step has at most 256 x 64 cells).
    static_assert(WORDS <= 4, "four steps to a 64-bit scan");
    __shared__ unsigned long long s_sum[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w0 = c * kThreads * WORDS + threadIdx.x;
    uint4* rec = g.rec + (size_t)b * g.words;
    unsigned long long bits[WORDS], mine = 0ull;
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
        const int w = w0 + i * kThreads;
        bits[i] = w < g.words ? rec_bits(rec[w]) : 0ull;
        mine |= (unsigned long long)__popcll(bits[i]) << (16 * i);
    }
    unsigned long long incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += t;
    }
    __syncthreads();                                     // s_sum has been read by the previous chunk
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    unsigned long long before = incl - mine, all = 0ull;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
        if (i < warp) before += s_sum[i];
        all += s_sum[i];
    }
    int total = 0;
#pragma unroll
    for (int i = 0; i < WORDS; ++i) total += (int)(all >> (16 * i) & 0xFFFFull);
    const int prefix = before_chunk(total), end = prefix + total;
    if (c == chunks - 1 && threadIdx.x == 0) {
        out_num[b] = end > max_voxels ? max_voxels : end;
        if (end > max_voxels) atomicOr(status, SESSD_STATUS_VOXEL_OVERFLOW);
    }
    int step0 = prefix;                                  // rows before the step
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
        const int w = w0 + i * kThreads;
        const int id = step0 + (int)(before >> (16 * i) & 0xFFFFull);
        step0 += (int)(all >> (16 * i) & 0xFFFFull);
        unsigned long long v = bits[i];
        uint32_t next = __shfl_down_sync(0xFFFFFFFFu, (uint32_t)v, 1);
        if (lane == 31 && w + 1 < g.words) next = rec[w + 1].x;
        next = next_cells(next, w, g, id + __popcll(v), max_voxels);
        if (id + __popcll(v) > max_voxels) {             // keep the first max_voxels - id cells
            int keep = max_voxels - id > 0 ? max_voxels - id : 0;
            unsigned long long kept = 0ull;
            for (; v && keep; --keep) {
                kept |= v & (0ull - v);
                v &= v - 1ull;
            }
            v = kept;
        }
        const uint32_t lost = v == 0ull && bits[i] != 0ull ? kLostCells : 0u;
        if (w < g.words) rec[w] = make_uint4((uint32_t)v, (uint32_t)(v >> 32), (uint32_t)id | lost, next);
        if (WRITE && __any_sync(0xFFFFFFFFu, v != 0ull))
            write_cells(out_coors + (size_t)b * max_voxels, b, g.xw, g.Y, w, v, min(id, max_voxels));
    }
    return end;
}

__global__ void __launch_bounds__(kThreads)
number_outputs_kernel(BitGrid g, int batch, int max_voxels, ScanState scan, int4* __restrict__ out_coors,
                      int32_t* __restrict__ out_num, int32_t* status) {
    const int chunks = scan_chunks(g.words), items = batch * chunks;
    int t = scan_first(scan.ticket, items);
    pdl_enter();
    for (; t >= 0; t = scan_next(scan.ticket, items, gridDim.x)) {
        const int c = t / batch, b = t - c * batch;
        number_chunk<1>(g, b, c, chunks, max_voxels, out_coors, out_num, status,
                        [&](int total) { return scan_prefix(scan.state + (size_t)b * chunks, c, total, status); });
    }
}

// Cells of word w of a level's grid that have an input cell in frame b's grid `in` of the level before: the marks of
// mark_levels, collected from the output's side. The words of the lines that a word's cells look at are OR-ed first; what x does
// to them (the layers of derivable_in_x) is the same for all.
__device__ __forceinline__ unsigned long long word_outputs(const BitGrid& in, const ConvGeom& geom, const BitGrid& g, int b, int w) {
    const int line = w / g.xw, wx = w - line * g.xw, z = line / g.Y;
    const int z0 = z * geom.S[0] - geom.P[0], y0 = (line - z * g.Y) * geom.S[1] - geom.P[1];
    const bool half = geom.K[2] == 3;                    // the word's cells lie over two words of `in`, and one cell before them
    const int w0 = half ? 2 * wx : wx;
    const uint4* rec = in.rec + (size_t)b * in.words;
    unsigned long long lo = 0ull, hi = 0ull, left = 0ull;
    for (int kz = 0; kz < geom.K[0]; ++kz) {
        if ((unsigned)(z0 + kz) >= (unsigned)in.Z) continue;
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            if (ky >= geom.K[1] || (unsigned)(y0 + ky) >= (unsigned)in.Y) continue;
            const uint4* at = rec + ((z0 + kz) * in.Y + y0 + ky) * in.xw + w0;
            if (w0 < in.xw) lo |= *reinterpret_cast<const unsigned long long*>(at);
            if (half && w0 + 1 < in.xw) hi |= *reinterpret_cast<const unsigned long long*>(at + 1);
            if (half && w0 > 0 && w0 <= in.xw) left |= *reinterpret_cast<const unsigned long long*>(at - 1) >> 63;
        }
    }
    if (half) {
        const unsigned long long odd = even_bits(lo >> 1) | (unsigned long long)even_bits(hi >> 1) << 32;
        lo = even_bits(lo) | (unsigned long long)even_bits(hi) << 32 | odd | odd << 1 | left;
    }
    const int cells = g.X - (wx << 6);
    return cells < 64 ? lo & ((1ull << cells) - 1ull) : lo;
}

// The levels below a level that had more rows than max_voxels must not see the rows it dropped: their cells are taken from the
// rows that are left, and numbered again. By one block, for a frame that has lost rows anyway, so that what counts is that few
// reads depend on one another: every row of the level before marking its outputs once more took 1.4 ms (one frame of 45,000 points
// in 60,000 rows: 1762 us, now 416; 20,000 points in 20,000 rows: 922 and 432).
__device__ __noinline__ void renumber_levels(const LevelChain& chain, int b, int l0, int max_voxels, int32_t* status) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto last_z = [&](int l) {                           // plane of the last row of a level that dropped some: they lie there or above
        return __ldcg(reinterpret_cast<const int4*>(chain.coors[l]) + (size_t)b * max_voxels + max_voxels - 1).y;
    };
    int z_in = last_z(l0 - 1);                           // first plane of the level before that may have changed
    for (int l = l0; l < chain.count; ++l) {
        const BitGrid &g = chain.grid[l], &in = chain.grid[l - 1];
        const ConvGeom& geom = chain.geom[l];
        uint4* rec = g.rec + (size_t)b * g.words;
        // planes below this one look at unchanged ones alone: their words and rows stay as they are
        const int z0 = (max(z_in + geom.P[0] - geom.K[0] + 1, 0) + geom.S[0] - 1) / geom.S[0];
        const int chunks = scan_chunks((g.words + 3) / 4), first = min(z0, g.Z) * g.Y * g.xw / (kThreads * 4) * (kThreads * 4);
        int rows = first < g.words ? (int)(rec[first].z & ~kLostCells) : __ldcg(chain.totals + b * LevelChain::kMax + l);
        // (words without a mark stay empty; marks that the first numbering removed have left kLostCells)
        for (int w0 = first + warp * 128; w0 < g.words; w0 += kThreads * 4) {   // 128 words to a warp, a lane to each that needs it
            unsigned long long todo[2] = {0ull, 0ull};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int w = w0 + i * 32 + lane;
                const uint4 r = w < g.words ? rec[w] : make_uint4(0u, 0u, 0u, 0u);
                const bool need = w < g.words && (r.x | r.y | (r.z & kLostCells)) != 0u;
                todo[i >> 1] |= (unsigned long long)__ballot_sync(0xFFFFFFFFu, need) << (32 * (i & 1));
            }
            const int n0 = __popcll(todo[0]), n = n0 + __popcll(todo[1]);
            for (int e = lane; e < n; e += 32) {
                const int w = w0 + (e < n0 ? nth_bit(todo[0], e) : 64 + nth_bit(todo[1], e - n0));
                *reinterpret_cast<unsigned long long*>(rec + w) = word_outputs(in, geom, g, b, w);
            }
        }
        __syncthreads();
        for (int c = first / (kThreads * 4); c < chunks; ++c)
            rows = number_chunk<4, false>(g, b, c, chunks, max_voxels, nullptr, chain.num[l], status, [&](int) { return rows; });
        __syncthreads();
        // the coordinates, by warps that need not wait for one another
        int4* coors = reinterpret_cast<int4*>(chain.coors[l]) + (size_t)b * max_voxels;
        auto fetch = [&](int w0) { return w0 + lane < g.words ? rec[w0 + lane] : make_uint4(0u, 0u, (uint32_t)rows, 0u); };
        uint4 next = fetch(first + warp * 32);
        for (int w0 = first + warp * 32; w0 < g.words; w0 += kThreads) {
            const uint4 r = next;
            next = fetch(w0 + kThreads);
            if (__any_sync(0xFFFFFFFFu, (r.x | r.y) != 0u))
                write_cells(coors, b, g.xw, g.Y, w0 + lane, rec_bits(r), min((int)(r.z & ~kLostCells), max_voxels));
        }
        __syncthreads();
        z_in = rows > max_voxels ? min(z0, last_z(l)) : z0;
    }
}

// All levels of a chain in one launch (blocks 0 .. number_blocks - 1), and beside it the point lists of the voxeliser's
// rows, which depend on the same kernel and on nothing here: by the other blocks, or where there are none by every block that
// finds no more chunks (both parts are chains of dependent reads; blocks of their own for the lists only start when a
// numbering block is through, and took two thirds of the kernel's 408 us on 32 frames x 120,000 points).
constexpr int kLevelBlocks = 6;
template <int WORDS>
__global__ void __launch_bounds__(kThreads, kLevelBlocks)   // (renumber_levels would take 104 registers; it may spill)
number_levels_kernel(const __grid_constant__ LevelChain chain, int batch, int max_voxels, int number_blocks, PointLists lists,
                     int32_t* status) {
    if ((int)blockIdx.x >= number_blocks) {
        pdl_enter();
        push_points(lists, batch, blockIdx.x - number_blocks, gridDim.x - number_blocks);
        return;
    }
    __shared__ int s_last;
    int per_frame = 0;
    for (int l = 0; l < chain.count; ++l) per_frame += scan_chunks((chain.grid[l].words + WORDS - 1) / WORDS);
    const int items = batch * per_frame;
    int t = scan_first(chain.ticket, items);
    pdl_enter();
    for (; t >= 0; t = scan_next(chain.ticket, items, number_blocks)) {
        const int b = t % batch;
        int c = t / batch, l = 0, chunks = 0;
        for (;; ++l) {
            chunks = scan_chunks((chain.grid[l].words + WORDS - 1) / WORDS);
            if (c < chunks) break;
            c -= chunks;
        }
        const int end = number_chunk<WORDS>(chain.grid[l], b, c, chunks, max_voxels, reinterpret_cast<int4*>(chain.coors[l]), chain.num[l],
                                            status, [&](int total) {
                                                return scan_prefix(chain.state[l] + (size_t)b * chunks, c, total, status);
                                            });
        if (c == chunks - 1 && threadIdx.x == 0) chain.totals[b * LevelChain::kMax + l] = end;
        // the frame's last block looks whether a level lost rows
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(chain.done + b, 1u) == (uint32_t)(per_frame - 1);
        __syncthreads();
        if (!s_last) continue;
        __threadfence();
        for (int k = 0; k + 1 < chain.count; ++k)
            if (__ldcg(chain.totals + b * LevelChain::kMax + k) > max_voxels) {
                renumber_levels(chain, b, k + 1, max_voxels, status);
                break;
            }
    }
    if (number_blocks == (int)gridDim.x) push_points(lists, batch, blockIdx.x, gridDim.x);
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
        int n = load_late(out_num + b);
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
                        const Buckets& t, const ConvGeom* mark, const BitGrid& out, int32_t* status, cudaStream_t stream) {
    const int4* c = reinterpret_cast<const int4*>(coors);
    if (mark)
        SESSD_LAUNCH(bucket_build_kernel<true>, persistent_grid(8), kThreads, 0, stream, c, voxel_num, batch, max_voxels,
                     shape[0], shape[1], shape[2], t, *mark, out, status);
    else
        SESSD_LAUNCH(bucket_build_kernel<false>, persistent_grid(8), kThreads, 0, stream, c, voxel_num, batch, max_voxels,
                     shape[0], shape[1], shape[2], t, ConvGeom{}, BitGrid{}, status);
    return SESSD_OK;
}

int launch_tile_mask(const int32_t* nbr, const int32_t* out_num, int batch, int max_voxels, int kvol,
                     uint32_t* tile_mask, cudaStream_t stream) {
    SESSD_LAUNCH(tile_mask_kernel, persistent_grid(8), kThreads, 0, stream, nbr, out_num, batch, max_voxels, kvol,
                 tile_mask, (max_voxels + 127) / 128);
    return SESSD_OK;
}

int launch_count_pairs(const int32_t* nbr, const uint32_t* tile_mask, const int32_t* out_num, int batch, int max_voxels, int kvol,
                       unsigned long long* total, cudaStream_t stream) {
    SESSD_LAUNCH(count_pairs_kernel, persistent_grid(8), kThreads, 0, stream, nbr, tile_mask, out_num, batch, max_voxels,
                 kvol, total);
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

// Fine grids: a row of the network's full resolution (92 M cells) has 3.4 candidate outputs and there are twice as many outputs as
// inputs, so that going by inputs touches less; one level down (12 M cells) there are fewer outputs than inputs, and a table is
// better at every size (by inputs and through a table, before a thread took a plane: 1 x 20,000 points 68 and 67 us, 1 x 120,000 142 and
// 96, 8 x 120,000 466 and 373). Small calls are latency, and the table's way is shorter (no clearing, no atomics on map entries); how
// many rows there are is on the device, so that the line is a capacity. Full resolution, by inputs and through a table: room for 60,000
// rows, 1 x 20,000 points 72.9 and 63.6; 200,000, 1 x 120,000 111 and 107; 240,000, 4 x 20,000 116 and 105; 400,000, 2 x 60,000
// 123 and 111; 480,000, 8 x 20,000 157 and 153; 600,000, 3 x 120,000 187 and 197; 960,000, 16 x 20,000 243 and 266.
// Between 200,000 and 500,000 the fill decides, which the host does not know. fp16 16 -> 32, room for half to four fifths (60,000 rows for
// 20,000 points, 200,000 for 120,000): 300,000 101 and 105, 360,000 119 and 115, 400,000 132 and 133, 480,000 136 and 135; room for
// hardly more than there is: 164,000 95 and 90, 205,000 102 and 111, 328,000 131 and 137, 410,000 152 and 169; room for five times as
// much: 400,000 89 and 67. The line is where the usual room breaks even.
bool scatter_rows_usable(const ConvGeom& g, int64_t rows) {
    return rows > 500000 && (uint64_t)g.in_shape[0] * g.in_shape[1] * g.in_shape[2] >= 1ull << 25;
}

int launch_scatter_rows(const int32_t* in_coors, const int32_t* in_num, const int32_t* out_num, int batch, int max_voxels,
                        const ConvGeom& g, const BitGrid& out, int32_t* nbr, uint32_t* tile_mask, const TailRows& tails,
                        cudaStream_t stream) {
    SESSD_LAUNCH(nbr_clear_kernel, persistent_grid(8), kThreads, 0, stream, nbr, out_num, batch, max_voxels, g.kvol, tails);
    SESSD_LAUNCH(scatter_rows_kernel, persistent_grid(8), kThreads, 0, stream, reinterpret_cast<const int4*>(in_coors), in_num,
                 batch, max_voxels, g, out, nbr, tile_mask);
    return SESSD_OK;
}

// Whether an output level's occupancy can be taken from its input level's grid word by word.
bool derivable_in_x(const ConvGeom& g) {
    return (g.K[2] == 3 && g.S[2] == 2 && g.P[2] == 1) || (g.K[2] == 1 && g.S[2] == 1 && g.P[2] == 0);
}

bool level_chain_usable(const ConvGeom* geoms, int count) {
    int halvings = 0;
    for (int l = 0; l < count; ++l) {
        if (!derivable_in_x(geoms[l])) return false;
        halvings += geoms[l].K[2] == 3 ? 1 : 0;
    }
    return count >= 1 && count <= LevelChain::kMax && halvings <= 6;   // a word's first cell stays even before each of them
}

int launch_number_outputs(const BitGrid& out, int batch, int max_voxels, const ScanState& scan, int32_t* out_coors,
                          int32_t* out_num, int32_t* status, cudaStream_t stream) {
    const int64_t items = (int64_t)batch * scan_chunks(out.words);
    const int grid = (int)(items < persistent_grid(8) ? items : persistent_grid(8));
    SESSD_LAUNCH(number_outputs_kernel, grid, kThreads, 0, stream, out, batch, max_voxels, scan,
                 reinterpret_cast<int4*>(out_coors), out_num, status);
    return SESSD_OK;
}

// As few words per thread (short chains) as let every chunk and the point lists have a resident block; else four, and
// rounds of a persistent grid. (One frame of the network's levels: 843 chunks of one word per thread took two waves of blocks, 22 us.)
int launch_number_levels(const LevelChain& chain, int batch, int max_voxels, const PointLists& lists, int32_t* status,
                         cudaStream_t stream) {
    const int resident = persistent_grid(kLevelBlocks);
    const int64_t point_chunks = (int64_t)batch * scan_chunks(lists.max_points);
    const int list_blocks = (int)(point_chunks < persistent_grid(2) ? point_chunks : persistent_grid(2));
    auto items = [&](int words) {
        int64_t n = 0;
        for (int l = 0; l < chain.count; ++l) n += (int64_t)batch * scan_chunks((chain.grid[l].words + words - 1) / words);
        return n;
    };
#define SESSD_LEVELS(WORDS, BLOCKS, LIST_BLOCKS)                                                                          \
    SESSD_LAUNCH(number_levels_kernel<WORDS>, (BLOCKS) + (LIST_BLOCKS), kThreads, 0, stream, chain, batch, max_voxels, (BLOCKS), \
                 lists, status)
    if (items(1) + list_blocks <= resident) {
        SESSD_LEVELS(1, (int)items(1), list_blocks);
    } else if (items(2) + list_blocks <= resident) {
        SESSD_LEVELS(2, (int)items(2), list_blocks);
    } else {
        SESSD_LEVELS(4, resident, 0);
    }
#undef SESSD_LEVELS
    return SESSD_OK;
}

int launch_rulebook_export(const int32_t* nbr, const uint32_t* tile_mask, const int32_t* out_num, int frame, int kvol,
                           int max_voxels, int32_t* pairs, uint32_t* pair_num, cudaStream_t stream) {
    SESSD_CUDA(cudaMemsetAsync(pairs, 0xFF, sizeof(int32_t) * 2 * (size_t)kvol * max_voxels, stream));
    SESSD_LAUNCH(rulebook_export_kernel, kvol, kThreads, 0, stream, nbr, tile_mask, out_num, frame, kvol, max_voxels,
                 pairs, pair_num);
    return SESSD_OK;
}

}  // namespace sessd
