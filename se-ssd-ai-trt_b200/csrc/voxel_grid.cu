// Point cloud -> voxels numbered in (z, y, x) order, for the fused front end.
//
// voxelize.cu numbers voxels by their first point, which is what the stand-alone voxeliser promises. Inside the front end
// nobody sees the order of the voxel rows, and (z, y, x) order is the better one: neighbouring rows are neighbouring
// cells, so the neighbour maps of the full-resolution layers, the gathers of their convolutions and the tiles of the
// tensor-core kernel all become coherent, and the level gets an occupancy grid like every other one, so that its maps are
// built like all others (no coordinate table, no input-stationary scatter, no clearing of a map).
//
// A full-resolution grid of a frame has 92 M cells and at most some 100,000 occupied ones, so the grid has two levels:
// a top record {bits lo, bits hi, words before} per 64 words of 64 x-neighbouring cells (0.36 MB per frame), and a
// record {bits lo, bits hi, rows before, word} per occupied word (at most one per point). Six passes:
//   1. every point finds its cell and sets its word's bit in the top level;
//   2. the words are numbered (one-pass scan) and their records cleared;
//   3. every point sets its cell's bit in its word;
//   4. the rows are numbered (one-pass scan): coordinates, row count, empty point lists; every word also marks the cells
//      that it reaches in the grids of all further levels, a few atomics for up to 64 cells;
//   5. (one launch with the numbering of the further levels) every point pushes its index through its row's ascending list of the max_points_per_voxel smallest indices (a
//      cascade of atomicMin, so the list does not depend on timing);
//   6. (one launch with the neighbour maps) every row averages its listed points, summed in ascending index order.
// What bounds it: the chain of dependent L2 reads of short kernels for one frame, the atomics of pass 5 and the random
// 16-byte point reads of pass 6 for a batch.
#include "rulebook.cuh"
#include "scan.cuh"
#include "voxel.cuh"

namespace sessd {

namespace {

// A point's key is word << 6 | bit of its cell, kEmpty outside the range.

__device__ __forceinline__ void set_bit(uint4* rec, int bit) {   // of a record's first 8 bytes
    unsigned long long* word = reinterpret_cast<unsigned long long*>(rec);
    const unsigned long long m = 1ull << bit;
    if (!(*reinterpret_cast<volatile unsigned long long*>(word) & m)) atomicOr(word, m);
}

__global__ void __launch_bounds__(kThreads)
point_mark_kernel(const float4* __restrict__ points, const int32_t* __restrict__ points_size, int batch, int max_points,
                  VoxGeom g, BitGrid grid, uint32_t* __restrict__ pt_key) {
    pdl_enter();
    for_points(points_size, batch, max_points, blockIdx.x, gridDim.x, [&](int b, int p) {
        const float4 pt = __ldg(&points[(size_t)b * max_points + p]);
        int ix, iy, iz;
        uint32_t key = kEmpty;
        if (voxel_cell(g, pt, &ix, &iy, &iz)) {
            const int word = (iz * grid.Y + iy) * grid.xw + (ix >> 6);
            key = (uint32_t)word << 6 | (uint32_t)(ix & 63);
            set_bit(grid.top + (size_t)b * grid.top_words + (word >> 6), word & 63);
        }
        pt_key[(size_t)b * max_points + p] = key;
    });
}

__global__ void __launch_bounds__(kThreads)
number_words_kernel(BitGrid grid, int batch, ScanState scan, int32_t* __restrict__ word_num, int32_t* status) {
    const int lane = threadIdx.x & 31;
    const int chunks = scan_chunks(grid.top_words), items = batch * chunks;
    int t = scan_first(scan.ticket, items);
    pdl_enter();
    for (; t >= 0; t = scan_next(scan.ticket, items, gridDim.x)) {
        const int c = t / batch, b = t - c * batch;
        const int w = c * kThreads + threadIdx.x;
        uint4* top = grid.top + (size_t)b * grid.top_words;
        const unsigned long long bits = w < grid.top_words ? rec_bits(top[w]) : 0ull;
        int end;
        const int id = scan_position(scan.state + (size_t)b * chunks, c, __popcll(bits), &end, status);
        if (c == chunks - 1 && threadIdx.x == 0) word_num[b] = end;
        if (w < grid.top_words) top[w].z = (uint32_t)id;
        uint4* rec = grid.rec + (size_t)b * grid.words;   // words never outnumber points, which grid.words allows for
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, bits != 0ull); todo; todo &= todo - 1u) {
            const int src = __ffs((int)todo) - 1;
            const unsigned long long v = __shfl_sync(0xFFFFFFFFu, bits, src);
            uint4* dst = rec + __shfl_sync(0xFFFFFFFFu, id, src);
            const uint32_t word = (uint32_t)(w - lane + src) << 6;
            const uint32_t v_lo = (uint32_t)v, v_hi = (uint32_t)(v >> 32), below = (1u << lane) - 1u;
            if ((v_lo >> lane) & 1u) dst[__popc(v_lo & below)] = make_uint4(0u, 0u, 0u, word + lane);
            if ((v_hi >> lane) & 1u) dst[__popc(v_lo) + __popc(v_hi & below)] = make_uint4(0u, 0u, 0u, word + 32 + lane);
        }
    }
}

__global__ void __launch_bounds__(kThreads)
point_bits_kernel(const int32_t* __restrict__ points_size, int batch, int max_points, BitGrid grid,
                  const uint32_t* __restrict__ pt_key) {
    pdl_enter();
    for_points(points_size, batch, max_points, blockIdx.x, gridDim.x, [&](int b, int p) {
        const uint32_t key = __ldg(pt_key + (size_t)b * max_points + p);
        if (key != kEmpty) set_bit(grid.rec + (size_t)b * grid.words + word_id(grid, b, key >> 6), key & 63);
    });
}

__global__ void __launch_bounds__(kThreads)
number_rows_kernel(BitGrid grid, const int32_t* __restrict__ word_num, int batch, int max_voxels, int max_points, int max_pts,
                   ScanState scan, int4* __restrict__ coors, int32_t* __restrict__ voxel_num,
                   uint32_t* __restrict__ lists, const __grid_constant__ LevelChain chain, int32_t* status) {
    const int lane = threadIdx.x & 31;
    const int chunks = scan_chunks(grid.words), items = batch * chunks;
    int t = scan_first(scan.ticket, items);
    pdl_enter();
    for (; t >= 0; t = scan_next(scan.ticket, items, gridDim.x)) {
        const int c = t / batch, b = t - c * batch;
        const int n = __ldg(word_num + b), used = n > 0 ? scan_chunks(n) : 1;
        if (c >= used) continue;                   // uniform over the block
        const int w = c * kThreads + threadIdx.x;
        uint4* rec = grid.rec + (size_t)b * grid.words;
        const uint4 r = w < n ? rec[w] : make_uint4(0u, 0u, 0u, 0u);
        const unsigned long long bits = rec_bits(r);
        const int cnt = __popcll(bits);
        int end;
        const int id = scan_position(scan.state + (size_t)b * chunks, c, cnt, &end, status);
        if (c == used - 1 && threadIdx.x == 0) voxel_num[b] = end;   // at most max_points rows, and those fit max_voxels
        if (w < n) rec[w].z = (uint32_t)id;
        if (w < n && chain.count) {
            const int row = (int)r.w / grid.xw;
            mark_levels(bits, row / grid.Y, row % grid.Y, (int)r.w - row * grid.xw, b, chain);
        }
        // the warp's rows are consecutive: their point lists in one run
        const int first = __shfl_sync(0xFFFFFFFFu, id, 0), last = __shfl_sync(0xFFFFFFFFu, id + cnt, 31);
        uint32_t* list = lists + (size_t)b * max_points * max_pts;
        for (int e = first * max_pts + lane; e < last * max_pts; e += 32) list[e] = kEmpty;
        if (first < last) write_cells(coors + (size_t)b * max_voxels, b, grid.xw, grid.Y, (int)r.w, bits, id);
    }
}

__global__ void __launch_bounds__(kThreads) point_list_kernel(PointLists lists, int batch) {
    pdl_enter();
    push_points(lists, batch, blockIdx.x, gridDim.x);
}

}  // namespace

bool voxel_grid_usable(const sessd_voxel_params* p, int max_points, const int level_shape[3]) {
    // Rows can be dropped only where there are more of them than max_voxels, and then the ones to keep are the first in
    // point order: with room for a row per point that cannot happen. Words are numbered with 26 bits.
    return max_points <= p->max_voxels &&
           (uint64_t)level_shape[0] * level_shape[1] * ((level_shape[2] + 63) / 64) < (1ull << 26);
}

void voxel_grid_layout(Bump& bump, const sessd_voxel_params* p, const int level_shape[3], int batch, int max_points,
                       VoxelGrid* w) {
    w->grid = bitgrid_shape(level_shape);
    w->grid.top_words = (w->grid.words + 63) / 64;
    if (w->grid.words > max_points) w->grid.words = max_points;   // records: one per occupied word
    w->grid.rec = bump.take<uint4>((size_t)batch * w->grid.words);
    w->pt_key = bump.take<uint32_t>((size_t)batch * max_points);
    w->lists = bump.take<uint32_t>((size_t)batch * max_points * p->max_points_per_voxel);
    w->word_num = bump.take<int32_t>(batch);
    // to be zero before a call
    const size_t top_bytes = (size_t)batch * w->grid.top_words * sizeof(uint4);
    const size_t words_bytes = scan_state_bytes(w->grid.top_words, batch), rows_bytes = scan_state_bytes(w->grid.words, batch);
    char* zero = bump.take<char>(top_bytes + words_bytes + rows_bytes);
    w->zero_base = zero;
    w->zero_bytes = top_bytes + words_bytes + rows_bytes;
    w->grid.top = reinterpret_cast<uint4*>(zero);
    w->scan_words = scan_state_at(zero ? zero + top_bytes : nullptr, w->grid.top_words, batch);
    w->scan_rows = scan_state_at(zero ? zero + top_bytes + words_bytes : nullptr, w->grid.words, batch);
}

int voxel_grid_run(const sessd_voxel_params* p, int batch, int max_points, const float* points, const int32_t* points_size,
                   int32_t* coors, int32_t* voxel_num, const VoxelGrid& w, const LevelChain& chain, int32_t* status,
                   cudaStream_t stream) {
    const VoxGeom g = voxel_geom(*p);
    const float4* pts = reinterpret_cast<const float4*>(points);
    const int max_pts = p->max_points_per_voxel;
    const int most = persistent_grid(8);
    auto blocks = [&](int entries) {
        const int64_t items = (int64_t)batch * scan_chunks(entries);
        return (int)(items < most ? items : most);
    };
    SESSD_LAUNCH(point_mark_kernel, blocks(max_points), kThreads, 0, stream, pts, points_size, batch, max_points, g, w.grid,
                 w.pt_key);
    SESSD_LAUNCH(number_words_kernel, blocks(w.grid.top_words), kThreads, 0, stream, w.grid, batch, w.scan_words, w.word_num,
                 status);
    SESSD_LAUNCH(point_bits_kernel, blocks(max_points), kThreads, 0, stream, points_size, batch, max_points, w.grid, w.pt_key);
    SESSD_LAUNCH(number_rows_kernel, blocks(w.grid.words), kThreads, 0, stream, w.grid, w.word_num, batch, p->max_voxels,
                 max_points, max_pts, w.scan_rows, reinterpret_cast<int4*>(coors), voxel_num, w.lists, chain, status);
    const PointLists lists{points_size, w.pt_key, w.lists, w.grid, max_points, max_pts};
    if (chain.count) return launch_number_levels(chain, batch, p->max_voxels, lists, status, stream);
    SESSD_LAUNCH(point_list_kernel, blocks(max_points), kThreads, 0, stream, lists, batch);
    return SESSD_OK;
}

}  // namespace sessd
