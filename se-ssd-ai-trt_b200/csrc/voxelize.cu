// Point cloud -> voxels with a mean voxel feature, for B independent frames per call.
//
// Replaces the reference's dense-grid voxeliser (voxelGenerator.cu:348-451, 255-321), which zeroes
// a 739 MB coordinate table every frame and lets a thread spin until another thread has published a
// voxel id. Here each frame owns a small open-addressing table keyed by the linear cell index:
//   pass 1 (insert)  every point claims its cell's slot, or finds the point that has and pushes its index through that
//                    one's ascending list of the max_points_per_voxel smallest other points (a cascade of atomicMin;
//                    which point claims a cell depends on timing, the cell's points do not);
//   pass 2 (emit)    the owner points (the smallest index of their cell) are numbered in point order with a
//                    one-pass scan (scan.cuh); the owner writes coordinates, count and the mean of the listed points,
//                    summed in ascending index order.
// Results are therefore bit-reproducible. A single frame is bound by the chain of dependent reads and launches, not by
// bytes: as seven launches (reset, insert, count, emit, three tails) 20,000 points took 46 us, as three 18. A batch is bound by
// the random accesses of pass 1: with the lists in the slots (24 or 32 bytes each) the table of 64 frames x 20,000 points
// did not fit L2 and the call took 133 - 136 us.
// The fused front end numbers its voxels in space instead where it can (voxel_grid.cu).
#include "fill.cuh"
#include "rulebook.cuh"
#include "scan.cuh"
#include "voxel.cuh"

namespace sessd {

namespace {

__global__ void __launch_bounds__(kThreads)
voxel_insert_kernel(const float4* __restrict__ points, const int32_t* __restrict__ points_size, int batch,
                    int max_points, VoxGeom g, VoxelTable t, int max_pts, int32_t* __restrict__ pt_claim,
                    int32_t* status) {
    pdl_enter();
    const int chunks = (max_points + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int b = it / chunks;
        const int p = (it - b * chunks) * kThreads + threadIdx.x;
        int n = points_size[b];
        n = n > max_points ? max_points : n;
        if (p >= n) continue;
        const float4 pt = __ldg(&points[(size_t)b * max_points + p]);
        int claim = -1;
        int ix, iy, iz;
        if (voxel_cell(g, pt, &ix, &iy, &iz)) {
            const uint32_t key = ((uint32_t)iz * g.gy + iy) * g.gx + ix;
            // Most cells have one point: a free slot takes it with one swap, made without looking first. A cell that meets another
            // goes on by a step of its own (odd, so that it comes round to every slot): the longest chain of swaps is what a small
            // call waits for, and to the next slot chains run together (64 x 20,000 points 79.7 us, so 77.3; 1 x 32,000 23.1 and 18.8. How
            // long the longest chain is depends on the frame: over eight frames in turn this kernel takes 9.7 and 8.9 us at
            // 1 x 20,000, 13.1 and 10.8 at 1 x 32,000, 13.2 and 12.0 at 1 x 120,000).
            unsigned long long* slots = t.slots + (size_t)b * t.cap;
            uint32_t h = hash_slot(key, t.shift);
            const uint32_t step = (key * 0x85EBCA6Bu >> 15) | 1u;   // (a multiplier of MurmurHash3's finaliser; any odd one that mixes)
            for (uint32_t probe = 0; probe < t.cap; ++probe, h = (h + step) & (t.cap - 1)) {
                const unsigned long long old = atomicCAS(slots + h, ~0ull, (unsigned long long)p << 32 | key);
                if (old != ~0ull && (uint32_t)old != key) continue;
                claim = old == ~0ull ? p : (int)(old >> 32);
                break;
            }
            if (claim < 0) atomicOr(status, SESSD_STATUS_HASH_FULL);
            else if (claim != p) list_push(t.lists + ((size_t)b * max_points + claim) * max_pts, max_pts, (uint32_t)p);
        }
        pt_claim[(size_t)b * max_points + p] = claim;
    }
}

template <typename T>
struct VoxelOut {
    T* voxels;
    int32_t* coors;
    int32_t* num_points;
    int32_t* voxel_num;
    int32_t* status;
    int max_voxels;
    int zero_tail;
};

// STEPS points per thread: point i of a thread is the chunk's point i * kThreads + threadIdx.x.
template <typename T, int STEPS>
__global__ void __launch_bounds__(kThreads, STEPS == 1 ? 5 : 4)
voxel_emit_kernel(const float4* __restrict__ points, const int32_t* __restrict__ points_size, int batch, int max_points,
                  VoxGeom g, VoxelTable t, int max_pts, const int32_t* __restrict__ pt_claim, ScanState scan, VoxelOut<T> out) {
    static_assert(STEPS <= 2 && kThreads < (1 << 16), "16 bits of a scan per step, two steps to a word");
    constexpr int CHUNK = kThreads * STEPS;
    __shared__ uint32_t s_sum[kThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunks = (max_points + CHUNK - 1) / CHUNK, items = batch * chunks;
    int ticket = scan_first(scan.ticket, items);
    pdl_enter();
    for (; ticket >= 0; ticket = scan_next(scan.ticket, items, gridDim.x)) {
        const int c = ticket / batch, b = ticket - c * batch;
        int n = points_size[b];
        n = n < 0 ? 0 : (n > max_points ? max_points : n);
        const int used = n > 0 ? (n + CHUNK - 1) / CHUNK : 1;
        if (c >= used) continue;                   // uniform over the block
        const int e0 = c * CHUNK + tid;
        const uint32_t* lists = t.lists + (size_t)b * max_points * max_pts;
        // a cell's points are the claiming one and those of its list: the first of them owns the cell
        int claim[STEPS];
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const int e = e0 + i * kThreads;
            claim[i] = e < n ? load_late(pt_claim + (size_t)b * max_points + e) : -1;
        }
        uint32_t owner = 0;                        // bit i
        uint32_t mine = 0u;                        // counts of the steps, 16 bits each
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const uint32_t head = claim[i] >= 0 ? lists[(size_t)claim[i] * max_pts] : kEmpty;
            const bool own = claim[i] >= 0 && min((uint32_t)claim[i], head) == (uint32_t)(e0 + i * kThreads);
            owner |= (own ? 1u : 0u) << i;
            mine |= (own ? 1u : 0u) << (16 * i);
        }
        uint32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += v;
        }
        if (lane == 31) s_sum[warp] = incl;        // (the ticket's barriers lie between this and the previous chunk's reads)
        __syncthreads();
        uint32_t before = incl - mine, all = 0u;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) {
            if (w < warp) before += s_sum[w];
            all += s_sum[w];
        }
        int total = 0;
#pragma unroll
        for (int i = 0; i < STEPS; ++i) total += (int)(all >> (16 * i) & 0xFFFFu);
        const int prefix = scan_prefix(scan.state + (size_t)b * chunks, c, total, out.status), end = prefix + total;
        if (c == used - 1 && tid == 0) {
            out.voxel_num[b] = end > out.max_voxels ? out.max_voxels : end;
            if (end > out.max_voxels) atomicOr(out.status, SESSD_STATUS_VOXEL_OVERFLOW);
        }
        int step0 = prefix;                        // owners before the step
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
            const int e = e0 + i * kThreads;
            const int id = step0 + (int)(before >> (16 * i) & 0xFFFFu);
            step0 += (int)(all >> (16 * i) & 0xFFFFu);
            if (!((owner >> i) & 1u)) {
                // The points that own no cell are as many as the rows between the voxel count and the point count: the
                // r-th of them zeroes the r-th of those rows from the end.
                const int row = n - 1 - (e - id);
                if (out.zero_tail && e < n && row < out.max_voxels) {
                    const size_t r = (size_t)b * out.max_voxels + row;
                    store_voxel(out.voxels, r, 0.f, 0.f, 0.f, 0.f);
                    reinterpret_cast<int4*>(out.coors)[r] = make_int4(0, 0, 0, 0);
                    out.num_points[r] = 0;
                }
                continue;
            }
            if (id >= out.max_voxels) continue;
            uint32_t pi[kMaxPointsPerVoxel];
            list_load(lists + (size_t)claim[i] * max_pts, max_pts, pi);
            uint32_t carry = (uint32_t)claim[i];
#pragma unroll
            for (int j = 0; j < kMaxPointsPerVoxel; ++j) {
                if (j >= max_pts) break;
                const uint32_t v = pi[j];
                pi[j] = min(v, carry), carry = max(v, carry);
            }
            int ix, iy, iz;
            voxel_cell(g, __ldg(points + (size_t)b * max_points + e), &ix, &iy, &iz);
            const size_t row = (size_t)b * out.max_voxels + id;
            reinterpret_cast<int4*>(out.coors)[row] = make_int4(b, iz, iy, ix);
            int cnt;
            const float4 m = voxel_mean(points + (size_t)b * max_points, max_pts, pi, &cnt);
            store_voxel(out.voxels, row, m.x, m.y, m.z, m.w);
            out.num_points[row] = cnt;
        }
    }
}

__global__ void __launch_bounds__(kThreads) fill_zero_kernel(uint4* __restrict__ p, size_t n16) {
    pdl_enter();
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += stride) p[i] = make_uint4(0, 0, 0, 0);
}

__global__ void __launch_bounds__(kThreads) prepare_kernel(FillRanges f, TailRows t) {
    pdl_enter();
    fill_ranges(f);
    zero_tails(t);
}

__global__ void publish_status_kernel(const int32_t* status, const int32_t* other, unsigned long long* host_word, uint32_t call) {
    pdl_enter();
    const unsigned long long v = (unsigned long long)call << 32 | (uint32_t)(*status | *other);
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(host_word), "l"(v) : "memory");
}

}  // namespace

// Stores `call` << 32 | *status | *other to mapped host memory behind the stream's work (sessd_read_status; not counted as a launch
// of the library's work).
cudaError_t launch_publish_status(const int32_t* status, const int32_t* other, unsigned long long* host_word, uint32_t call,
                                  cudaStream_t stream) {
    return launch_kernel(true, publish_status_kernel, 1, 1, 0, stream, status, other, host_word, call);
}

// The first launch of a call. A call that ends with tensor-core convolutions leaves the SMs set up for 200 KB of shared
// memory and a small L1; an SM changes that only when it is empty, and with overlapping launches throughout it never
// is: the table kernels that follow would run on the small L1 (32 frames x 120,000 points: insert 196 -> 453 us, emit
// 509 -> 737, neighbour map 551 -> 958). So there this launch waits for its predecessor to leave the SMs. It overlaps
// where that costs more than it gives: after calls that end otherwise, and for front ends of so few points that L1 hardly matters
// (overlapping and not: 20,000 points 251 and 255 us, two such frames 340 and 343, three 398 and 398, four 459 and 458, eight 727 and
// 712; one frame of 60,000 points 345 and 347, of 120,000 431 and 429: the line at 40,000 points could lie at 60,000 as well).
int launch_prepare(const FillRanges& f, const TailRows& t, bool overlap, cudaStream_t stream) {
    SESSD_LAUNCH_IMPL(overlap, "prepare_kernel", prepare_kernel, persistent_grid(8), kThreads, 0, stream, f, t);
    return SESSD_OK;
}

int launch_fill_zero(void* ptr, size_t bytes, cudaStream_t stream) {
    if (bytes == 0) return SESSD_OK;
    SESSD_LAUNCH(fill_zero_kernel, persistent_grid(8), kThreads, 0, stream, static_cast<uint4*>(ptr), bytes / 16);
    return SESSD_OK;
}

void voxel_workspace_layout(Bump& bump, const sessd_voxel_params* p, int batch, int max_points, VoxelWorkspace* w) {
    const uint32_t cap = pow2_at_least(2ull * (uint64_t)max_points);
    const size_t slots = (size_t)batch * cap;
    const size_t lists = ((size_t)batch * max_points * p->max_points_per_voxel + 3) / 4 * 4;   // (filled 16 bytes at a time)
    uint32_t* block = bump.take<uint32_t>(2 * slots + lists);   // contiguous, so that one fill resets both
    w->table = VoxelTable{reinterpret_cast<unsigned long long*>(block), block ? block + 2 * slots : nullptr, cap, 32 - ilog2(cap)};
    w->table_base = block;
    w->table_bytes = (2 * slots + lists) * sizeof(uint32_t);
    w->pt_claim = bump.take<int32_t>((size_t)batch * max_points);
    w->zero_bytes = scan_state_bytes(max_points, batch);
    char* zero = bump.take<char>(w->zero_bytes);
    w->zero_base = zero;
    w->scan = scan_state_at(zero, max_points, batch);
    w->num_points = bump.take<int32_t>((size_t)batch * p->max_voxels);
}

int voxelize_run(const sessd_voxel_params* p, int batch, int max_points, int out_dtype, const float* points,
                 const int32_t* points_size, void* voxels, int32_t* coors, int32_t* voxel_num, const VoxelWorkspace& w,
                 bool zero_tail, cudaStream_t stream) {
    const VoxGeom g = voxel_geom(*p);
    const float4* pts = reinterpret_cast<const float4*>(points);
    const int64_t items = (int64_t)batch * scan_chunks(max_points);
    const int grid = (int)(items < persistent_grid(8) ? items : persistent_grid(8));
    SESSD_LAUNCH(voxel_insert_kernel, grid, kThreads, 0, stream, pts, points_size, batch, max_points, g, w.table,
                 p->max_points_per_voxel, w.pt_claim, w.status);
    auto emit = [&](auto kernel, const auto& o, int steps) -> int {
        const int64_t chunks = (int64_t)batch * ((max_points + steps * kThreads - 1) / (steps * kThreads));
        SESSD_LAUNCH_NAMED("voxel_emit_kernel", kernel, (int)(chunks < persistent_grid(8) ? chunks : persistent_grid(8)), kThreads, 0, stream,
                           pts, points_size, batch, max_points, g, w.table, p->max_points_per_voxel, w.pt_claim, w.scan, o);
        return SESSD_OK;
    };
    // A block's chunk is a chain of some five accesses that wait for one another, so that two points per thread pay once there are
    // more chunks of one than blocks at a time (in us, one point and two: 64 x 20,000 points 84.1 and 80.0, 12 x 120,000 110 and 100,
    // 16 x 20,000 34.6 and 33.0; 8 x 20,000, 632 chunks, 25.1 and 25.6, 1 x 20,000 16.9 and 17.5; four: 80.1, 99, 33.8, 27.9, 19.7).
    const bool two = (int64_t)batch * scan_chunks(max_points) > persistent_grid(5);
    if (out_dtype == SESSD_F32) {
        const VoxelOut<float> o{static_cast<float*>(voxels), coors, w.num_points, voxel_num, w.status, p->max_voxels, zero_tail};
        return two ? emit(voxel_emit_kernel<float, 2>, o, 2) : emit(voxel_emit_kernel<float, 1>, o, 1);
    }
    const VoxelOut<__half> o{static_cast<__half*>(voxels), coors, w.num_points, voxel_num, w.status, p->max_voxels, zero_tail};
    return two ? emit(voxel_emit_kernel<__half, 2>, o, 2) : emit(voxel_emit_kernel<__half, 1>, o, 1);
}

}  // namespace sessd
