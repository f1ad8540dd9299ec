// Neighbour maps: nbr[b][k][p] = input row under kernel offset k of the output row at position p, or -1, and the offsets
// that each 128-position tile has any neighbour under.
//
// Output-stationary: a thread walks the K0 x K1 lines of its row's receptive field (in = out*stride - pad + k, the inverse
// of the offset formula at submConv3dlayer.cu:328) and asks an index of the input level for the K2 x-neighbours of each.
// The index is the level's occupancy grid where it has one, else an x-grouped coordinate table (rows handed in by a
// caller).
//
// Grids: a block takes a window of 2048 output rows, collects their entries in shared memory, and orders the rows by which of
// the six outer planes of the kernel (first and last in z, y and x) hold a neighbour: a counting sort with 64 bins, in Gray
// order, because a tile spans several bins and neighbouring ones should differ little (1 to 3 % fewer pairs than in binary order).
// Tiles of such rows need fewer (tile, offset) pairs, which is what the convolutions' time depends on: for the strided
// layers of the network a third fewer, for the 64-channel submanifold layers a seventh (a full sort by the 27-bit mask
// does worse, because its most significant offsets say little about the others). order[b][p] is the row at position p;
// what a row computes does not depend on its position. The entries leave as whole 128-byte runs, and runs of offsets
// that a tile has no neighbour under are not written at all.
//
// Larger windows leave fewer pairs: 2048 rows instead of 1024, 3 % fewer for the submanifold and 7 % for the strided layers
// (32 frames x 120,000 points: this kernel 940 -> 1002 us, the convolutions after it 4,820 -> 4,660).
//
// Row by row without windows, six launches of this took 1.00 ms for 32 frames x 120,000 points, and the full-resolution
// maps another 0.9 through a table and an input-stationary scatter.
#include "fill.cuh"
#include "rulebook.cuh"
#include "voxel.cuh"

namespace sessd {

namespace {

constexpr int kWindow = 2048;              // rows of a window (sixteen tiles)
constexpr int kMapThreads = 1024;          // two rows per thread
constexpr int kMapBlocks = 1;              // per SM: 64 registers (with 40 they spill, and it is an eighth slower)
constexpr int kMapKvol = 27;
constexpr int kGroups = kWindow / 32;      // groups of 32 rows, one per warp and step

struct MapShared {
    int32_t base[9][kWindow];              // per line of the receptive field: the input row of its first neighbour
    uint32_t bits[kWindow];                // which offsets have a neighbour (none for rows past the frame's)
    union {
        uint16_t count[64][kGroups];       // rows per bin and group of 32 rows; then where they start
        uint16_t src[kWindow];             // row of the window at each position
    };
    alignas(16) uint32_t group_bits[kGroups];          // offsets that 32 positions have any neighbour under
    int warp_sum[kMapThreads / 32];
};

// Through a level's occupancy grid. The K2 x-neighbours x0 .. x0 + K2 - 1 of a line (z, y) are neighbouring bits that may
// straddle two words, and rows are numbered along the line, so a line is told by its bits and the row of its first
// neighbour: all that the window keeps of it. What the lines of one output row share (Row) is worked out once; a line is
// then told by its distance from the row's first line. Reads go in two steps, so that a thread has the reads of several lines in
// flight.
struct BitsIndex {
    const uint4* rec;      // of the frame
    const uint4* top;      // of the frame, or null (one-level grid)
    int Y, X, xw;
    struct Row {
        int word;
        uint32_t sh, below_lo, below_hi;   // first bit of the window (mod 32), bits of the word before it
        uint32_t lead;                     // cells of the window before the line (x < 0; up to the padding, 2)
        bool upper, two;                   // window starts in the word's upper half; goes on in the next word
    };
    static __device__ __forceinline__ BitsIndex make(const MapJob& j, int b) {
        const BitGrid& g = j.in;
        return BitsIndex{g.rec + (size_t)b * g.words, g.top ? g.top + (size_t)b * g.top_words : nullptr, g.Y, g.X, g.xw};
    }
    __device__ __forceinline__ Row row(int z, int y, int x0, int count) const {
        const int lo = max(x0, 0), hi = min(x0 + count, X) - 1;
        const uint32_t sh = lo & 31, below = (1u << sh) - 1u;
        const bool upper = lo & 32;
        return Row{(z * Y + y) * xw + (lo >> 6), sh, upper ? ~0u : below, upper ? below : 0u, (uint32_t)(lo - x0), upper,
                   (hi >> 6) > (lo >> 6)};
    }
    __device__ __forceinline__ int step(int kz, int ky) const { return (kz * Y + ky) * xw; }
    template <bool TOP>
    __device__ __forceinline__ uint4 first(int w, bool on) const {   // (off: some record, which finish() then ignores)
        return __ldg(TOP ? top + (on ? w >> 6 : 0) : rec + (on ? w : 0));
    }
    // Record of word w of a two-level grid, given its top record; empty when the word is.
    __device__ __forceinline__ uint4 word_record(int w, const uint4& t) const {
        const uint32_t bit = 1u << (w & 31);
        const bool upper = w & 32;
        if (!((upper ? t.y : t.x) & bit)) return make_uint4(0u, 0u, 0u, 0u);
        return __ldg(rec + ((int)t.z + __popc(upper ? t.x : 0u) + __popc((upper ? t.y : t.x) & (bit - 1u))));
    }
    template <bool TOP>
    __device__ __forceinline__ void second(const Row& r, int w, bool on, uint4* l) const {
        if (!TOP) return;
        if (on) *l = word_record(w, *l);
        l->w = 0u;
        if (r.two && on) {
            const uint4 next = word_record(w + 1, __ldg(top + ((w + 1) >> 6)));
            if (!(l->x | l->y)) l->z = next.z;   // the rows of the window are then all of the second word
            l->w = next.x & 3u;
        }
    }
    // Neighbours of a line as bits, and the row of the first.
    template <int COUNT>
    __device__ __forceinline__ uint32_t finish(const Row& r, const uint4& l, bool on, int* base) const {
        const uint32_t w = __funnelshift_r(r.upper ? l.y : l.x, r.upper ? l.w : l.y, r.sh) << r.lead;
        *base = (int)l.z + __popc(l.x & r.below_lo) + __popc(l.y & r.below_hi);
        return w & (on ? (1u << COUNT) - 1u : 0u);
    }
};

// Neighbours of the row whose first input cell is (z, y, x), as a mask of offsets; put(line, row of its first neighbour).
// KZ, KY, KX: the kernel.
template <int KZ, int KY, int KX, bool TOP, class Put>
__device__ __forceinline__ uint32_t grid_row(const BitsIndex& in, int Z, int z, int y, int x, bool live, Put put) {
    constexpr int BATCH = TOP ? 1 : KZ;                      // planes whose reads are in flight together
    const BitsIndex::Row row = in.row(z, y, x, KX);
    bool y_ok[KY];
#pragma unroll
    for (int ky = 0; ky < KY; ++ky) y_ok[ky] = live && (unsigned)(y + ky) < (unsigned)in.Y;
    uint32_t bits = 0;
#pragma unroll
    for (int kz0 = 0; kz0 < KZ; kz0 += BATCH) {
        uint4 l[BATCH * KY];
        bool on[BATCH * KY];
#pragma unroll
        for (int i = 0; i < BATCH * KY; ++i) {
            const int kz = kz0 + i / KY, ky = i % KY;
            on[i] = y_ok[ky] && (unsigned)(z + kz) < (unsigned)Z;
            l[i] = in.template first<TOP>(row.word + in.step(kz, ky), on[i]);
        }
#pragma unroll
        for (int i = 0; i < BATCH * KY; ++i) in.template second<TOP>(row, row.word + in.step(kz0 + i / KY, i % KY), on[i], &l[i]);
#pragma unroll
        for (int i = 0; i < BATCH * KY; ++i) {
            int base;
            bits |= in.template finish<KX>(row, l[i], on[i], &base) << ((kz0 * KY + i) * KX);
            put(kz0 * KY + i, base);
        }
    }
    return bits;
}

// Any other kernel up to 3 x 3 x 3: one line at a time.
template <class Put>
__device__ __noinline__ uint32_t grid_row_any(const BitsIndex& in, const ConvGeom& g, int z, int y, int x, bool live, Put put) {
    const BitsIndex::Row row = in.row(z, y, x, g.K[2]);
    uint32_t bits = 0;
    for (int kz = 0; kz < g.K[0]; ++kz)
        for (int ky = 0; ky < g.K[1]; ++ky) {
            const bool on = live && (unsigned)(z + kz) < (unsigned)g.in_shape[0] && (unsigned)(y + ky) < (unsigned)in.Y;
            const int w = row.word + in.step(kz, ky), line = kz * g.K[1] + ky;
            uint4 l = in.top ? in.first<true>(w, on) : in.first<false>(w, on);
            if (in.top) in.second<true>(row, w, on, &l);
            int base;
            bits |= (in.finish<3>(row, l, on, &base) & ((1u << g.K[2]) - 1u)) << (line * g.K[2]);
            put(line, base);
        }
    return bits;
}

template <class Put>
__device__ __forceinline__ uint32_t grid_entries(const BitsIndex& in, const MapJob& job, const int4& c, bool live, Put put) {
    const ConvGeom& g = job.g;
    const int z = c.y * g.S[0] - g.P[0], y = c.z * g.S[1] - g.P[1], x = c.w * g.S[2] - g.P[2];
    switch (job.shape) {                                     // uniform over the block
        case 333:
            if (in.top) return grid_row<3, 3, 3, true>(in, g.in_shape[0], z, y, x, live, put);
            return grid_row<3, 3, 3, false>(in, g.in_shape[0], z, y, x, live, put);
        case 311:
            if (!in.top) return grid_row<3, 1, 1, false>(in, g.in_shape[0], z, y, x, live, put);
            [[fallthrough]];
        default: return grid_row_any(in, g, z, y, x, live, put);
    }
}

// The entries of one position for the offsets in m; its row of the window is r, with neighbours w.
template <int KX>
__device__ __forceinline__ void write_entries(const MapShared& s, int r, uint32_t w, uint32_t m, int lines, int32_t* out) {
#pragma unroll
    for (int line = 0; line < 9; ++line, w >>= KX) {
        if (line >= lines) break;
        const uint32_t t = m >> (line * KX);
        if (!(t & ((1u << KX) - 1u))) continue;              // uniform over the warp
        const int base = s.base[line][r];
#pragma unroll
        for (int k = 0; k < KX; ++k)
            if ((t >> k) & 1u)
                out[(line * KX + k) * kNbrRun] = (w >> k) & 1u ? base + __popc(w & ((1u << k) - 1u)) : -1;
    }
}

// Through the x-grouped table: the three x-neighbours lie in at most two 32-byte buckets.
// Same division of the work as above, but the rows are in no order: a line is its three rows.
struct BucketIndex {
    const uint32_t* data;   // of the frame
    uint32_t cap;
    int shift, Y, X;
    struct Row { uint32_t cell; int lo, hi; };              // cell: key of (z, y, x0); the line's cells are x0 + lo .. x0 + hi
    struct Line { uint4 lo[2], hi[2]; uint32_t key[2]; };
    static __device__ __forceinline__ BucketIndex make(const MapJob& j, int b) {
        return BucketIndex{j.table.data + (size_t)b * j.table.cap * 8, j.table.cap, j.table.shift, j.g.in_shape[1], j.g.in_shape[2]};
    }
    __device__ __forceinline__ Row row(int z, int y, int x0, int count) const {
        return Row{(uint32_t)((z * Y + y) * X + x0), x0 < 0 ? -x0 : 0, min(x0 + count, X) - 1 - x0};
    }
    __device__ __forceinline__ int step(int kz, int ky) const { return (kz * Y + ky) * X; }
    __device__ __forceinline__ void first(const Row& r, int step, bool on, Line* l) const {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            l->lo[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
            l->hi[i] = make_uint4(kEmpty, 0u, 0u, 0u);
            l->key[i] = kEmpty;
            if (!on || r.lo > r.hi) continue;
            const uint32_t key = (r.cell + (uint32_t)step + (uint32_t)(i == 0 ? r.lo : r.hi)) >> 2;
            if (i == 1 && key == l->key[0]) continue;
            l->key[i] = key;
            // the whole 32-byte bucket with one 256-bit load (one request to L1 instead of two)
            asm volatile("ld.global.nc.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(l->lo[i].x), "=r"(l->lo[i].y), "=r"(l->lo[i].z), "=r"(l->lo[i].w), "=r"(l->hi[i].x),
                           "=r"(l->hi[i].y), "=r"(l->hi[i].z), "=r"(l->hi[i].w)
                         : "l"(data + (size_t)hash_slot(key, shift) * 8));
        }
    }
    __device__ __forceinline__ void second(const Row&, int, Line* l) const {   // first slot taken by another group: keep probing
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (l->key[i] == kEmpty || l->hi[i].x == l->key[i]) continue;
            uint32_t h = hash_slot(l->key[i], shift);
            uint4 lo = make_uint4(~0u, ~0u, ~0u, ~0u);
            uint32_t cur = l->hi[i].x;
            for (uint32_t probe = 1; probe < cap && cur != kEmpty; ++probe) {
                h = (h + 1) & (cap - 1);
                const uint4* bk = reinterpret_cast<const uint4*>(data + (size_t)h * 8);
                cur = __ldg(bk + 1).x;
                if (cur == l->key[i]) {
                    lo = __ldg(bk);
                    break;
                }
            }
            l->lo[i] = lo;
        }
    }
    static __device__ __forceinline__ int pick(const uint4& v, uint32_t i) {
        return (int)(i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)));
    }
    template <int COUNT>
    __device__ __forceinline__ uint32_t finish(const Row& r, int step, const Line& l, int (&rows)[3]) const {
        uint32_t w = 0;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            rows[e] = -1;
            if (e >= COUNT || e < r.lo || e > r.hi || l.key[0] == kEmpty) continue;
            const uint32_t key = r.cell + (uint32_t)step + (uint32_t)e;
            rows[e] = pick((key >> 2) == l.key[0] ? l.lo[0] : l.lo[1], key & 3u);
            w |= (rows[e] >= 0 ? 1u : 0u) << e;
        }
        return w;
    }
};

// Entries of the row whose first input cell is (z, y, x) under plane kz of the kernel: put(offset, input row or -1) for every
// offset, and as a mask of the offsets that have one.
template <int KY, int KX, class Index, class Put>
__device__ __forceinline__ uint32_t map_plane(const Index& in, int Z, int kz, int z, int y, int x, bool live, Put put) {
    const typename Index::Row row = in.row(z, y, x, KX);
    uint32_t bits = 0;
    const bool z_ok = live && (unsigned)(z + kz) < (unsigned)Z;
    typename Index::Line l[KY];
#pragma unroll
    for (int ky = 0; ky < KY; ++ky)
        in.first(row, in.step(kz, ky), z_ok && (unsigned)(y + ky) < (unsigned)in.Y, &l[ky]);
#pragma unroll
    for (int ky = 0; ky < KY; ++ky) in.second(row, in.step(kz, ky), &l[ky]);
#pragma unroll
    for (int ky = 0; ky < KY; ++ky) {
        int rows[3];
        const int k0 = (kz * KY + ky) * KX;
        bits |= in.template finish<KX>(row, in.step(kz, ky), l[ky], rows) << k0;
#pragma unroll
        for (int kx = 0; kx < KX; ++kx) put(k0 + kx, rows[kx]);
    }
    return bits;
}

// Any other kernel up to 3 x 3 x 3: one line at a time.
template <class Index, class Put>
__device__ __noinline__ uint32_t map_row_any(const Index& in, const ConvGeom& g, int z, int y, int x, bool live, Put put) {
    const typename Index::Row row = in.row(z, y, x, g.K[2]);
    uint32_t bits = 0;
    for (int kz = 0; kz < g.K[0]; ++kz)
        for (int ky = 0; ky < g.K[1]; ++ky) {
            const bool on = live && (unsigned)(z + kz) < (unsigned)g.in_shape[0] && (unsigned)(y + ky) < (unsigned)in.Y;
            typename Index::Line l;
            int rows[3];
            in.first(row, in.step(kz, ky), on, &l);
            in.second(row, in.step(kz, ky), &l);
            const uint32_t w = in.template finish<3>(row, in.step(kz, ky), l, rows);
            const int k0 = (kz * g.K[1] + ky) * g.K[2];
            for (int kx = 0; kx < g.K[2]; ++kx) put(k0 + kx, rows[kx]);
            bits |= (w & ((1u << g.K[2]) - 1u)) << k0;
        }
    return bits;
}

// Planes `plane`, `plane` + STEP, ..
template <int STEP, class Index, class Put>
__device__ __forceinline__ uint32_t map_entries(const Index& in, const MapJob& job, int plane, const int4& c, bool live, Put put) {
    const ConvGeom& g = job.g;
    const int z = c.y * g.S[0] - g.P[0], y = c.z * g.S[1] - g.P[1], x = c.w * g.S[2] - g.P[2];
    uint32_t bits = 0;
    switch (job.shape) {                                     // uniform over the block
        case 333:
#pragma unroll
            for (int k = 0; k < 3; k += STEP) bits |= map_plane<3, 3>(in, g.in_shape[0], plane + k, z, y, x, live, put);
            return bits;
        case 311:
#pragma unroll
            for (int k = 0; k < 3; k += STEP) bits |= map_plane<1, 1>(in, g.in_shape[0], plane + k, z, y, x, live, put);
            return bits;
        default: return plane == 0 ? map_row_any(in, g, z, y, x, live, put) : 0u;
    }
}

template <typename T>
__device__ __forceinline__ void row_means(const RowMeans& m, T* voxels, int batch, int max_voxels, int block, int blocks) {
    const int chunks = (m.max_points + kMapThreads - 1) / kMapThreads;   // rows never outnumber points
    for (int it = block; it < batch * chunks; it += blocks) {
        const int b = it / chunks;
        const int row = (it - b * chunks) * kMapThreads + threadIdx.x;
        if (row >= load_late(m.voxel_num + b)) continue;
        uint32_t pi[kMaxPointsPerVoxel];
        list_load(m.lists + ((size_t)b * m.max_points + row) * m.max_pts, m.max_pts, pi);
        int cnt;
        const float4 v = voxel_mean(m.points + (size_t)b * m.max_points, m.max_pts, pi, &cnt);
        store_voxel(voxels, (size_t)b * max_voxels + row, v.x, v.y, v.z, v.w);
    }
}

__global__ void __launch_bounds__(kMapThreads, kMapBlocks)
map_windows_kernel(const __grid_constant__ MapJobs jobs, int batch, int max_voxels, int tiles_per_frame, RowMeans means) {
    pdl_enter();
    extern __shared__ __align__(16) uint8_t map_smem[];
    MapShared& s = *reinterpret_cast<MapShared*>(map_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // The windows that hold rows, numbered over (job, frame) pairs: a walk that only moves forward, 32 pairs at a time
    // (lane = pair), the same in every warp.
    const int pairs = jobs.count * batch;
    auto pair_rows = [&](int p) {
        if (p >= pairs) return 0;
        const int j = p / batch;
        const int v = load_late(jobs.job[j].out_num + (p - j * batch));
        return v > max_voxels ? max_voxels : (v < 0 ? 0 : v);
    };
    int pair0 = 0, before = 0, my_rows = pair_rows(lane), incl = 0;
    auto running = [&]() {
        incl = (my_rows + kWindow - 1) / kWindow;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += t;
        }
    };
    running();
    struct Window { int job, frame, first, rows; };
    auto locate = [&](int it) {                              // the it-th window (rows = 0: there is none)
        for (int total = __shfl_sync(0xFFFFFFFFu, incl, 31); it >= before + total && pair0 < pairs;
             total = __shfl_sync(0xFFFFFFFFu, incl, 31)) {
            before += total;
            pair0 += 32;
            my_rows = pair_rows(pair0 + lane);
            running();
        }
        if (pair0 >= pairs) return Window{0, 0, 0, 0};
        const int src_lane = __ffs((int)__ballot_sync(0xFFFFFFFFu, it < before + incl)) - 1;
        const int ji = (pair0 + src_lane) / batch;
        const int first = (it - before - __shfl_sync(0xFFFFFFFFu, incl - (my_rows + kWindow - 1) / kWindow, src_lane)) * kWindow;
        return Window{ji, pair0 + src_lane - ji * batch, first, min(__shfl_sync(0xFFFFFFFFu, my_rows, src_lane) - first, kWindow)};
    };
    // The coordinates of a window's rows are requested a window ahead: one block per SM does not hide that latency.
    int4 coor[2];
    auto fetch = [&](const Window& w) {
        const int4* c = reinterpret_cast<const int4*>(jobs.job[w.job].out_coors) + (size_t)w.frame * max_voxels + w.first;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            coor[i] = make_int4(0, 0, 0, 0);
            if (tid + i * kMapThreads < w.rows) coor[i] = __ldg(c + tid + i * kMapThreads);
        }
    };
    Window next = locate(blockIdx.x);
    fetch(next);
    for (int it = blockIdx.x; next.rows > 0;) {
        const int b = next.frame, w0 = next.first, n = next.rows;   // (rows of this window)
        const MapJob& job = jobs.job[next.job];
        const BitsIndex in = BitsIndex::make(job, b);
        it += gridDim.x;
        next = locate(it);
        __syncthreads();                                     // the previous window has been written out
        for (int e = tid; e < 64 * kGroups / 2; e += kMapThreads) reinterpret_cast<uint32_t*>(s.count)[e] = 0u;
        __syncthreads();
        // entries of this thread's rows, and the rows' offsets
        uint32_t mask[2], rank[2], bin[2];
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const int r = tid + i * kMapThreads;
            const bool live = r < n;
            const uint32_t bits = grid_entries(in, job, i == 0 ? coor[0] : coor[1], live, [&](int line, int base) { s.base[line][r] = base; });
            s.bits[r] = bits;
            uint32_t key = 64u;                              // dead rows (the frame's last window): they stay behind
            if (live) {
                key = 0u;
                if (job.order)
#pragma unroll
                    for (int q = 0; q < 6; ++q) key = key << 1 | ((bits & job.plane[q]) ? 1u : 0u);
                key ^= key >> 1, key ^= key >> 2, key ^= key >> 4;   // rank of the bin in Gray order
            }
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
            const uint32_t before = __popc(peers & ((1u << lane) - 1u));
            if (live && before == 0u) s.count[key][warp + i * (kMapThreads / 32)] = (uint16_t)__popc(peers);
            if (i == 0) mask[0] = bits, rank[0] = before, bin[0] = key;
            else mask[1] = bits, rank[1] = before, bin[1] = key;
        }
        fetch(next);
        __syncthreads();
        {   // running totals over (bin, group), four entries per thread
            uint2* at = reinterpret_cast<uint2*>(s.count) + tid;
            const uint2 v = *at;
            const int c0 = v.x & 0xFFFFu, c1 = v.x >> 16, c2 = v.y & 0xFFFFu, c3 = v.y >> 16;
            const int sum = c0 + c1 + c2 + c3;
            int incl = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= d) incl += t;
            }
            if (lane == 31) s.warp_sum[warp] = incl;
            __syncthreads();
            int base = incl - sum;
            for (int w = 0; w < warp; ++w) base += s.warp_sum[w];
            *at = make_uint2((uint32_t)base | (uint32_t)(base + c0) << 16,
                             (uint32_t)(base + c0 + c1) | (uint32_t)(base + c0 + c1 + c2) << 16);
        }
        __syncthreads();
        int pos[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            pos[i] = tid + i * kMapThreads;
            if (bin[i] < 64u) pos[i] = s.count[bin[i]][warp + i * (kMapThreads / 32)] + (int)rank[i];
        }
        __syncthreads();                                     // src takes the counts' place
#pragma unroll
        for (int i = 0; i < 2; ++i) s.src[pos[i]] = (uint16_t)(tid + i * kMapThreads);
        __syncthreads();
        // a warp takes 32 positions of a tile, and again 32
        int from[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int p = tid + i * kMapThreads;
            from[i] = s.src[p];
            mask[i] = s.bits[from[i]];                       // of the position from here on (dead rows: none)
            const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, mask[i]);
            if (lane == 0) s.group_bits[p >> 5] = any;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int p = tid + i * kMapThreads;
            const int tile0 = p & ~127;
            if (tile0 >= n) break;                           // a tile without rows (uniform over the warp)
            const uint4 g = *reinterpret_cast<const uint4*>(&s.group_bits[tile0 >> 5]);
            uint32_t m = g.x | g.y | g.z | g.w;
            if ((p & 127) == 0) {
                job.tile_mask[(size_t)b * tiles_per_frame + ((w0 + p) >> 7)] = m;
                *reinterpret_cast<uint4*>(job.nbr + nbr_runs_index(job.g.kvol, max_voxels, b, w0 + p)) = g;
            }
            // a consumer that fetches `group` offsets at a time wants all of them as soon as it wants one
            if (job.group >= 2) m |= (m & 0x55555555u) << 1 | ((m >> 1) & 0x55555555u);
            if (job.group >= 4) m |= (m & 0x33333333u) << 2 | ((m >> 2) & 0x33333333u);
            if (job.order && p < n) job.order[(size_t)b * max_voxels + w0 + p] = w0 + from[i];
            int32_t* out = job.nbr + nbr_index(job.g.kvol, max_voxels, b, 0, w0 + p);
            if (job.g.kvol < kMapKvol) m &= (1u << job.g.kvol) - 1u;
            const int lines = job.g.K[0] * job.g.K[1];
            switch (job.g.K[2]) {                            // uniform over the block
                case 3: write_entries<3>(s, from[i], mask[i], m, lines, out); break;
                case 2: write_entries<2>(s, from[i], mask[i], m, lines, out); break;
                default: write_entries<1>(s, from[i], mask[i], m, lines, out);
            }
        }
    }
    // Beside the maps: the means of the voxeliser's rows. From the last block down, which has the fewest windows.
    if (means.points) {
        const int block = (int)(gridDim.x - 1 - blockIdx.x);
        if (means.half) row_means(means, static_cast<__half*>(means.voxels), batch, max_voxels, block, gridDim.x);
        else row_means(means, static_cast<float*>(means.voxels), batch, max_voxels, block, gridDim.x);
    }
}

// Maps through a table: rows as a caller (or the voxeliser, in point order) numbered them. Every line is one or two
// scattered 32-byte reads, which bounds an SM (a block of 1024 rows took 40 us for its 18 reads per row), so the rows are
// spread over as many SMs as there are tiles: a block per tile, no ordering. PLANES threads share a row, one or all three of the
// kernel's planes each: the launch's choice. Also zeroes the tails of the call's outputs, whose row counts are known by now.
template <int PLANES>
__global__ void __launch_bounds__(128 * PLANES)
map_tiles_kernel(const __grid_constant__ MapJob job, int batch, int max_voxels, int tiles_per_frame, TailRows tails, int runs) {
    pdl_enter();
    zero_tails(tails);
    __shared__ uint32_t s_mask[4 * PLANES];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, plane = tid >> 7, row = tid & 127;
    for (int it = blockIdx.x; it < batch * tiles_per_frame; it += gridDim.x) {
        const int b = it / tiles_per_frame, p0 = (it - b * tiles_per_frame) * 128;
        int n = load_late(job.out_num + b);
        n = n > max_voxels ? max_voxels : n;
        if (p0 >= n) continue;
        const bool live = p0 + row < n;
        int4 c = make_int4(0, 0, 0, 0);
        if (live) c = __ldg(reinterpret_cast<const int4*>(job.out_coors) + (size_t)b * max_voxels + p0 + row);
        int32_t* out = job.nbr + nbr_index(job.g.kvol, max_voxels, b, 0, p0 + row);
        const uint32_t bits = map_entries<PLANES>(BucketIndex::make(job, b), job, plane, c, live, [&](int k, int v) { out[k * kNbrRun] = v; });
        const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, bits);
        __syncthreads();
        if (lane == 0) s_mask[warp] = any;
        __syncthreads();
        if (tid == 0) {
            uint32_t m = 0;
#pragma unroll
            for (int w = 0; w < 4 * PLANES; ++w) m |= s_mask[w];
            job.tile_mask[it] = m;
        }
        if (runs && tid < 4) {                               // of 32 rows each
            uint32_t m = 0;
#pragma unroll
            for (int p = 0; p < PLANES; ++p) m |= s_mask[4 * p + tid];
            job.nbr[nbr_runs_index(job.g.kvol, max_voxels, b, p0 + 32 * tid)] = (int32_t)m;
        }
    }
}

}  // namespace

MapJob make_map_job(const ConvGeom& g, const int32_t* out_coors, const int32_t* out_num, int cin, int32_t* nbr,
                    uint32_t* tile_mask, int32_t* order) {
    MapJob j{};
    j.out_coors = out_coors;
    j.out_num = out_num;
    j.g = g;
    j.nbr = nbr;
    j.tile_mask = tile_mask;
    j.order = order;
    j.shape = g.K[0] * 100 + g.K[1] * 10 + g.K[2];
    j.group = cin >= 64 ? 1 : (cin >= 32 ? 2 : 4);       // 64 / cin offsets per stage of the tensor-core kernel
    for (int k = 0; k < g.kvol; ++k) {
        const int at[3] = {k / (g.K[1] * g.K[2]), k / g.K[2] % g.K[1], k % g.K[2]};
        for (int d = 0; d < 3; ++d) {
            if (g.K[d] < 2) continue;
            if (at[d] == 0) j.plane[2 * d] |= 1u << k;
            if (at[d] == g.K[d] - 1) j.plane[2 * d + 1] |= 1u << k;
        }
    }
    return j;
}

int launch_map_windows(const MapJobs& jobs, int batch, int max_voxels, const RowMeans& means, cudaStream_t stream) {
    if (jobs.count == 0 && !means.points) return SESSD_OK;
    static_assert(sizeof(MapShared) <= 227 * 1024, "a window does not fit the shared memory of one SM");
    // the attribute belongs to the device's context: set it once per device (repeating it is harmless)
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    SESSD_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        SESSD_CUDA(cudaFuncSetAttribute(map_windows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MapShared)));
        configured.fetch_or(bit, std::memory_order_release);
    }
    const int64_t items = (int64_t)(jobs.count > 0 ? jobs.count : 1) * batch * ((max_voxels + kWindow - 1) / kWindow);
    const int most = persistent_grid(kMapBlocks);
    SESSD_LAUNCH(map_windows_kernel, (int)(items < most ? items : most), kMapThreads, sizeof(MapShared), stream, jobs, batch,
                 max_voxels, (max_voxels + 127) / 128, means);
    return SESSD_OK;
}

int launch_map_tiles(const MapJob& job, int batch, int max_voxels, const TailRows& tails, cudaStream_t stream) {
    const int tiles = (max_voxels + 127) / 128;
    const int64_t items = (int64_t)batch * tiles;
    const int runs = (int64_t)batch * max_voxels > kRunRows ? 1 : 0;
    // A thread per plane up to room for twelve tiles per SM: the planes of a row one after the other are what a small call waits for.
    // Beyond that the reads bound the SMs, and three times the threads read coordinates and row counts. (This kernel in us, a thread
    // per row and three, 4 -> 16, 32 -> 32 and 64 -> 64 channels: room for 469 tiles, 1 x 20,000 points 17.1 and 11.3, 19.1 and 13.0,
    // 9.8 and 6.3; 1,563, 1 x 120,000 30.8 and 28.8, 35.9 and 37.4, 10.1 and 8.0; 1,876, 2 x 60,000 24.3 and 24.0, 34.9 and 32.8, 11.0
    // and 9.8; 1,876, 4 x 20,000 23.0 and 21.5, 27.4 and 28.2, 11.7 and 12.0; 2,345, 5 x 20,000 24.3 and 24.0, 31.8 and 33.4, 12.7 and
    // 13.2; 2,814, 3 x 60,000 28.5 and 31.7, 41.4 and 44.8, 13.1 and 14.2; 3,126, 2 x 120,000 36.2 and 44.0, 55.0 and 62.3, 12.6 and
    // 13.2; 5,628, 12 x 20,000 45.4 and 51.0, 62.4 and 74.1, 25.2 and 30.0.)
    if (items <= persistent_grid(12)) {
        SESSD_LAUNCH(map_tiles_kernel<3>, (int)items, 384, 0, stream, job, batch, max_voxels, tiles, tails, runs);
        return SESSD_OK;
    }
    // four rounds of the nine blocks that are resident: with six per SM the reads in flight did not cover their latency, and in few
    // rounds the blocks whose tiles are empty leave SMs idle (calls of 8 x 120,000 points, 4 -> 16 channels: six 334 us, nine 318,
    // eighteen 307, thirty-six 304; 4 x 20,000 points, 16 -> 16: 54, 53, 44, 44)
    const int most = persistent_grid(36);
    SESSD_LAUNCH(map_tiles_kernel<1>, (int)(items < most ? items : most), 128, 0, stream, job, batch, max_voxels, tiles, tails, runs);
    return SESSD_OK;
}

}  // namespace sessd
