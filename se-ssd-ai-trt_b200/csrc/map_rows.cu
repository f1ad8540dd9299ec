// Neighbour maps: nbr[b][k][p] = input row under kernel offset k of the output row at position p, or -1, and the offsets
// that each 128-position tile has any neighbour under.
//
// Output-stationary: a thread walks the K0 x K1 lines of its row's receptive field (in = out*stride - pad + k, the inverse
// of the offset formula at submConv3dlayer.cu:328) and asks an index of the input level for the K2 x-neighbours of each.
// The index is the level's occupancy grid where it has one, else an x-grouped coordinate table (rows handed in by a
// caller).
//
// A block takes a window of 1024 output rows, collects their entries in shared memory, and orders the rows by which of
// the six outer planes of the kernel (first and last in z, y and x) hold a neighbour: a counting sort with 64 bins.
// Tiles of such rows need fewer (tile, offset) pairs, which is what the convolutions' time depends on: for the strided
// layers of the network a third fewer, for the 64-channel submanifold layers a seventh (a full sort by the 27-bit mask
// does worse, because its most significant offsets say little about the others). order[b][p] is the row at position p;
// what a row computes does not depend on its position. The entries leave as whole 128-byte runs, and runs of offsets
// that a tile has no neighbour under are not written at all.
//
// Row by row without windows, six launches of this took 1.00 ms for 32 frames x 120,000 points, and the full-resolution
// maps another 0.9 through a table and an input-stationary scatter.
#include "fill.cuh"
#include "rulebook.cuh"

namespace sessd {

namespace {

constexpr int kWindow = 1024;              // rows of a window (eight tiles)
constexpr int kMapThreads = 512;           // two rows per thread; two blocks per SM
constexpr int kMapKvol = 27;
constexpr int kGroups = kWindow / 32;      // groups of 32 rows, one per warp and step

struct MapShared {
    int32_t ids[kMapKvol][kWindow];
    union {
        uint16_t count[64][kGroups];       // rows per bin and group of 32 rows; then where they start
        uint16_t src[kWindow];             // row of the window at each position
    };
    uint32_t tile[kWindow / 128];
    int warp_sum[kMapThreads / 32];
};

// Rows of the input level through its occupancy grid. Line probes in two steps, so that a thread has the reads of
// several lines in flight.
struct BitsIndex {
    BitGrid g;
    struct Probe { uint4 a, b; int w; bool two; };
    // Record of an occupied word of a two-level grid, given its top record; empty when the word is.
    __device__ __forceinline__ uint4 word_record(int b, int word, const uint4& t) const {
        const unsigned long long tb = rec_bits(t), bit = 1ull << (word & 63);
        if (!(tb & bit)) return make_uint4(0u, 0u, 0u, 0u);
        return __ldg(g.rec + (size_t)b * g.words + (int)t.z + __popcll(tb & (bit - 1ull)));
    }
    __device__ __forceinline__ void probe_first(int b, int z, int y, int x0, int count, bool on, Probe* p) const {
        p->a = p->b = make_uint4(0u, 0u, 0u, 0u);
        p->two = false;
        p->w = -1;
        if (!on) return;
        const int lo = x0 < 0 ? 0 : x0, hi = x0 + count - 1 >= g.X ? g.X - 1 : x0 + count - 1;
        if (lo > hi) return;
        p->w = (z * g.Y + y) * g.xw + (lo >> 6);
        p->two = (hi >> 6) != (lo >> 6);
        if (!g.top) return;
        p->a = __ldg(g.top + (size_t)b * g.top_words + (p->w >> 6));
        if (p->two) p->b = __ldg(g.top + (size_t)b * g.top_words + ((p->w + 1) >> 6));
    }
    __device__ __forceinline__ void probe_second(int b, Probe* p) const {
        if (p->w < 0) return;
        if (g.top) {
            p->a = word_record(b, p->w, p->a);
            if (p->two) p->b = word_record(b, p->w + 1, p->b);
            if (rec_bits(p->a) == 0ull) p->a.z = p->b.z;   // the rows of the window are then all of the second word
        } else {
            const uint4* rec = g.rec + (size_t)b * g.words + p->w;
            p->a = __ldg(rec);
            if (p->two) p->b = __ldg(rec + 1);
        }
    }
    // Rows of the cells x0 .. x0 + count - 1 (count <= 3): neighbouring bits of a window that may straddle two words, and
    // rows are numbered along the line, so the row of a set cell is the row of the window's first cell plus the set
    // cells before it.
    __device__ __forceinline__ void finish(int, int, int, int x0, int count, const Probe& p, int (&rows)[3]) const {
        const int lo = x0 < 0 ? 0 : x0;
        const int sh = lo & 63;
        const unsigned long long a = rec_bits(p.a), b = p.two ? rec_bits(p.b) : 0ull;
        const unsigned long long window = sh ? (a >> sh) | (b << (64 - sh)) : a;
        const int base = (int)p.a.z + __popcll(a & ((1ull << sh) - 1ull));
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int x = x0 + e, pos = x - lo;
            const bool set = e < count && x >= 0 && x < g.X && ((window >> pos) & 1ull);
            rows[e] = set ? base + __popcll(window & ((1ull << pos) - 1ull)) : -1;
        }
    }
};

// The same through the x-grouped table: the three x-neighbours lie in at most two 32-byte buckets.
struct BucketIndex {
    Buckets t;
    int Z, Y, X;
    struct Probe { uint4 lo[2], hi[2]; uint32_t key[2]; };
    __device__ __forceinline__ uint32_t cell(int z, int y, int x) const { return ((uint32_t)z * Y + y) * X + x; }
    __device__ __forceinline__ void probe_first(int b, int z, int y, int x0, int count, bool on, Probe* p) const {
        const int lo = x0 < 0 ? 0 : x0, hi = x0 + count - 1 >= X ? X - 1 : x0 + count - 1;
        const uint32_t* base = t.data + (size_t)b * t.cap * 8;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            p->lo[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
            p->hi[i] = make_uint4(kEmpty, 0u, 0u, 0u);
            p->key[i] = kEmpty;
            if (!on || lo > hi) continue;
            p->key[i] = cell(z, y, i == 0 ? lo : hi) >> 2;
            if (i == 1 && p->key[1] == p->key[0]) {
                p->key[1] = kEmpty;
                continue;
            }
            // the whole 32-byte bucket with one 256-bit load (one request to L1 instead of two)
            asm volatile("ld.global.nc.v8.u32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                         : "=r"(p->lo[i].x), "=r"(p->lo[i].y), "=r"(p->lo[i].z), "=r"(p->lo[i].w), "=r"(p->hi[i].x),
                           "=r"(p->hi[i].y), "=r"(p->hi[i].z), "=r"(p->hi[i].w)
                         : "l"(base + (size_t)hash_slot(p->key[i], t.shift) * 8));
        }
    }
    __device__ __forceinline__ void probe_second(int b, Probe* p) const {   // first slot taken by another group: keep probing
        const uint32_t* base = t.data + (size_t)b * t.cap * 8;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (p->key[i] == kEmpty || p->hi[i].x == p->key[i]) continue;
            uint32_t h = hash_slot(p->key[i], t.shift);
            uint4 lo = make_uint4(~0u, ~0u, ~0u, ~0u);
            uint32_t cur = p->hi[i].x;
            for (uint32_t probe = 1; probe < t.cap && cur != kEmpty; ++probe) {
                h = (h + 1) & (t.cap - 1);
                const uint4* bk = reinterpret_cast<const uint4*>(base + (size_t)h * 8);
                cur = __ldg(bk + 1).x;
                if (cur == p->key[i]) {
                    lo = __ldg(bk);
                    break;
                }
            }
            p->lo[i] = lo;
        }
    }
    static __device__ __forceinline__ int pick(const uint4& v, uint32_t i) {
        return (int)(i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)));
    }
    __device__ __forceinline__ void finish(int, int z, int y, int x0, int count, const Probe& p, int (&rows)[3]) const {
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const int x = x0 + e;
            rows[e] = -1;
            if (e >= count || x < 0 || x >= X || p.key[0] == kEmpty) continue;
            const uint32_t key = cell(z, y, x);
            rows[e] = pick((key >> 2) == p.key[0] ? p.lo[0] : p.lo[1], key & 3u);
        }
    }
};

template <class Index>
struct MapIndexOf;
template <>
struct MapIndexOf<BitsIndex> {
    static constexpr int BLOCKS = 2;
    static __device__ __forceinline__ BitsIndex make(const MapJob& j) { return BitsIndex{j.in}; }
};
template <>
struct MapIndexOf<BucketIndex> {
    static constexpr int BLOCKS = 1;       // the six buckets of a kz plane need more registers
    static __device__ __forceinline__ BucketIndex make(const MapJob& j) {
        return BucketIndex{j.table, j.g.in_shape[0], j.g.in_shape[1], j.g.in_shape[2]};
    }
};

template <class Index>
__global__ void __launch_bounds__(kMapThreads, MapIndexOf<Index>::BLOCKS)
map_rows_kernel(const __grid_constant__ MapJobs jobs, int batch, int max_voxels, int tiles_per_frame, TailRows tails) {
    pdl_enter();
    zero_tails(tails);
    extern __shared__ __align__(16) uint8_t map_smem[];
    MapShared& s = *reinterpret_cast<MapShared*>(map_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int windows = (max_voxels + kWindow - 1) / kWindow;
    const int per_job = batch * windows, items = per_job * jobs.count;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int ji = it / per_job;
        const MapJob& job = jobs.job[ji];
        const ConvGeom& g = job.g;
        const Index in = MapIndexOf<Index>::make(job);
        const int b = (it - ji * per_job) / windows;
        const int w0 = (it - ji * per_job - b * windows) * kWindow;
        int n = __ldg(job.out_num + b);
        n = (n > max_voxels ? max_voxels : n) - w0;          // rows of this window
        if (n <= 0) continue;
        n = n > kWindow ? kWindow : n;
        const int K0 = g.K[0], K1 = g.K[1], K2 = g.K[2];
        __syncthreads();                                     // the previous window has been written out
        for (int e = tid; e < 64 * kGroups / 2; e += kMapThreads) reinterpret_cast<uint32_t*>(s.count)[e] = 0u;
        if (tid < kWindow / 128) s.tile[tid] = 0u;
        __syncthreads();
        // entries of this thread's rows, and the rows' offsets
        uint32_t mask[2], rank[2], bin[2];
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const int r = tid + i * kMapThreads;
            const bool live = r < n;
            int4 c = make_int4(0, 0, 0, 0);
            if (live) c = __ldg(reinterpret_cast<const int4*>(job.out_coors) + (size_t)b * max_voxels + w0 + r);
            const int bz = c.y * g.S[0] - g.P[0], by = c.z * g.S[1] - g.P[1], bx = c.w * g.S[2] - g.P[2];
            uint32_t bits = 0;
#pragma unroll
            for (int kz = 0; kz < 3; ++kz) {
                if (kz >= K0) break;
                const int z = bz + kz;
                const bool z_ok = live && z >= 0 && z < g.in_shape[0];
                typename Index::Probe pb[3];
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) {
                    if (ky >= K1) break;
                    const int y = by + ky;
                    in.probe_first(b, z, y, bx, K2, z_ok && y >= 0 && y < g.in_shape[1], &pb[ky]);
                }
#pragma unroll
                for (int ky = 0; ky < 3; ++ky)
                    if (ky < K1) in.probe_second(b, &pb[ky]);
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) {
                    if (ky >= K1) break;
                    int rows3[3];
                    in.finish(b, z, by + ky, bx, K2, pb[ky], rows3);
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx) {
                        if (kx >= K2) break;
                        const int k = (kz * K1 + ky) * K2 + kx;
                        s.ids[k][r] = rows3[kx];
                        bits |= (rows3[kx] >= 0 ? 1u : 0u) << k;
                    }
                }
            }
            uint32_t key = 64u;                              // dead rows (the frame's last window): they stay behind
            if (live) {
                key = 0u;
                if (job.order)
#pragma unroll
                    for (int q = 0; q < 6; ++q) key = key << 1 | ((bits & job.plane[q]) ? 1u : 0u);
            }
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
            const uint32_t before = __popc(peers & ((1u << lane) - 1u));
            if (live && before == 0u) s.count[key][warp + i * (kMapThreads / 32)] = (uint16_t)__popc(peers);
            if (i == 0) mask[0] = bits, rank[0] = before, bin[0] = key;
            else mask[1] = bits, rank[1] = before, bin[1] = key;
        }
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
        for (int i = 0; i < 2; ++i) {
            s.src[pos[i]] = (uint16_t)(tid + i * kMapThreads);
            if (mask[i]) atomicOr(&s.tile[pos[i] >> 7], mask[i]);
        }
        __syncthreads();
        // write-out: a warp takes 32 positions of a tile
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            const int p = tid + i * kMapThreads;
            const int tile0 = p & ~127;
            if (tile0 >= n) break;                           // a tile without rows (uniform over the warp)
            uint32_t m = s.tile[p >> 7];
            if ((p & 127) == 0) job.tile_mask[(size_t)b * tiles_per_frame + ((w0 + p) >> 7)] = m;
            // a consumer that fetches `group` offsets at a time wants all of them as soon as it wants one
            if (job.group >= 2) m |= (m & 0x55555555u) << 1 | ((m >> 1) & 0x55555555u);
            if (job.group >= 4) m |= (m & 0x33333333u) << 2 | ((m >> 2) & 0x33333333u);
            const int r = s.src[p];
            if (job.order && p < n) job.order[(size_t)b * max_voxels + w0 + p] = w0 + r;
            int32_t* out = job.nbr + nbr_index(g.kvol, max_voxels, b, 0, w0 + p);
#pragma unroll
            for (int k = 0; k < kMapKvol; ++k) {
                if (k >= g.kvol) break;
                if ((m >> k) & 1u) out[k * kNbrRun] = p < n ? s.ids[k][r] : -1;
            }
        }
    }
}

template <class Index>
int launch_maps(const char* name, const MapJobs& jobs, int batch, int max_voxels, const TailRows& tails, cudaStream_t stream) {
    static_assert(MapIndexOf<BitsIndex>::BLOCKS * (sizeof(MapShared) + 1024) <= 228 * 1024, "two windows per SM");
    // the attribute belongs to the device's context: set it once per device (repeating it is harmless)
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    SESSD_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        SESSD_CUDA(cudaFuncSetAttribute(map_rows_kernel<Index>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)sizeof(MapShared)));
        configured.fetch_or(bit, std::memory_order_release);
    }
    const int64_t items = (int64_t)jobs.count * batch * ((max_voxels + kWindow - 1) / kWindow);
    const int most = persistent_grid(MapIndexOf<Index>::BLOCKS);
    SESSD_LAUNCH_NAMED(name, map_rows_kernel<Index>, (int)(items < most ? items : most), kMapThreads, sizeof(MapShared), stream,
                       jobs, batch, max_voxels, (max_voxels + 127) / 128, tails);
    return SESSD_OK;
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

int launch_map_rows(const MapJobs& jobs, int batch, int max_voxels, const TailRows& tails, cudaStream_t stream) {
    if (jobs.count == 0) return SESSD_OK;
    if (jobs.job[0].table.data) return launch_maps<BucketIndex>("map_rows<table>", jobs, batch, max_voxels, tails, stream);
    return launch_maps<BitsIndex>("map_rows<grid>", jobs, batch, max_voxels, tails, stream);
}

}  // namespace sessd
