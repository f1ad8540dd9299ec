// Shared host/device helpers of the sparse front end library (sm_100a only).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <vector>

#include "sessd.h"

namespace sessd {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;   // empty key / unset rank in a coordinate table
constexpr size_t kAlign = 256;             // sub-buffer alignment inside a workspace
constexpr int kStatusInts = 256;           // status block: 1 KB; word 0 is the status, bytes 256.. hold 64 pair counters
constexpr int kThreads = 256;
constexpr int kMaxBatch = 4096;

// ---- host side ---------------------------------------------------------------------------

extern std::atomic<uint64_t> g_launches;
void set_cuda_error(cudaError_t e, const char* what);

// Optional per-launch timing: while a recorder is installed on the calling thread, every launch
// made through SESSD_LAUNCH is bracketed by two events on its stream.
struct StageRecorder {
    std::vector<cudaEvent_t> events;   // 2 per launch
    std::vector<const char*> names;
    void before(cudaStream_t s);
    void after(const char* name, cudaStream_t s);
};
extern thread_local StageRecorder* g_recorder;

#define SESSD_CUDA(call)                                   \
    do {                                                   \
        cudaError_t e__ = (call);                          \
        if (e__ != cudaSuccess) {                          \
            ::sessd::set_cuda_error(e__, #call);           \
            return SESSD_ERR_CUDA;                         \
        }                                                  \
    } while (0)

// Cleared for the scope of a pipeline run with several stream slots: the blocks of a waiting kernel would hold registers
// and shared memory that another slot's running kernel can use (128 frames x 120,000 points on two slots: 40.1 ms with
// overlapping launches, 37.9 without).
extern thread_local bool g_overlap_launches;

// Launches `kernel` so that its blocks may start while the stream's previous kernel still runs (programmatic dependent
// launch): what a kernel reads or writes of earlier kernels' data comes after its pdl_enter() / pdl_wait(). Launching
// costs about the same, but a kernel's start-up then overlaps its predecessor's last blocks: of the 40 short kernels
// of a single 20,000-point frame each used to leave the GPU idle for a microsecond or more.
template <typename... P, typename... A>
inline cudaError_t launch_kernel(bool overlap, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap && g_overlap_launches ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Launches `kernel` and accounts for it under `name`; returns from the caller on a launch error.
#define SESSD_LAUNCH_IMPL(overlap, name, kernel, grid, block, smem, stream, ...)                                       \
    do {                                                                                                               \
        if (::sessd::g_recorder) ::sessd::g_recorder->before(stream);                                                  \
        const cudaError_t e_launch__ =                                                                                 \
            ::sessd::launch_kernel((overlap), kernel, (grid), (block), (smem), (stream), __VA_ARGS__);                 \
        ::sessd::g_launches.fetch_add(1, std::memory_order_relaxed);                                                   \
        if (::sessd::g_recorder) ::sessd::g_recorder->after(name, stream);                                             \
        SESSD_CUDA(e_launch__);                                                                                        \
    } while (0)
#define SESSD_LAUNCH_NAMED(name, kernel, grid, block, smem, stream, ...) \
    SESSD_LAUNCH_IMPL(true, name, kernel, grid, block, smem, stream, __VA_ARGS__)
#define SESSD_LAUNCH(kernel, grid, block, smem, stream, ...) \
    SESSD_LAUNCH_IMPL(true, #kernel, kernel, grid, block, smem, stream, __VA_ARGS__)

// A workspace's status word by synchronisation and copy: allocates nothing (sessd_read_status: pinned memory for a thread's first call).
int copy_status(const void* workspace, cudaStream_t stream);

// Number of SMs of the current device (cached per device).
int sm_count();
// Grid for a persistent grid-stride kernel: `per_sm` blocks on every SM.
inline int persistent_grid(int per_sm) { return sm_count() * per_sm; }

// Two-pass workspace layout: with base == nullptr it only measures.
// A caller's workspace must start on a kAlign boundary (cudaMalloc and TensorRT workspaces do): the kernels use
// 16- and 32-byte vector accesses relative to it.
inline bool workspace_aligned(const void* p) { return reinterpret_cast<uintptr_t>(p) % kAlign == 0; }

struct Bump {
    char* base;
    size_t off;
    explicit Bump(void* b) : base(static_cast<char*>(b)), off(0) {}
    template <typename T>
    T* take(size_t count) {
        off = (off + kAlign - 1) / kAlign * kAlign;
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += count * sizeof(T);
        return p;
    }
    size_t total() const { return (off + kAlign - 1) / kAlign * kAlign; }
};

inline uint32_t pow2_at_least(uint64_t v) {
    uint32_t c = 64;
    while (c < v) c <<= 1;
    return c;
}
inline int ilog2(uint32_t v) {
    int l = 0;
    while ((1u << l) < v) ++l;
    return l;
}

// One open-addressing coordinate table per frame: frame b owns slots [b*cap, (b+1)*cap).
// keys: linear cell index inside the frame's grid, kEmpty when free.
// vals: row index of the key, -1 when the key has no row.
struct Table {
    uint32_t* keys;
    int32_t* vals;
    uint32_t cap;       // power of two
    int shift;          // 32 - log2(cap)
};

// The voxeliser's table. A slot is (point that claimed the cell) << 32 | key, ~0 when free; the cell's other points are listed
// under the claiming point. Most cells have one point, so that little beside the slots is touched at random, and what
// belongs to a point lies in point order.
struct VoxelTable {
    unsigned long long* slots;   // [B][cap]
    uint32_t* lists;             // [B][max_points][max_points_per_voxel], ascending, kEmpty when free
    uint32_t cap;                // power of two
    int shift;                   // 32 - log2(cap)
};

// x-grouped coordinate table of one resolution level: frame b owns buckets [b*cap, (b+1)*cap), a
// bucket is 8 words = {row of cell x&3 == 0..3, group key (cell index >> 2), 3 unused}; all words are
// 0xFFFFFFFF when free.
struct Buckets {
    uint32_t* data;
    uint32_t cap;   // buckets per frame, power of two
    int shift;      // 32 - log2(cap)
};

// Occupancy grid of one resolution level. Word w of a frame covers the 64 cells x = 64*(w % xw) .. +63 of line
// (z, y) = w / xw. Rows are numbered in word order, i.e. in (z, y, x) order.
// One level (top == nullptr): frame b owns records [b*words, (b+1)*words), record w = {bits lo, bits hi, rows before this
// word, first two cells of the line's next word} of word w.
// Two levels (the voxeliser's level, whose words are nearly all empty): top record w / 64 = {bits lo, bits hi, occupied
// words before, unused} says which of 64 words are occupied, and frame b's records [b*words, ..) hold the occupied words
// alone, in order: {bits lo, bits hi, rows before this word, w}.
struct BitGrid {
    uint4* rec;
    int Z, Y, X;
    int xw;      // words per x line
    int words;   // records per frame
    uint4* top;
    int top_words;   // top records per frame
};
inline BitGrid bitgrid_shape(const int shape[3]) {
    BitGrid g{};
    g.Z = shape[0], g.Y = shape[1], g.X = shape[2];
    g.xw = (g.X + 63) / 64;
    g.words = g.Z * g.Y * g.xw;
    return g;
}

// Neighbour maps are tile-major: [frame][tile of 128 output rows][kernel offset][kNbrRun], entry (k, o) of a frame
// holding the input row under offset k of output row o, or -1. All offsets of a tile lie side by side, kNbrRun
// words apart (the 128 entries and 16 bytes of padding), which is also how the tensor-core kernel keeps them in
// shared memory: the offsets of one of its stages arrive with a single copy, already spaced for its index reads.
constexpr int kNbrRun = 132;
__host__ __device__ inline size_t nbr_frame_words(int kvol, int max_voxels) {
    return (size_t)((max_voxels + 127) / 128) * kvol * kNbrRun;
}
__host__ __device__ inline size_t nbr_index(int kvol, int max_voxels, int b, int k, int o) {
    return (size_t)b * nbr_frame_words(kvol, max_voxels) + ((size_t)(o >> 7) * kvol + k) * kNbrRun + (o & 127);
}
// The padding behind a tile's first offset holds four words, for each 32 of its rows a mask of offsets: at least those that any of
// the 32 has a neighbour under (all ones where a map's builder does not say; bits that the tile's mask lacks mean nothing).
// (map_tiles_kernel writes them where a call has room for more than kRunRows rows: conv_rows.cu, which reads them, takes no others.)
constexpr int kRunRows = 300000;
__host__ __device__ inline size_t nbr_runs_index(int kvol, int max_voxels, int b, int o) {
    return nbr_index(kvol, max_voxels, b, 0, o & ~127) + 128 + ((o >> 5) & 3);
}

// Geometry of one sparse convolution (z, y, x order everywhere).
struct ConvGeom {
    int K[3], S[3], P[3];
    int dil;
    int in_shape[3];
    int out_shape[3];
    int kvol;
    int span_max[3];  // most candidate outputs one input can have per axis
    int ncand;        // product of span_max
};

// ---- device side -------------------------------------------------------------------------

// Every kernel of the library is launched with programmatic serialisation (launch_kernel above), so it may start before
// the stream's previous kernel has finished. pdl_wait() returns when that kernel has completed and its writes can be
// seen; pdl_release() allows the next kernel to start. A kernel releases only after its own wait: when a kernel runs,
// everything before its predecessor is therefore complete, and it may read that even before its own wait.
// What the predecessor itself has written (and, in a call's first kernel, any input) must not be read as a constant right behind the
// wait: __ldg and reads through const __restrict__ parameters may be moved ahead of it by the compiler (seen with a tile's mask, which
// came back as the call before had left it). Such a read is a load_late, unless what it reads or whether it is made depends on a
// value that came from one.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
    pdl_wait();
    pdl_release();
}

__device__ __forceinline__ int load_late(const int32_t* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t load_late(const uint32_t* p) { return (uint32_t)load_late(reinterpret_cast<const int32_t*>(p)); }
__device__ __forceinline__ float load_late(const float* p) { return __int_as_float(load_late(reinterpret_cast<const int32_t*>(p))); }
__device__ __forceinline__ __half load_late(const __half* p) {
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return __ushort_as_half(v);
}
__device__ __forceinline__ uint4 load_late(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t hash_slot(uint32_t key, int shift) {
    return (key * 0x9E3779B1u) >> shift;
}

// Finds or claims the slot of `key`. Returns the slot index inside the frame's table or -1
// when `cap` probes found neither the key nor a free slot.
__device__ __forceinline__ int table_insert(uint32_t* keys, uint32_t cap, int shift, uint32_t key) {
    uint32_t h = hash_slot(key, shift);
    for (uint32_t probe = 0; probe < cap; ++probe) {
        uint32_t cur = keys[h];
        if (cur == key) return (int)h;
        if (cur == kEmpty) {
            uint32_t old = atomicCAS(&keys[h], kEmpty, key);
            if (old == kEmpty || old == key) return (int)h;
        }
        h = (h + 1) & (cap - 1);
    }
    return -1;
}

__device__ __forceinline__ int table_find(const uint32_t* __restrict__ keys, uint32_t cap, int shift, uint32_t key) {
    uint32_t h = hash_slot(key, shift);
    for (uint32_t probe = 0; probe < cap; ++probe) {
        uint32_t cur = __ldg(&keys[h]);
        if (cur == key) return (int)h;
        if (cur == kEmpty) return -1;
        h = (h + 1) & (cap - 1);
    }
    return -1;
}

// Exclusive prefix sum of `v` over the block (blockDim.x == kThreads); *total gets the block sum.
__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
    __shared__ int warp_sums[kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += t;
    }
    __syncthreads();  // protects warp_sums against a previous call
    if (lane == 31) warp_sums[wid] = incl;
    __syncthreads();
    int base = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        int s = warp_sums[w];
        if (w < wid) base += s;
        sum += s;
    }
    *total = sum;
    return base + incl - v;
}

__device__ __forceinline__ int block_sum(int v) {
    int total;
    block_exclusive_scan(v, &total);
    return total;
}

// ---- pieces shared between translation units --------------------------------------------

// One launch for the resets a call needs. Range r is n16[r] 16-byte words at ptr[r] (16-byte aligned), 0xFF bytes when
// ones[r] is set, else zeros; unused ranges have n16 = 0. status: words status_from .. kStatusInts - 1 of the status
// block to zero, or null.
struct FillRanges {
    static constexpr int kMax = 5;
    uint4* ptr[kMax];
    size_t n16[kMax];
    int ones[kMax];
    int32_t* status;
    int status_from;
};
// Output tensors [batch][max_rows][row_bytes] whose rows from min(counts[b], most) on are to be zero (row_bytes % 2 == 0;
// null: unused).
struct TailRows {
    static constexpr int kMax = 3;
    void* tensor[kMax];
    int row_bytes[kMax];
    const int32_t* counts;
    int batch, max_rows, most;
};
// overlap: whether the launch may start while the stream's previous kernel runs (see its definition)
int launch_prepare(const FillRanges& f, const TailRows& t, bool overlap, cudaStream_t stream);
int launch_fill_zero(void* ptr, size_t bytes, cudaStream_t stream);  // bytes % 16 == 0, ptr 16-byte aligned

// What a one-pass numbering kernel (scan.cuh) keeps in global memory: a word per chunk of kThreads entries and a ticket
// counter; all zero before the kernel.
struct ScanState {
    unsigned long long* state;   // [batch][scan_chunks(entries)]
    uint32_t* ticket;
};
__host__ __device__ inline int scan_chunks(int entries) { return (entries + kThreads - 1) / kThreads; }
// Bytes of the state of a numbering of `entries` per frame (a multiple of 16; the last word is the ticket counter), and
// that state at p.
inline size_t scan_state_bytes(int entries, int batch) {
    return ((size_t)batch * scan_chunks(entries) + 2) / 2 * 2 * sizeof(unsigned long long);
}
inline ScanState scan_state_at(char* p, int entries, int batch) {
    if (!p) return ScanState{nullptr, nullptr};
    return ScanState{reinterpret_cast<unsigned long long*>(p),
                     reinterpret_cast<uint32_t*>(p + scan_state_bytes(entries, batch) - sizeof(unsigned long long))};
}

// rulebook.cu
int conv_geom_from_params(const sessd_conv_params* p, ConvGeom* g);
int launch_table_build(const int32_t* coors, const int32_t* voxel_num, int batch, int max_voxels, const int shape[3],
                       const Table& t, int32_t* status, cudaStream_t stream);
int launch_nbr_build(const int32_t* out_coors, const int32_t* out_num, int batch, int max_voxels, const ConvGeom& g,
                     const Table& in_table, int32_t* nbr, cudaStream_t stream);
// Strided layers: set the bit of every candidate output, then number the set bits in (z, y, x) order.
int launch_mark_outputs(const int32_t* in_coors, const int32_t* in_num, int batch, int max_voxels, const ConvGeom& g,
                        const BitGrid& out, cudaStream_t stream);
bool derivable_in_x(const ConvGeom& g);
// Their maps by input rows, once the outputs are numbered; tile_mask zero before. Where the rule says so.
bool scatter_rows_usable(const ConvGeom& g, int64_t rows);   // rows: capacity of the call
int launch_scatter_rows(const int32_t* in_coors, const int32_t* in_num, const int32_t* out_num, int batch, int max_voxels,
                        const ConvGeom& g, const BitGrid& out, int32_t* nbr, uint32_t* tile_mask, const TailRows& tails,
                        cudaStream_t stream);

// The levels that a chain of strided layers makes from the voxeliser's level, when the occupancy of all of them follows
// word by word from the voxeliser's grid (level_chain_usable): marked by one kernel and numbered by one.
struct LevelChain {
    static constexpr int kMax = 6;
    int count;
    BitGrid grid[kMax];
    ConvGeom geom[kMax];                 // of the layer that makes the level
    unsigned long long* state[kMax];     // numbering state
    int32_t* coors[kMax];
    int32_t* num[kMax];
    uint32_t* ticket;
    int32_t* totals;                     // [B][kMax] rows of a level before the cut at max_voxels
    uint32_t* done;                      // [B] chunks numbered
};
bool level_chain_usable(const ConvGeom* geoms, int count);
// What the voxeliser's point lists are made from (voxel_grid.cu).
struct PointLists {
    const int32_t* points_size;
    const uint32_t* pt_key;
    uint32_t* lists;
    BitGrid grid;
    int max_points, max_pts;
};
int launch_number_levels(const LevelChain& chain, int batch, int max_voxels, const PointLists& lists, int32_t* status,
                         cudaStream_t stream);
int launch_bucket_build(const int32_t* coors, const int32_t* voxel_num, int batch, int max_voxels, const int shape[3],
                        const Buckets& t, const ConvGeom* mark, const BitGrid& out, int32_t* status, cudaStream_t stream);
// map_rows.cu: neighbour maps + tile masks of layers (any kernel up to 3x3x3, any stride) whose input level has an
// occupancy grid (`in`: launch_map_windows, one launch for up to MapJobs::kMax layers) or an x-grouped table of its rows
// (`table`: launch_map_tiles).
struct MapJob {
    const int32_t* out_coors;
    const int32_t* out_num;
    ConvGeom g;
    BitGrid in;
    Buckets table;
    int32_t* nbr;
    uint32_t* tile_mask;
    int32_t* order;      // [B][max_voxels] output row at each position of the map, or null: positions are rows
    int shape;           // kernel size as K0 K1 K2
    int group;           // offsets that the map's consumers fetch together
    uint32_t plane[6];   // offsets of the kernel's outer planes: first and last in z, y, x
};
struct MapJobs {
    static constexpr int kMax = 8;
    MapJob job[kMax];
    int count;
};
// Everything of a job but its index; cin: input channels of the layers that read the map (the smallest).
MapJob make_map_job(const ConvGeom& g, const int32_t* out_coors, const int32_t* out_num, int cin, int32_t* nbr,
                    uint32_t* tile_mask, int32_t* order);
struct RowMeans;
int launch_map_windows(const MapJobs& jobs, int batch, int max_voxels, const RowMeans& means, cudaStream_t stream);
int launch_map_tiles(const MapJob& job, int batch, int max_voxels, const TailRows& tails, cudaStream_t stream);
int launch_tile_mask(const int32_t* nbr, const int32_t* out_num, int batch, int max_voxels, int kvol,
                     uint32_t* tile_mask, cudaStream_t stream);
// conv_simt.cu
struct ConvLaunch {
    const void* in;        // [B][max_voxels][Cin]
    void* out;             // [B][max_voxels][Cout]
    const int32_t* nbr;    // neighbour map, tile-major (nbr_index); only the offsets that tile_mask names are written
    const int32_t* order;  // [B][max_voxels] output row at each position of the map, or null: positions are rows
    const int32_t* out_num;// [B]
    const uint32_t* tile_mask; // [B][ceil(max_voxels/128)]: bit k set when offset k has a neighbour in the tile
    const void* weights;   // [kvol][Cin][Cout] in the feature dtype
    const void* umma_weights; // fp16 weights pre-tiled for the tensor-core kernel, or null
    const float* scale;    // [Cout] or null
    const float* shift;    // [Cout] or null
    int relu;
    int batch, max_voxels, kvol, cin, cout, dtype, subm;
    int64_t most_rows;     // no more rows than this can be in use, all frames together
    // Optional fused BEV scatter (last layer): when dense != null the result row is also written to
    // dense[b][c*D + z][y][x] using out_coors.
    void* dense;
    const int32_t* out_coors;
    int D, H, W;
    int32_t* status;       // device status word (tensor-core path reports wait timeouts there)
    int* tile_counter;     // tensor-core path: zero before the launch; hands out the tiles of the few-tiles path
    int maps_ready;        // neighbour map, masks and row counts are older than the kernel launched just before
    int debug_withhold_weights;   // tests only: whoever streams the weights stays silent (waits run out)
    int weights_finite;           // every weight is a finite number of the feature dtype
    const float* scale_host;      // [Cout <= 64] host copies of scale / shift (ones / zeros without batch norm), or null
    const float* shift_host;
};
int launch_conv_simt(const ConvLaunch& c, cudaStream_t stream);
bool conv_simt_supported(int cin, int cout);

// conv_rows.cu (narrow layers of calls with many rows: a warp per 64 positions of the map)
bool conv_rows_takes(const ConvLaunch& c);
int launch_conv_rows(const ConvLaunch& c, cudaStream_t stream);

// conv_f32.cu (fp32 storage, a register tile per warp)
bool conv_f32_supported(int cin, int cout, int kvol);
int launch_conv_f32(const ConvLaunch& c, cudaStream_t stream);

// conv_umma.cu (tcgen05 implicit GEMM, fp16 storage)
bool conv_umma_supported(int cin, int cout);
int conv_umma_pack_weights(const float* weights, int kvol, int cin, int cout, void** device_out);
int launch_conv_umma(const ConvLaunch& c, cudaStream_t stream);

// sparse2dense.cu
int launch_sparse2dense(const void* feat, const int32_t* coors, const int32_t* voxel_num, int batch, int max_voxels,
                        int C, int D, int H, int W, int top, int bottom, int left, int right, int dtype, void* dense,
                        cudaStream_t stream);
// [planes][H][W] -> [planes][top+H+bottom][left+W+right], zero border.
int launch_zero_pad2d(const void* in, void* out, size_t planes, int H, int W, int top, int bottom, int left, int right,
                      int dtype, cudaStream_t stream);

// voxelize.cu
struct VoxelWorkspace {
    int32_t* status;
    VoxelTable table;
    int32_t* pt_claim;    // [B][max_points] the point that claimed the point's cell, -1 outside the range
    ScanState scan;       // numbering of the owner points
    void* zero_base;      // the scan's words, to be zero before a call
    size_t zero_bytes;
    int32_t* num_points;  // [B][max_voxels]
    size_t table_bytes;   // bytes to set to 0xFF before a call (slots and lists)
    void* table_base;
};
void voxel_workspace_layout(Bump& bump, const sessd_voxel_params* p, int batch, int max_points, VoxelWorkspace* w);
// The points of a batch -> rows; the caller has reset the table, the scan's words and the status (and, for a call that
// returns whole tensors, the rows past each frame's point count). zero_tail: also zero the rows between a frame's voxel
// count and its point count.
int voxelize_run(const sessd_voxel_params* p, int batch, int max_points, int out_dtype, const float* points,
                 const int32_t* points_size, void* voxels, int32_t* coors, int32_t* voxel_num, const VoxelWorkspace& w,
                 bool zero_tail, cudaStream_t stream);

int launch_number_outputs(const BitGrid& out, int batch, int max_voxels, const ScanState& scan, int32_t* out_coors,
                          int32_t* out_num, int32_t* status, cudaStream_t stream);

// voxel_grid.cu: rows in (z, y, x) order and an occupancy grid of the level
struct VoxelGrid {
    BitGrid grid;
    uint32_t* pt_key;     // [B][max_points]
    uint32_t* lists;      // [B][max_points][max_points_per_voxel], by row
    int32_t* word_num;    // [B] occupied words
    ScanState scan_words, scan_rows;
    void* zero_base;      // to be zero before a call
    size_t zero_bytes;
};
bool voxel_grid_usable(const sessd_voxel_params* p, int max_points, const int level_shape[3]);
void voxel_grid_layout(Bump& bump, const sessd_voxel_params* p, const int level_shape[3], int batch, int max_points,
                       VoxelGrid* w);
// Points -> rows, their point lists, and the levels of `chain` (count 0: none). The rows' means follow with
// launch_map_windows.
int voxel_grid_run(const sessd_voxel_params* p, int batch, int max_points, const float* points, const int32_t* points_size,
                   int32_t* coors, int32_t* voxel_num, const VoxelGrid& w, const LevelChain& chain, int32_t* status,
                   cudaStream_t stream);
// What launch_map_windows does besides: the means of the voxeliser's rows (points == nullptr: nothing).
struct RowMeans {
    const float4* points;
    const int32_t* voxel_num;
    const uint32_t* lists;
    void* voxels;
    int max_points, max_pts, half;
};

struct sessd_conv_weights_impl {
    void* w;        // device, [kvol][Cin][Cout] in dtype
    void* umma_w;   // device, tensor-core tiling of the same weights (fp16) or null
    float* scale;   // device or null
    float* shift;   // device or null
    int relu, dtype, kvol, cin, cout;
    int finite;           // every weight is a finite number of dtype
    int debug_withhold;   // tests of the time-out path: whoever streams the weights stays silent
    // host copies of scale and shift (ones and zeros without batch norm) for kernels that take them as launch
    // parameters; filled for out_channel <= 64
    float host_scale[64], host_shift[64];
};

}  // namespace sessd
