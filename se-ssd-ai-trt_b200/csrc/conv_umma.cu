// Sparse convolution as an implicit GEMM on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// Replaces, for fp16 features and 16/32/64 channels, the reference's per-offset scalar kernel
// (submConv3dlayer.cu:479-518, launched kvol times per layer, :632-638). A tile is 128 output rows. For
// every group of kernel offsets ("stage": 64/Cin offsets side by side) the 128 neighbour rows are gathered
// into shared memory as a K-major, 128-byte-swizzled A operand (one 128-byte row per output row, missing
// neighbours zero-filled), the matching pre-tiled weight block is streamed in as the B operand with a bulk
// asynchronous copy, and tcgen05.mma (M = 128, N = Cout, K = 16 x 4) accumulates into an fp32 accumulator in
// tensor memory that stays resident across all offsets. A CTA iteration ("group") covers four tiles with
// the offset loop outermost, so that a weight block is fetched once per four tiles; (tile, stage) pairs
// without any neighbour are skipped using the per-tile offset masks the rulebook kernels produce. The
// epilogue reads the accumulator with tcgen05.ld, applies the folded BatchNorm scale/shift and ReLU, and
// stores fp16 rows (and, for the last layer, scatters them into the dense BEV map). Layers of few tiles, and those with the scatter,
// go through a path of their own (umma_few) instead of groups.
//
// One persistent CTA per SM; every role has warps of its own and walks the same sequence of groups:
//   warps 0-3    epilogue (warp w reads tensor-memory lanes 32w .. 32w+31). The accumulators are double
//                buffered (2 sets x 4 tiles x Cout columns), so the epilogue of one group runs while the
//                other roles are already working on the next group. A thread holds one row and stores it 32 bytes
//                at a time; 64 -> 64 channels with many offsets go through a small staging area of the warp.
//   warps 4-7    MMA issuers; issuer t owns tile t of every group. The warp works out the group's schedule
//                once (lane g for stage g); it goes through it together, or with 64 input channels one elected lane alone,
//                and that lane issues the tcgen05.mma and commit instructions (each costs its thread on the order of a
//                hundred cycles, so four share).
//   warp  8      streams the weight blocks (cp.async.bulk) into a three-slot ring.
//   warp  9      prefetches the neighbour indices of upcoming (tile, stage) items into a ring of index blocks
//                with bulk copies, sixteen items side by side (one lane each), two to three slot cycles ahead.
//   warps 10..   gather. The A ring has one 16 KB slot per gather warp: item q (the q-th (tile, stage) pair
//                of the CTA's life) lives in slot q % NSLOT and is filled by warp q % NSLOT alone with
//                sixteen-byte cp.async copies that publish the slot themselves (mbarrier arrival of the
//                copies). With ten slots in flight the latency chain of one slot (issue, landing, MMA,
//                commit) is covered and no barrier is shared between gather warps.
// Every barrier has one waiting role that sees each of its phases in order (a parity wait is only safe
// then): a_full exists per (issuer, slot); index block j is always read by gather warp j % NSLOT.
// A CTA walks a contiguous range of the occupied row tiles, cut so that every CTA gets the same number of
// (tile, stage) items (row counts and masks are read on the device). Every wait is bounded by a clock limit,
// after which the CTA raises SESSD_STATUS_TIMEOUT (and reports which wait in the status block), stops issuing
// work, waits for its own copies and MMAs, frees its tensor memory and returns.
#include <atomic>
#include <cstring>
#include <string>
#include <vector>

#include "mbarrier.cuh"

namespace sessd {

namespace {

constexpr int TILE_M = 128;
constexpr int TILES = 4;                     // row tiles per group; they share each weight block
constexpr int EPI_WARPS = 4;                 // warps 0-3
constexpr int MMA_WARPS = TILES;             // warps 4-7: issuer t owns tile t
constexpr int WEIGHT_WARP = EPI_WARPS + MMA_WARPS;
constexpr int INDEX_WARP = WEIGHT_WARP + 1;
constexpr int FIRST_GATHER_WARP = INDEX_WARP + 1;
constexpr int NSLOT_MAX = 10;
constexpr int NIDX_MAX = 30;
constexpr int B_STAGES = 3;                  // weight ring: a group needs up to 27 blocks, each an L2 round trip away
constexpr int ROW_BYTES = 128;               // 64 halves per A/B row
constexpr int A_BYTES = TILE_M * ROW_BYTES;  // 16 KB
constexpr int KVOL_MAX = 27;
// Few-tiles path: up to this many tiles per CTA. It fetches a weight block per item instead of one for up to four tiles, but is
// through sooner, shares the tiles out by a counter and pays nothing for a group's boundary. The line lies where they cross, which
// depends on whether the rows of the map are ordered by their neighbours (a front end's) or not (a plugin call's: more items, and more of
// their rows missing neighbours, whose zeros groups leave out where they are still there). Layers in us (events around the launch),
// groups and this path, by tiles per CTA. Front ends:
//   16 -> 16  13 (3 x 120,000 points) 29 and 27, 17 33 and 33, 18 (20 x 20,000) 33 and 35, 26 43.5 and 45.5, 35 52 and 58
//   16 -> 32  8 23 and 23, 10 (5 x 20,000) 25 and 25, 12 27 and 29, 17 (2 x 120,000) 33 and 36, 26 41.5 and 48, 50 68 and 84
//   32 -> 32  20 (10 x 20,000) 60 and 57, 40 105 and 101, 64 158 and 152, 129 306 and 296, 193 453 and 458, 257 600 and 637; frames of 120,000:
//             17 56 and 54, 34 93 and 97, 51 136 and 138, 69 179 and 179, 103 265 and 261, 137 353 and 342
//   32 -> 64  14 (10 x 20,000) 48 and 45.5, 28 80 and 76, 45 115 and 112, 67 161 and 165, 90 210 and 218; frames of 120,000: 25 74 and 72, 58 152
//             and 148, 132 332 and 318
//   64 -> 64  11 (8 x 20,000) 66 and 58, 33 (8 x 120,000) 152 and 144, 67 293 and 277, 132 (32 x 120,000) 567 and 532, 197 842 and 791;
//             strided 12 58 and 54, 25 99 and 92, 49 180 and 170, 77 269 and 257
// Plugin calls:
//   16 -> 16  11 (12 x 20,000) 33 and 29, 18.5 43.5 and 39.4, 22 45.5 and 45.5, 31 58 and 60, 46 84.5 and 86.5
//   16 -> 32  12 (6 x 20,000) 31 and 29, 20 43.5 and 41.4, 24 to 43 the same, 64 107 and 109
//   32 -> 32  10 (5 x 20,000) 41.5 and 37.4, 24 76 and 74, 40 119 and 115, 64 177 and 177; frames of 120,000: 17 60 and 58, 34 103 and 104,
//             51 146 and 149.5
//   32 -> 64  8 (6 x 20,000) 39.4 and 37.4, 17 62 and 61, 25 84.5 and 84.5, 41 129.5 and 133.5
//   64 -> 64  11 (8 x 20,000) 74 and 66, 33 (8 x 120,000) 170 and 166, 66 322 and 318, 83 400 and 396, 132 633 and 621; strided 12 77 and 74, 25 131.5
//             and 131.5, 37 185 and 189, 49 238 and 246; strided, three offsets, 10 29 and 29, 21 41.5 and 45.5, 42 66 and 78
__host__ __device__ constexpr int few_tiles(int cin, int cout, bool subm, bool ordered) {
    if (ordered) return cin == 16 ? (cout == 16 ? 17 : 10) : (cin == 32 ? (cout == 32 ? 150 : 60) : 200);
    return cin == 16 ? 22 : (cin == 32 ? (cout == 32 ? 42 : 25) : (subm ? 130 : 20));
}
constexpr int FEW_SLOTS = 8;                 // few-tiles path: stages in flight, an A slot and a weight block each
// The slot of a gather warp there (-1: none). Warps 12 and 16 stay out: they share a scheduler, and its queue for shared-memory
// instructions, with the issuer.
__host__ __device__ constexpr int few_slot(int warp) {
    const int s = warp - 10 - (warp > 12 ? 1 : 0) - (warp > 16 ? 1 : 0);
    return warp >= 10 && warp != 12 && warp != 16 && s < FEW_SLOTS ? s : -1;
}
constexpr int FEW_IDX = 28;                  // offsets of a tile's index block there (27, and those of the last stage past them)
// Words from one offset's 128 indices to the next offset's inside an index block: 16 bytes more than the indices
// take, so that lanes reading different offsets of a stage (32- and 16-channel inputs) use different banks too.
constexpr int TAP_WORDS = kNbrRun;
static_assert(kNbrRun == TILE_M + 4, "the map's spacing between offsets is the index block's");

// Gather slots (= gather warps): as many as fit beside the weight ring, the index blocks and, with 64 -> 64 channels, the epilogue's
// staging area.
// The index ring is deeper than the A ring (index rows come from DRAM, several microseconds away under load):
// block j = q % NIDX, with NIDX a multiple of NSLOT so that block j is always read by gather warp j % NSLOT.
template <int CIN>
struct Ring {
    static constexpr int NSLOT = 10;
    static constexpr int NIDX = (CIN == 16 ? 2 : 3) * NSLOT;
    static constexpr int THREADS = (FIRST_GATHER_WARP + NSLOT) * 32;
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// 16-byte copy that writes zeros instead when index < 0 (the source address is then not touched), and
// nothing at all when `was_zero` is set as well: the destination still holds the zeros an earlier copy wrote.
__device__ __forceinline__ void cp_async_16_or_zero_once(uint32_t dst, const void* src, int index, uint32_t was_zero) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.lt.s32 p, %2, 0;\n\t"
        "setp.ne.and.b32 q, %3, 0, p;\n\t"
        "@!q cp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(dst),
        "l"(src), "r"(index), "r"(was_zero)
        : "memory");
}
// 16-byte copy that writes zeros instead when index < 0 (the source address is then not touched).
__device__ __forceinline__ void cp_async_16_or_zero(uint32_t dst, const void* src, int index) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.lt.s32 p, %2, 0;\n\t"
        "cp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(dst),
        "l"(src), "r"(index)
        : "memory");
}
// Arrival on `bar` that fires when all cp.async copies this thread has issued so far have landed
// (the barrier's expected count must include it).
__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024
// bytes apart (stride byte offset), leading byte offset unused by swizzled K-major layouts (set to 1),
// descriptor version 1, layout type 2 (SWIZZLE_128B). The start address sits in the low 14 bits in units
// of 16 bytes, so stepping 32 bytes along K adds 2 to the descriptor.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor, kind::f16: fp32 accumulate, fp16 A and B, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t umma_idesc(int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
        "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

struct SharedCtl {
    // a_full[t][s]: slot s has landed, for the issuer of tile t. One barrier per (issuer, slot) keeps a single
    // waiter per barrier: parity waits are only safe when the waiter has itself seen every earlier phase.
    unsigned long long a_full[MMA_WARPS][NSLOT_MAX];
    unsigned long long a_empty[NSLOT_MAX];   // the MMAs that read slot s have completed (commit of its issuer)
    unsigned long long i_full[NIDX_MAX];     // index block j has landed
    unsigned long long i_empty[NIDX_MAX];    // gather warp j % NSLOT has read index block j
    unsigned long long b_full[B_STAGES];
    unsigned long long b_empty[B_STAGES];    // every issuer has released the block (commit of its MMAs, or a plain arrival)
    unsigned long long acc_full[2];          // every issuer has committed its tile of the group (per accumulator set)
    unsigned long long acc_empty[2];         // the epilogue has read the set
    unsigned long long mma_drain;            // aborting CTA only: completes when the issuers' outstanding MMAs have finished
    uint32_t tmem_base;
    int abort_flag;
    int abort_where;   // code of the first wait that ran out (role and ring position), for the status block
    // per gather warp: the (stage << 2 | tile) codes of the current group's items in ring order, so that a warp
    // steps straight to the items it owns
    uint8_t stage_list[NSLOT_MAX][TILES * 32];
    uint8_t idx_list[TILES * 32];            // the same list for the index warp
    uint8_t issue[MMA_WARPS][KVOL_MAX + 1];  // per issuer: the current group's stages with work, as it meets them
    unsigned long long few_acc_empty[2];     // few-tiles path: the epilogue has read the accumulator
    unsigned long long tile_free[2];         // few-tiles path: every role is through with the tile's indices and its entry below
    int tile[2][4];                          // few-tiles path: frame (-1: none left), first row, the frame's rows, mask
    uint32_t scan_warp[32];                  // work split: per-warp totals of the block scan
    int range_lo, range_hi;                  // work split: this CTA's tiles
    uint32_t idx_uses[NIDX_MAX];             // bulk copies issued into index block j so far (for the abort path)
};

// Epilogue warps of the few-tiles path: with 64 channels a column block each for eight (warps 5-8 have nothing else to do there).
template <int COUT>
__host__ __device__ constexpr int few_epi_warps() { return COUT == 64 ? 2 * EPI_WARPS : EPI_WARPS; }
constexpr int STAGE_BYTES = 32 * 64;         // room of an epilogue warp of groups that are staged (store_tile_staged)
// Buffers of the two paths, which share their place.
template <int CIN, int COUT, bool STAGED>
__host__ __device__ constexpr int ring_bytes() {
    constexpr int groups = Ring<CIN>::NSLOT * A_BYTES + B_STAGES * COUT * ROW_BYTES + Ring<CIN>::NIDX * (64 / CIN) * TAP_WORDS * 4 +
                           (STAGED ? EPI_WARPS * STAGE_BYTES : 0);
    constexpr int few = FEW_SLOTS * (A_BYTES + COUT * ROW_BYTES) + 2 * FEW_IDX * TAP_WORDS * 4;
    return groups > few ? groups : few;
}
template <int CIN, int COUT, bool STAGED>
constexpr int umma_smem_bytes() { return 1024 /*alignment slack*/ + ring_bytes<CIN, COUT, STAGED>() + (int)sizeof(SharedCtl); }

// Offsets g*KG .. g*KG+KG-1 of a tile's 27-bit offset mask.
template <int KG>
__device__ __forceinline__ bool stage_active(uint32_t kmask, int g) {
    return ((kmask >> (g * KG)) & ((1u << KG) - 1u)) != 0u;
}

// One bit per stage (at bit position g * KG) that is set when the tile has a neighbour under any offset of the stage.
template <int KG>
__device__ __forceinline__ uint32_t stage_bits(uint32_t kmask) {
    if (KG == 1) return kmask;
    if (KG == 2) return (kmask | (kmask >> 1)) & 0x55555555u;
    uint32_t v = kmask | (kmask >> 1);
    v |= v >> 2;
    return v & 0x11111111u;
}

// Bit t set when row tile t has a neighbour under the offsets of stage g. The masks are only ever indexed
// with compile-time constants, so they stay in registers.
template <int KG>
__device__ __forceinline__ uint32_t active_tiles(const uint32_t (&m)[TILES], int g) {
    uint32_t bits = 0;
#pragma unroll
    for (int t = 0; t < TILES; ++t) bits |= (stage_active<KG>(m[t], g) ? 1u : 0u) << t;
    return bits;
}

// Advances to the next (stage g, tile t) item with work, in the order stage-major, tile-minor; `rem` holds
// the tiles of stage g not yet visited. Start with g = -1, rem = 0.
template <int KG>
__device__ __forceinline__ bool next_item(const uint32_t (&m)[TILES], int nstages, int& g, uint32_t& rem, int& t) {
    while (rem == 0u) {
        if (++g >= nstages) return false;
        rem = active_tiles<KG>(m, g);
    }
    t = __ffs((int)rem) - 1;
    rem &= rem - 1u;
    return true;
}

// Folded batch-norm scale and shift of the layer as launch parameters: the epilogue's multiply-adds then take them
// straight from the constant bank (its column loops are unrolled, so every index is a constant), where the
// earlier shared-memory copies cost two loads per channel pair and row on the pipe the gather copies keep busy.
struct EpiConst {
    float scale[64];
    float shift[64];
};

// Lane g holds `bits`, the tiles with work under stage g. Returns the number of (tile, stage) items of the stages
// before g and, in blocks_before, the number of those stages that have any work. Five warp votes: a vote answers
// in a few cycles, while a shuffle scan (five to ten shuffles, each a trip through the shared-memory pipe that the
// gather copies keep busy) cost every role some thousand cycles at each group boundary.
__device__ __forceinline__ int items_before_stage(uint32_t bits, int lane, int* blocks_before = nullptr) {
    const uint32_t lt = (1u << lane) - 1u;
    int items = 0;
#pragma unroll
    for (int t = 0; t < TILES; ++t) items += __popc(__ballot_sync(0xFFFFFFFFu, (bits >> t) & 1u) & lt);
    if (blocks_before) *blocks_before = __popc(__ballot_sync(0xFFFFFFFFu, bits != 0u) & lt);
    return items;
}

// Epilogue of channels FROM .. TO - 1 of a tile for one of four warps: lane = position `pos` of the map, output row `row`, accumulators
// at tensor-memory address taddr (zeros instead when !have). A lane stores its own row, 32 bytes to an instruction where the rows
// start at multiples of 32 bytes (wide): whole sectors. (16 bytes at a time an instruction touches half of 32 sectors. Through
// shared memory, so that a row leaves as one run, the warp's stores, reads and shuffles queue behind the gather warps' copies: a tile
// of 64 channels took a warp 5,900 cycles, which bound every layer of few items to a tile.)
template <int COUT, int FROM = 0, int TO = COUT>
__device__ __forceinline__ void store_tile(uint32_t taddr, bool have, const EpiConst& epi, int relu, int pos, int row, int n, int b,
                                           int max_voxels, __half* __restrict__ out, bool wide, __half* __restrict__ dense,
                                           const int4* __restrict__ out_coors, int D, int H, int W) {
    // Column blocks of CB channels keep the register footprint small (of 64 channels 32 at a time: these kernels spill).
    constexpr int CB = COUT == 32 ? 32 : 16;
    __half* to = out + ((size_t)b * max_voxels + row) * COUT;
#pragma unroll
    for (int cb = FROM; cb < TO; cb += CB) {
        float acc[CB];
        if (have) {
            if constexpr (CB == 32) {
                uint32_t r32[32];
                tmem_ld32(taddr + cb, r32);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[j] = __uint_as_float(r32[j]);
            } else {
                uint32_t r16[16];
                tmem_ld16(taddr + cb, r16);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[j] = __uint_as_float(r16[j]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < CB; ++j) acc[j] = 0.f;
        }
        uint32_t pk[CB / 2];
#pragma unroll
        for (int j = 0; j < CB / 2; ++j) {
            const int ch = cb + 2 * j;        // a constant after unrolling
            const __half2 h =
                __floats2half2_rn(fmaf(acc[2 * j], epi.scale[ch], epi.shift[ch]), fmaf(acc[2 * j + 1], epi.scale[ch + 1], epi.shift[ch + 1]));
            pk[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        if (relu) {
#pragma unroll
            for (int j = 0; j < CB / 2; ++j) {
                const __half2 h = __hmax2(*reinterpret_cast<const __half2*>(&pk[j]), __half2(__half(0.f), __half(0.f)));   // (a NaN becomes 0)
                pk[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
        if (pos < n) {
#pragma unroll
            for (int j = 0; j < CB / 2; j += 8) {
                if (wide) {
                    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(to + cb + 2 * j), "r"(pk[j]), "r"(pk[j + 1]),
                                 "r"(pk[j + 2]), "r"(pk[j + 3]), "r"(pk[j + 4]), "r"(pk[j + 5]), "r"(pk[j + 6]), "r"(pk[j + 7])
                                 : "memory");
                } else {
                    *reinterpret_cast<uint4*>(to + cb + 2 * j) = make_uint4(pk[j], pk[j + 1], pk[j + 2], pk[j + 3]);
                    *reinterpret_cast<uint4*>(to + cb + 2 * j + 8) = make_uint4(pk[j + 4], pk[j + 5], pk[j + 6], pk[j + 7]);
                }
            }
            if (dense) {
                // fused BEV scatter (sparse2Dense.cu:201-206): channel c*D + z, pixel (y, x)
                const int4 c4 = __ldg(&out_coors[(size_t)b * max_voxels + row]);
                const size_t plane = (size_t)D * H * W;
                __half* d = dense + ((size_t)b * COUT + cb) * plane + ((size_t)c4.y * H + c4.z) * W + c4.w;
#pragma unroll
                for (int j = 0; j < CB / 2; ++j, d += 2 * plane) {
                    const __half2 h = *reinterpret_cast<const __half2*>(&pk[j]);
                    d[0] = __low2half(h);
                    d[plane] = __high2half(h);
                }
            }
        }
    }
}

// The same through the warp's staging area (32 rows of 64 bytes), four lanes to a row, without the scatter: groups of 64 -> 64 channels
// with more than 18 offsets. Where a tile has twenty items the epilogue has time, and what counts is how often it looks into L1, whose
// tags the gather warps' copies keep busy: 64 lines of 128 bytes per 32 rows, where stores by row look 128 times. (In us, stores by row
// and through here: 27 offsets at 1/4 resolution, 16 x 120,000 points 326 and 322, 24 477 and 473, 32 639 and 631, 40 798 and 789, 64 x
// 20,000 432 and 428; 18 offsets, 20 x 120,000, 299 and 299; nine 191 and 203, six 154 and 173, three 125 and 150. The other layers have
// fewer items to a tile: 32 -> 64, 32 x 120,000, 396 and 445; 32 -> 32, 16 x 120,000, 379 and 380.)
constexpr int STAGED_KVOL = 18;
template <int COUT>
__device__ __forceinline__ void store_tile_staged(uint32_t taddr, bool have, const EpiConst& epi, int relu, uint8_t* stage, int lane,
                                                  int pos, int row, int n, int b, int max_voxels, __half* __restrict__ out) {
    constexpr int CB = 32, RB = CB * 2, CPR = RB / 16;   // channels and bytes of a row's column block, its 16-byte pieces
    static_assert(COUT % CB == 0, "whole column blocks");
    // pieces XOR-swizzled by row, so that neither the writes nor the reads below meet in a bank
    auto swizzled = [](int r, int piece) { return r * RB + ((piece ^ ((r >> 1) & 3)) << 4); };
#pragma unroll
    for (int cb = 0; cb < COUT; cb += CB) {
#pragma unroll
        for (int p0 = 0; p0 < CPR; p0 += 2) {            // sixteen columns
            uint32_t acc[16] = {};
            if (have) {
                tmem_ld16(taddr + cb + 8 * p0, acc);
                tmem_ld_wait();
            }
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                uint32_t pk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int a = 8 * p + 2 * j, ch = cb + 8 * p0 + a;   // constants after unrolling
                    __half2 h = __floats2half2_rn(fmaf(__uint_as_float(acc[a]), epi.scale[ch], epi.shift[ch]),
                                                  fmaf(__uint_as_float(acc[a + 1]), epi.scale[ch + 1], epi.shift[ch + 1]));
                    if (relu) h = __hmax2(h, __half2(__half(0.f), __half(0.f)));
                    pk[j] = *reinterpret_cast<const uint32_t*>(&h);
                }
                *reinterpret_cast<uint4*>(stage + swizzled(lane, p0 + p)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < CPR; ++i) {
            const int r = lane / CPR + i * (32 / CPR), p = lane % CPR;
            const uint4 v = *reinterpret_cast<const uint4*>(stage + swizzled(r, p));
            const int to = __shfl_sync(0xFFFFFFFFu, row, r);
            if (pos - lane + r < n) *reinterpret_cast<uint4*>(out + ((size_t)b * max_voxels + to) * COUT + cb + p * 8) = v;
        }
        __syncwarp();
    }
}

// ---- few tiles ----
// With few tiles per CTA the pipeline below is latency in good part: a group of one or two tiles uses a weight block once or
// twice, so that three of them in flight bound it (390 ns per item on a single 20,000-point frame), everything before
// the first gather (5.8 us: work split, masks, index copy) comes on top of every launch, and whole groups divide badly. This path
// takes one tile at a time, with eight slots in flight that hold a stage's rows and its weight block, and all of a tile's indices in one
// copy. What does not
// depend on the preceding kernel comes before the wait for that kernel: barriers, tensor memory, tile, indices and the
// first weight blocks. Tiles are handed out by a counter, one ahead of the tile in work (two index blocks, two accumulators: the
// next tile's gathers run while this one is stored): a CTA that starts late, because the preceding kernel still held its
// SM, leaves the further tiles to the others. A tile's offsets are added up in the same order as in the other path, so the results are
// the same bits.
template <int CIN, int COUT>
__device__ __forceinline__ uint32_t umma_few(SharedCtl* ctl, uint8_t* sA, int32_t* s_idx, bool wide, uint32_t tmem,
                                         bool leader, const __half* __restrict__ in, __half* __restrict__ out,
                                         const int32_t* __restrict__ nbr, const int32_t* __restrict__ order,
                                         const uint32_t* __restrict__ tile_mask, const int32_t* __restrict__ out_num,
                                         const uint8_t* __restrict__ wtiles, const EpiConst& epi, int relu, int batch,
                                         int max_voxels, int kvol, __half* __restrict__ dense,
                                         const int4* __restrict__ out_coors, int D, int H, int W, int* tile_counter, uint32_t first_mask,
                                         bool ahead, bool wait_first, int withhold_weights) {   // returns a gather warp's uses of its slot
    constexpr int KG = 64 / CIN, CPO = CIN / 8, B_BYTES = COUT * ROW_BYTES;
    constexpr uint32_t IDESC = umma_idesc(COUT);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles_per_frame = (max_voxels + TILE_M - 1) / TILE_M;
    volatile int* abort_flag = &ctl->abort_flag;
    uint8_t* sB = sA + FEW_SLOTS * A_BYTES;
    // barriers of the other path with the same arrival counts
    unsigned long long *full = ctl->a_full[0], *empty = ctl->a_empty, *tile_full = ctl->i_full, *tile_free = ctl->tile_free,
                       *acc_full = ctl->i_full + 2, *acc_empty = ctl->few_acc_empty;
    volatile int(*tile)[4] = ctl->tile;
    uint32_t items = 0;                        // items of the tiles so far
    uint32_t sums = 0;                         // tiles so far that had any: accumulator sets are used for those alone
    uint32_t uses = 0;                         // gather warps: times that the slot has been filled
    bool waited = wait_first;                  // the preceding kernel's writes may be read
    // Every role goes through the CTA's tiles in the same order; entry and index block `round & 1`. Waits for another role are
    // bounded, the one for the preceding kernel is not: a role is behind that one before it waits for what a role does behind it.
    if (few_slot(warp) >= 0) {
        // gather, as in the other path; slot s belongs to this warp
        const int s = few_slot(warp);
        const int c = lane & 7, jrow = (lane >> 3) * 8, koff = c / CPO;
        const uint32_t a_base = smem_u32(sA + s * A_BYTES) + jrow * ROW_BYTES;
        bool ok = true;
        for (uint32_t round = 0; ok; ++round) {
            const uint32_t r = round & 1u;
            ok = mbar_wait(smem_u32(tile_full + r), (round >> 1) & 1u, abort_flag, 1 | (int)(items << 4));
            if (!ok) break;
            const int b = tile[r][0], row0 = tile[r][1], n = tile[r][2];
            if (b < 0) break;
            const uint32_t stages = stage_bits<KG>((uint32_t)tile[r][3]);   // bit g * KG for stage g
            const __half* lane_base = in + (size_t)b * max_voxels * CIN + (c % CPO) * 8;
            const int rows_left = n - (row0 + jrow);
            // this warp's items: every FEW_SLOTS-th stage of the tile
            int e = (s + FEW_SLOTS - (int)(items % FEW_SLOTS)) % FEW_SLOTS;
            uint32_t left = stages;
            for (int i = 0; i < e; ++i) left &= left - 1u;
            for (; left; e += FEW_SLOTS) {
                const uint32_t q = items + (uint32_t)e;
                const int g = (__ffs((int)left) - 1) / KG;
#pragma unroll
                for (int i = 0; i < FEW_SLOTS; ++i) left &= left - 1u;
                const uint32_t idx_base = smem_u32(s_idx + r * (FEW_IDX * TAP_WORDS) + (g * KG + koff) * TAP_WORDS + jrow);
                const bool k_ok = g * KG + koff < kvol;
                const bool plain = g * KG + KG <= kvol && row0 + TILE_M <= n;   // uniform over the warp
                int vv[32];
#pragma unroll
                for (int w4 = 0; w4 < 8; ++w4) {
                    int4 v;
                    asm volatile("ld.shared.v4.s32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                 : "r"(idx_base + 128 * (w4 >> 1) + 16 * (w4 & 1)));
                    vv[4 * w4] = v.x, vv[4 * w4 + 1] = v.y, vv[4 * w4 + 2] = v.z, vv[4 * w4 + 3] = v.w;
                }
                ok = mbar_wait(smem_u32(empty + s), ((q / FEW_SLOTS) & 1u) ^ 1u, abort_flag, 2 | (int)(q << 4));
                if (!ok) break;
                if (lane == 0) {               // (this lane's arrival for the phase comes with its copies below)
                    mbar_expect_tx(smem_u32(full + s), B_BYTES);
                    if (!withhold_weights) {
                        bulk_load(smem_u32(sB + s * B_BYTES), wtiles + (size_t)g * B_BYTES, B_BYTES, smem_u32(full + s));
                        ++uses;
                    }
                }
                if (!waited) {
                    pdl_enter();
                    waited = true;
                }
                if (!plain) {
#pragma unroll
                    for (int p = 0; p < 32; ++p)
                        if (!(k_ok && 32 * (p >> 3) + (p & 7) < rows_left)) vv[p] = -1;
                }
#pragma unroll
                for (int p = 0; p < 32; ++p)
                    cp_async_16_or_zero(a_base + (32 * (p >> 3) + (p & 7)) * ROW_BYTES + ((c ^ (p & 7)) << 4),
                                        lane_base + (ptrdiff_t)vv[p] * CIN, vv[p]);
                cp_async_arrive_noinc(smem_u32(full + s));
            }
            items += (uint32_t)__popc(stages);
            mbar_arrive(smem_u32(tile_free + r));   // (behind the copies, which have consumed the indices)
            if (!waited) {                     // (no item in the first tile)
                pdl_enter();
                waited = true;
            }
        }
    } else if (warp < EPI_WARPS || (COUT == 64 && warp > EPI_WARPS && warp <= WEIGHT_WARP)) {
        // epilogue: a warp reads the tensor-memory lanes of its number modulo four
        const int quarter = warp & 3, part = warp < EPI_WARPS ? 0 : 1;
        for (uint32_t round = 0;; ++round) {
            const uint32_t r = round & 1u;
            bool ok = mbar_wait(smem_u32(tile_full + r), (round >> 1) & 1u, abort_flag, 3 | (int)(round << 4));
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            const int b = tile[r][0], row0 = tile[r][1], n = tile[r][2];
            const bool have = tile[r][3] != 0;
            if (b < 0) break;
            const int pos = row0 + quarter * 32 + lane;
            const int row = order && pos < n ? __ldg(order + (size_t)b * max_voxels + pos) : pos;
            mbar_arrive(smem_u32(tile_free + r));
            if (!waited) {                     // (out is another kernel's input until then)
                pdl_enter();
                waited = true;
            }
            const uint32_t set = sums & 1u;
            if (have) {
                ok = mbar_wait(smem_u32(acc_full + set), (sums >> 1) & 1u, abort_flag, 3 | (int)(round << 4));
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) break;
                tc_fence_after();
            }
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + set * COUT;
            if constexpr (COUT < 64) {
                store_tile<COUT>(taddr, have, epi, relu, pos, row, n, b, max_voxels, out, wide, dense, out_coors, D, H, W);
            } else {
                if (part == 0)
                    store_tile<COUT, 0, COUT / 2>(taddr, have, epi, relu, pos, row, n, b, max_voxels, out, wide, dense, out_coors, D, H, W);
                else
                    store_tile<COUT, COUT / 2, COUT>(taddr, have, epi, relu, pos, row, n, b, max_voxels, out, wide, dense, out_coors, D, H, W);
            }
            if (have) {
                tc_fence_before();
                mbar_arrive(smem_u32(acc_empty + set));
                ++sums;
            }
        }
    } else if (warp == EPI_WARPS) {
        // Issuer. One thread, so that nothing holds the lanes together, and one barrier per slot for both operands. (As a warp, with
        // a barrier for each, an item took some 500 cycles and the issuer was what bound the chain of a tile's items: front end of a
        // 20,000-point frame 250 us, then 240. Looking at the next item's barrier ahead of time gave nothing.) What an item takes is a
        // slot's round trip over the slots in flight: of 2,200 cycles with seven slots a gather warp's copies were 1,100, their landing
        // 950, the MMAs and their commit 430. Seven and eight slots: front end of 1 x 20,000 points 198.5 and 193.5 us, 1 x 120,000
        // 363.6 and 353 to 360; nine and ten where narrower layers leave room 194.5 and 361.
        if (leader) {
            if (!waited) {
                pdl_enter();
                waited = true;
            }
            bool ok = true;
            uint32_t s = 0, phase = 0;
            for (uint32_t round = 0; ok; ++round) {
                const uint32_t r = round & 1u;
                ok = mbar_wait<false, true>(smem_u32(tile_full + r), (round >> 1) & 1u, abort_flag, 4 | (int)(round << 4));
                if (!ok || tile[r][0] < 0) break;
                const int n_items = __popc(stage_bits<KG>((uint32_t)tile[r][3]));
                mbar_arrive(smem_u32(tile_free + r));
                if (!n_items) continue;
                const uint32_t set = sums & 1u, d_tmem = tmem + set * COUT;
                // the epilogue must have read this set's previous contents (two tiles back)
                ok = mbar_wait<false, true>(smem_u32(acc_empty + set), ((sums >> 1) & 1u) ^ 1u, abort_flag, 4 | (int)(round << 4));
#pragma unroll 2
                for (int e = 0; e < n_items; ++e) {
                    if (!ok) break;
                    ok = mbar_wait<false, true>(smem_u32(full + s), phase, abort_flag, 5 | (int)((items + e) << 4));
                    if (!ok) break;
                    fence_proxy_async();       // the gathered rows were written through the generic proxy
                    tc_fence_after();
                    const uint32_t at = s;
                    if (++s == FEW_SLOTS) s = 0, phase ^= 1u;
                    const uint64_t adesc = umma_desc(smem_u32(sA + at * A_BYTES));
                    const uint64_t bdesc = umma_desc(smem_u32(sB + at * B_BYTES));
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16(d_tmem, adesc + 2 * kk, bdesc + 2 * kk, IDESC, (e > 0 || kk > 0) ? 1u : 0u);
                    umma_commit(smem_u32(empty + at));
                }
                if (ok) umma_commit(smem_u32(acc_full + set));
                items += (uint32_t)n_items;
                ++sums;
            }
        }
        __syncwarp();
    } else if (warp == INDEX_WARP) {
        // the CTA's tiles and their indices. ahead: there are more tiles than CTAs, and the next one is taken while the last one is in
        // work.
        for (uint32_t round = 0;; ++round) {
            const uint32_t r = round & 1u;
            if (!waited && round >= 2u) {
                pdl_enter();
                waited = true;
            }
            // the first tile is that of the CTA's number, the others are handed out
            int t = blockIdx.x;
            if (round > 0 && ahead) {
                if (lane == 0) t = (int)gridDim.x + atomicAdd(tile_counter, 1);
                t = __shfl_sync(0xFFFFFFFFu, t, 0);
            }
            int frame = -1, first = 0, rows = 0;
            for (int f0 = 0; f0 < batch && frame < 0 && (round == 0 || ahead); f0 += 32) {
                int n = f0 + lane < batch ? load_late(out_num + f0 + lane) : 0;
                n = n > max_voxels ? max_voxels : (n < 0 ? 0 : n);
                const int tiles = (n + TILE_M - 1) / TILE_M;
                int incl = tiles;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (lane >= d) incl += v;
                }
                const uint32_t hit = __ballot_sync(0xFFFFFFFFu, t < incl);
                if (hit) {
                    const int src = __ffs((int)hit) - 1;
                    frame = f0 + src;
                    first = (t - __shfl_sync(0xFFFFFFFFu, incl - tiles, src)) * TILE_M;
                    rows = __shfl_sync(0xFFFFFFFFu, n, src);
                }
                t -= __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
            int mask = (int)first_mask;
            if (round > 0 || batch > 1) mask = (int)load_late(tile_mask + (size_t)(frame < 0 ? 0 : frame) * tiles_per_frame + first / TILE_M);
            if (frame < 0) mask = 0;
            bool ok = mbar_wait(smem_u32(tile_free + r), ((round >> 1) & 1u) ^ 1u, abort_flag, 7 | (int)(round << 4));
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok) break;
            if (lane == 0) {
                tile[r][0] = frame, tile[r][1] = first, tile[r][2] = rows, tile[r][3] = mask;
                ctl->idx_uses[r] = (round >> 1) + 1u;
                if (frame < 0) {
                    mbar_arrive(smem_u32(tile_full + r));
                } else {
                    mbar_arrive_expect_tx(smem_u32(tile_full + r), (uint32_t)(kvol * TAP_WORDS * 4));
                    bulk_load(smem_u32(s_idx + r * (FEW_IDX * TAP_WORDS)), nbr + nbr_index(kvol, max_voxels, frame, 0, first),
                              (uint32_t)(kvol * TAP_WORDS * 4), smem_u32(tile_full + r));
                }
            }
            if (frame < 0) break;
        }
    }
    if (!waited) pdl_enter();                  // every CTA waits: the next kernel counts on what came before this one
    return uses;
}

// STAGED: groups store their rows through shared memory. (A kernel of its own: with the choice made inside, 64 -> 64 groups are 8 % slower.)
template <int CIN, int COUT, bool STAGED>
__global__ void __launch_bounds__(Ring<CIN>::THREADS, 1)
conv_umma_kernel(const __half* __restrict__ in, __half* __restrict__ out, const int32_t* __restrict__ nbr,
                 const int32_t* __restrict__ order, const uint32_t* __restrict__ tile_mask, const int32_t* __restrict__ out_num,
                 const uint8_t* __restrict__ wtiles, const __grid_constant__ EpiConst epi, int relu, int batch,
                 int max_voxels, int kvol, __half* __restrict__ dense, const int4* __restrict__ out_coors, int D, int H,
                 int W, int32_t* status, int* tile_counter, int few_line, int maps_ready, int withhold_weights) {
    // Whatever does not depend on the preceding kernel comes before the wait for it. maps_ready: neighbour map, masks and
    // row counts are older than that kernel.
    if (!maps_ready) pdl_enter();
    // withhold_weights (tests of the time-out path only): the weight streamer stays silent, or the gather warps that ask for the
    // weights in the few-tiles path do, so the MMA issuers' bounded wait for the first weight block runs out and every CTA
    // with work leaves through the abort path.
    constexpr int KG = 64 / CIN;            // kernel offsets sharing one 128-byte A row
    constexpr int CPO = CIN / 8;            // 16-byte chunks per offset
    constexpr int B_BYTES = COUT * ROW_BYTES;
    constexpr int NSLOT = Ring<CIN>::NSLOT;
    constexpr int NIDX = Ring<CIN>::NIDX;
    constexpr int THREADS = Ring<CIN>::THREADS;
    constexpr int IDX_WORDS = KG * TAP_WORDS;  // one index block: KG offsets x 128 rows
    constexpr int IDX_BATCH = 16;           // items the index warp handles side by side (must stay below NIDX)
    constexpr int SET_COLS = TILES * COUT;  // accumulator columns of one set
    constexpr int TMEM_COLS = 2 * SET_COLS < 32 ? 32 : 2 * SET_COLS;
    constexpr uint32_t IDESC = umma_idesc(COUT);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;
    uint8_t* sB = sA + NSLOT * A_BYTES;
    int32_t* s_idx = reinterpret_cast<int32_t*>(sB + B_STAGES * B_BYTES);
    uint8_t* s_stage = reinterpret_cast<uint8_t*>(s_idx + NIDX * IDX_WORDS);   // (groups that are staged)
    SharedCtl* ctl = reinterpret_cast<SharedCtl*>(smem + ring_bytes<CIN, COUT, STAGED>());
    const bool wide = reinterpret_cast<uintptr_t>(out) % 32 == 0;   // (rows are 32, 64 or 128 bytes)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nstages = (kvol + KG - 1) / KG;
    const int tiles_per_frame = (max_voxels + TILE_M - 1) / TILE_M;
    // few-tiles path, a single frame: the mask of the CTA's first tile, requested before anything else
    uint32_t first_mask = 0;
    if (warp == INDEX_WARP && batch == 1 && (int)blockIdx.x < tiles_per_frame) first_mask = load_late(tile_mask + blockIdx.x);

    if (tid < THREADS / 2) {   // side by side: one thread would take half a microsecond for the hundred and more barriers
        if (tid < NSLOT) {
            for (int i = 0; i < MMA_WARPS; ++i)
                mbar_init(smem_u32(&ctl->a_full[i][tid]), 32);   // the lanes of the gather warp that owns the slot
            mbar_init(smem_u32(&ctl->a_empty[tid]), 1);
        }
        if (tid >= 32 && tid < 32 + NIDX) {
            const int j = tid - 32;
            ctl->idx_uses[j] = 0;
            mbar_init(smem_u32(&ctl->i_full[j]), 1);             // the lane of the index warp that issues the block's copy
            mbar_init(smem_u32(&ctl->i_empty[j]), 32);           // the lanes of the gather warp
        }
        if (tid >= 96 && tid < 96 + B_STAGES) {
            mbar_init(smem_u32(&ctl->b_full[tid - 96]), 1);
            mbar_init(smem_u32(&ctl->b_empty[tid - 96]), MMA_WARPS);
        }
        if (tid >= 128 && tid < 130) {
            mbar_init(smem_u32(&ctl->acc_full[tid - 128]), MMA_WARPS);          // every MMA issuer reports its tile
            mbar_init(smem_u32(&ctl->acc_empty[tid - 128]), EPI_WARPS * 32);    // every epilogue thread
            mbar_init(smem_u32(&ctl->tile_free[tid - 128]), (FEW_SLOTS + few_epi_warps<COUT>()) * 32 + 1);   // gather, epilogue, issuer
            mbar_init(smem_u32(&ctl->few_acc_empty[tid - 128]), few_epi_warps<COUT>() * 32);
        }
        if (tid == 160) {
            mbar_init(smem_u32(&ctl->mma_drain), MMA_WARPS);
            ctl->abort_flag = 0;
            ctl->abort_where = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    volatile int* abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();   // one lane per warp, the same one for the whole kernel

    uint32_t a_it = 0, b_it = 0, acc_it = 0;  // items, weight blocks and accumulator sets used so far; every role advances them identically
    uint32_t full_phase = 0;                  // MMA issuers: bit s = parity of the next phase of their a_full[t][s]
    uint32_t b_issued = 0;                    // weight streamer: blocks whose bulk copy has been started
    uint32_t few_uses = 0;                    // few-tiles path, gather warps (lane 0): weight blocks asked for
    uint32_t zero_rows = 0;                   // gather warps: bit p = this lane's chunk of row p of its slot holds zeros

    // Balanced split: the occupied 128-row tiles of all frames, laid end to end, are cut into gridDim.x
    // contiguous ranges of equal work (row counts and tile masks are read from the device, so no host round
    // trip); a CTA walks its range in groups of up to TILES tiles of one frame. The work of a tile is the number
    // of its (tile, stage) items plus a constant for its epilogue: rows numbered in spatial order make
    // neighbouring tiles alike, so dense and sparse regions would otherwise load the CTAs unevenly.
    // Every CTA computes the same cut points from the same masks: thread t sums the weights of its slice of the
    // tile sequence, a block scan turns the sums into running totals, and the threads whose slice holds cut
    // point blockIdx.x or blockIdx.x + 1 walk the slice to the tile where the running total passes the target.
    auto frame_rows = [&](int f) {
        const int v = load_late(out_num + f);
        return v > max_voxels ? max_voxels : (v < 0 ? 0 : v);
    };
    // Tiles before every frame, in shared memory that nothing uses yet. (Row counts and masks are read side by side: one
    // after the other they were most of the 15 to 19 us that a launch over 32 frames cost beside its work.) With few frames
    // every thread adds and walks by itself: those launches are all latency, and the hand-over takes half a microsecond. (Front end,
    // frames of 20,000 points, by itself and handed over: 2 frames 340 and 347 us, 6 592 and 595, 8 711 and 711, 9 779 and 778, 12 963
    // and 958, 32 2230 and 2191.)
    int* first_tile = reinterpret_cast<int*>(sA);             // [batch]
    static_assert(kMaxBatch * 4 <= NSLOT * A_BYTES, "a word per frame");
    constexpr int FEW_FRAMES = 8;
    int total_tiles = 0;
    if (batch <= FEW_FRAMES) {
        for (int f = 0; f < batch; ++f) total_tiles += (frame_rows(f) + TILE_M - 1) / TILE_M;
    } else {
        for (int f = tid; f < batch; f += THREADS) first_tile[f] = (frame_rows(f) + TILE_M - 1) / TILE_M;
        __syncthreads();
        if (warp == 0) {
            int before = 0;
            for (int f0 = 0; f0 < batch; f0 += 32) {
                const int v = f0 + lane < batch ? first_tile[f0 + lane] : 0;
                int incl = v;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (lane >= d) incl += u;
                }
                if (f0 + lane < batch) first_tile[f0 + lane] = before + incl - v;
                before += __shfl_sync(0xFFFFFFFFu, incl, 31);
            }
            if (lane == 0) ctl->range_hi = before;
        }
        __syncthreads();
        total_tiles = ctl->range_hi;
    }
    // A layer with the BEV scatter takes the few-tiles path whatever its size. The scatter's stores, two bytes to a channel and row, are
    // most of what it does, and a group's four tiles leave together, which the other roles wait for. (In us, groups and here, with up
    // to 181 tiles per SM: 64 -> 64 of three offsets, 96 x 120,000 points, 535 and 390, of 27 1614 and 1029; 32 -> 32 of 27 756 and 560;
    // 16 -> 16 of three 340 and 306, of 27 2835 and 852; 16 -> 32 of 27 414 and 351; at 14 to 18 tiles per SM 80 and 64, 245 and 154, 105
    // and 84, 48 and 41, 76 and 66, 117 and 86.)
    const bool few = dense != nullptr || total_tiles <= few_line * (int)gridDim.x;
    if (few) {
        static_assert(FEW_IDX % KG == 0 && FEW_IDX >= KVOL_MAX, "whole stages of indices");
        int32_t* few_idx = reinterpret_cast<int32_t*>(sA + FEW_SLOTS * (A_BYTES + B_BYTES));
        few_uses = umma_few<CIN, COUT>(ctl, sA, few_idx, wide, tmem, leader, in, out, nbr, order, tile_mask, out_num, wtiles, epi,
                                       relu, batch, max_voxels, kvol, dense, out_coors, D, H, W, tile_counter,
                                       first_mask, total_tiles > (int)gridDim.x, !maps_ready, withhold_weights);
    }
    if (!few) {
        if (tid == 0) ctl->range_lo = 0, ctl->range_hi = total_tiles;   // (the next barrier comes before anyone's cut point)
        const int per = (total_tiles + THREADS - 1) / THREADS;
        const int first = tid * per, last = first + per < total_tiles ? first + per : total_tiles;
        // a tile costs its items plus its share of the group hand-over and of the epilogue, about eight items' worth
        // (fitted to the CTA lifetimes of 1/4-resolution launches)
        auto tile_weight = [&](uint32_t mask) { return (uint32_t)(__popc(stage_bits<KG>(mask)) + 8); };
        // Pass 0: the weight of this thread's slice, and the weights before it. Passes 1 and 2: cut points c and c + 1, each the
        // first tile whose running total (inclusive) exceeds grand * c / gridDim.x; a thread whose slice holds one walks the
        // slice again. (One copy of the walk: a kernel's first launch in a while fetches its code from L2, and two
        // copies cost a single frame 1 %.)
        uint32_t mine = 0, excl = 0, grand = 0;
#pragma unroll 1
        for (int pass = 0; pass < 3; ++pass) {
            uint32_t run = excl, target = ~0u;
            if (pass > 0) {
                const unsigned long long c = blockIdx.x + pass - 1;
                if (c == 0 || c >= gridDim.x) continue;   // 0 and total_tiles are preset
                target = (uint32_t)((unsigned long long)grand * c / gridDim.x);
                if (mine == 0 || target < excl || target >= excl + mine) continue;
            }
            int cut = last;
            if (batch <= FEW_FRAMES) {
                int f = 0, start = 0, tiles = (frame_rows(0) + TILE_M - 1) / TILE_M;
                for (int i = first; i < last; ++i) {
                    while (i >= start + tiles) {
                        start += tiles;
                        tiles = (frame_rows(++f) + TILE_M - 1) / TILE_M;
                    }
                    run += tile_weight(__ldg(tile_mask + (size_t)f * tiles_per_frame + (i - start)));
                    if (run > target) {
                        cut = i;
                        break;
                    }
                }
            } else if (first < last) {
                int f = 0;                                    // frame of the slice's first tile: the last that starts at or before it
                for (int n = batch; n > 1;) {
                    const int half = n / 2;
                    if (first_tile[f + half] <= first) f += half;
                    n -= half;
                }
                for (int i0 = first; i0 < last && cut == last; i0 += 4) {   // the masks of four tiles requested together
                    uint32_t w[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        while (i0 + u < last && f + 1 < batch && first_tile[f + 1] <= i0 + u) ++f;
                        w[u] = i0 + u < last ? tile_weight(__ldg(tile_mask + (size_t)f * tiles_per_frame + (i0 + u - first_tile[f]))) : 0u;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        run += w[u];
                        if (run > target && cut == last) cut = i0 + u;
                    }
                }
            }
            if (pass > 0) {
                if (pass == 1) ctl->range_lo = cut;
                else ctl->range_hi = cut;
                continue;
            }
            mine = run;
            uint32_t incl = mine;   // inclusive block scan of `mine`
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= d) incl += v;
            }
            if (lane == 31) ctl->scan_warp[warp] = incl;
            __syncthreads();
            uint32_t before = 0;
            for (int w = 0; w < THREADS / 32; ++w) {
                const uint32_t v = ctl->scan_warp[w];
                if (w < warp) before += v;
                grand += v;
            }
            excl = before + incl - mine;   // weight of all tiles before this thread's slice
        }
    }
    __syncthreads();
    const int range_lo = ctl->range_lo, range_hi = ctl->range_hi;
    // The walk is one group ahead of the work: the masks of the next group are requested when the current group
    // starts, so that no role sits in the latency of those reads at a group boundary (every role of the CTA would
    // stall there at about the same time and drain the pipeline).
    int c_b = 0, c_first = 0;                   // cursor: frame and the global index of its first tile
    int c_n = batch > 0 ? frame_rows(0) : 0;
    int c_tiles = (c_n + TILE_M - 1) / TILE_M;
    int c_cur = range_lo;
    int nx_b = 0, nx_n = 0, nx_tile0 = 0, nx_cnt = 0;   // the next group
    uint32_t nx_m[TILES] = {0u, 0u, 0u, 0u};
    auto fetch_next = [&]() {
        nx_cnt = 0;
        if (c_cur >= range_hi) return;
        while (c_cur >= c_first + c_tiles) {
            c_first += c_tiles;
            ++c_b;
            c_n = frame_rows(c_b);
            c_tiles = (c_n + TILE_M - 1) / TILE_M;
        }
        nx_b = c_b;
        nx_n = c_n;
        nx_tile0 = c_cur - c_first;
        int cnt = range_hi - c_cur;
        cnt = cnt > TILES ? TILES : cnt;
        cnt = cnt > c_tiles - nx_tile0 ? c_tiles - nx_tile0 : cnt;
        nx_cnt = cnt;
        c_cur += cnt;
#pragma unroll
        for (int t = 0; t < TILES; ++t)
            nx_m[t] = t < cnt ? __ldg(tile_mask + (size_t)nx_b * tiles_per_frame + nx_tile0 + t) : 0u;
    };
    if (!few) fetch_next();
    // Rows are read and written by the gather and epilogue warps alone: indices and weights are older than the preceding kernel and
    // start right away. (Front end with every warp behind the wait: 2 x 20,000 points 339.8 us, now 331.6; 5 x 77,000 730 and 724.)
    // Their warps wait for that kernel once their rings are full, and the issuers before the first rows: a bounded wait for rows
    // that are gathered behind the other one would count the rest of that kernel, however long it runs. (Issuers that wait before
    // anything else: 8 x 20,000 points 672.9 us instead of 670.0.)
    bool early = maps_ready && !few;          // not behind the wait for the preceding kernel yet
    if (early && (warp < EPI_WARPS || warp >= FIRST_GATHER_WARP)) {
        pdl_enter();
        early = false;
    }

    while (nx_cnt > 0) {
        const int b = nx_b, n = nx_n, tile0 = nx_tile0, cnt = nx_cnt;
        const int row0 = tile0 * TILE_M;
        uint32_t m[TILES];
        uint32_t any = 0;
#pragma unroll
        for (int t = 0; t < TILES; ++t) {
            m[t] = nx_m[t];
            any |= m[t];
        }
        fetch_next();   // reads issued now, used at the top of the next iteration
        if (*abort_flag) break;
        // items and weight blocks this group consumes
        const uint32_t sb0 = stage_bits<KG>(m[0]), sb1 = stage_bits<KG>(m[1]), sb2 = stage_bits<KG>(m[2]),
                       sb3 = stage_bits<KG>(m[3]);
        const int n_a = __popc(sb0) + __popc(sb1) + __popc(sb2) + __popc(sb3);
        const int n_b = __popc(sb0 | sb1 | sb2 | sb3);
        const uint32_t set = acc_it & 1u;           // accumulator set of this group (groups without work use none)
        const uint32_t set_phase = (acc_it >> 1) & 1u;

        if (warp >= FIRST_GATHER_WARP) {
            // ---------------- gather producers ----------------
            // Gather warp s fills slot s with every NSLOT-th item and issues all of its copies: while one warp
            // sits in the latency of its barrier hand-offs the others keep the copy pipe busy.
            // Lane = (row group j, 16-byte chunk c): the eight lanes j*8..j*8+7 copy, in step p, chunk c of row
            // 32 (p / 8) + 8 j + p % 8 of the item to chunk c ^ (row & 7) of the slot's row (128-byte swizzle).
            // With the rows of a group in runs of eight, the four groups' 16-byte index reads of one instruction
            // lie 32 bytes apart (different banks: one pass), where runs of 32 rows put them 128 bytes apart
            // (the same banks: four passes).
            const int s = warp - FIRST_GATHER_WARP;
            const int c = lane & 7;                // 16-byte chunk of the 128-byte row
            const int jrow = (lane >> 3) * 8;      // first row of this lane group's first run of eight
            const int koff = c / CPO;              // offset of the stage's group this chunk belongs to
            const int csub = (c % CPO) * 8;        // first channel of the chunk
            const __half* in_b = in + (size_t)b * max_voxels * CIN;
            // list of this group's items: lane g holds stage g's tiles, a warp scan places them
            uint8_t* list = ctl->stage_list[s];
            {
                const uint32_t bits = lane < nstages ? active_tiles<KG>(m, lane) : 0u;
                int at = items_before_stage(bits, lane);
#pragma unroll
                for (int tt = 0; tt < TILES; ++tt)
                    if ((bits >> tt) & 1u) list[at++] = (uint8_t)((lane << 2) | tt);
                __syncwarp();
            }
            const int first = (s + NSLOT - (int)(a_it % NSLOT)) % NSLOT;
            const uint32_t idx_lane = smem_u32(&s_idx[koff * TAP_WORDS + jrow]);
            const uint32_t a_base = smem_u32(sA + s * A_BYTES) + jrow * ROW_BYTES;
            for (int e = first; e < n_a; e += NSLOT) {
                const uint32_t q = a_it + (uint32_t)e;
                const uint32_t use = (q / NSLOT) & 1u;   // parity of this use of the slot
                const uint32_t ji = q % NIDX;            // index block of the item
                const uint32_t iuse = (q / NIDX) & 1u;
                const uint32_t idx_base = idx_lane + ji * (IDX_WORDS * 4);
                const int code = list[e];
                const int g = code >> 2, t = code & 3;
                // row indices of this item, fetched ahead of time by the index warp
                if (!mbar_wait(smem_u32(&ctl->i_full[ji]), iuse, abort_flag, 1 | (int)(q << 4))) break;

                // all 32 indices first (the copies below are compiler barriers, a load could not move above them)
                int vv[32];
#pragma unroll
                for (int w4 = 0; w4 < 8; ++w4) {
                    int4 v;
                    asm volatile("ld.shared.v4.s32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                 : "r"(idx_base + 128 * (w4 >> 1) + 16 * (w4 & 1)));   // rows 32 (w4 / 2) + 8 j + 4 (w4 % 2) ..
                    vv[4 * w4] = v.x, vv[4 * w4 + 1] = v.y, vv[4 * w4 + 2] = v.z, vv[4 * w4 + 3] = v.w;
                }
                if (!mbar_wait(smem_u32(&ctl->a_empty[s]), use ^ 1u, abort_flag, 2 | (int)(q << 4))) break;
                const bool k_ok = g * KG + koff < kvol;
                const int rows_left = n - (row0 + t * TILE_M + jrow);   // step p's row lies inside the frame when 32 (p / 8) + p % 8 < rows_left
                // Every instruction of this loop is on the critical path of the item, so the common case - all
                // offsets of the stage exist and the whole tile lies inside the frame - takes three instructions
                // per row: a predicate from the sign of the index, the address, and a copy that writes zeros when
                // the predicate says the neighbour is missing.
                const bool plain = g * KG + KG <= kvol && row0 + (t + 1) * TILE_M <= n;   // uniform over the warp
                const __half* lane_base = in_b + csub;
                if (plain) {
                    // Of the rows of 64 -> 64 items at 1/4 resolution 18 % are missing neighbours, of others more, and many are
                    // missing in two consecutive uses of the slot: their zeros are still there, so the copy is left out (the
                    // shared-memory write of a zero row costs the same as that of a real one).
                    uint32_t zero_now = 0;
#pragma unroll
                    for (int p = 0; p < 32; ++p) {
                        cp_async_16_or_zero_once(a_base + (32 * (p >> 3) + (p & 7)) * ROW_BYTES + ((c ^ (p & 7)) << 4),
                                                 lane_base + (ptrdiff_t)vv[p] * CIN, vv[p], zero_rows & (1u << p));
                        zero_now |= ((uint32_t)vv[p] >> 31) << p;
                    }
                    zero_rows = zero_now;
                } else {
                    zero_rows = 0;   // (the general path writes every row)
#pragma unroll
                    for (int p = 0; p < 32; ++p) {
                        const int id = (k_ok && 32 * (p >> 3) + (p & 7) < rows_left) ? vv[p] : -1;
                        const __half* src = in_b + (size_t)(id < 0 ? 0 : id) * CIN + csub;
                        cp_async_16(a_base + (32 * (p >> 3) + (p & 7)) * ROW_BYTES + ((c ^ (p & 7)) << 4), src,
                                    id < 0 ? 0u : 16u);
                    }
                }
                // The index block may be refilled now: every index has been consumed by a copy above (the arrival
                // sits behind the copies so that it depends on the registers the index loads wrote; released
                // earlier, right after the loads were issued, the last of them were seen to return the next
                // item's indices). The ring is three slot cycles deep, so nothing waits for this.
                mbar_arrive(smem_u32(&ctl->i_empty[ji]));
                // publishes the slot, when the copies land, to the issuer that owns row tile t
                cp_async_arrive_noinc(smem_u32(&ctl->a_full[t][s]));
            }
        } else if (warp < EPI_WARPS) {
            // ---------------- epilogue ----------------
            // output rows of this thread's positions (the map may hold the rows in another order), requested before the wait
            int out_row[TILES];
#pragma unroll
            for (int t = 0; t < TILES; ++t) {
                const int pos = row0 + t * TILE_M + tid;
                out_row[t] = order && t < cnt && pos < n ? __ldg(order + (size_t)b * max_voxels + pos) : pos;
            }
            bool got = true;
            if (any) {
                got = mbar_wait<true>(smem_u32(&ctl->acc_full[set]), set_phase, abort_flag, 3 | (int)(acc_it << 4));
                got = __all_sync(0xFFFFFFFFu, got);
                if (got) tc_fence_after();
            }
#pragma unroll 1
            for (int t2 = 0; t2 < cnt; ++t2) {
                const int pos = row0 + t2 * TILE_M + tid;
                const int row = t2 == 0 ? out_row[0] : (t2 == 1 ? out_row[1] : (t2 == 2 ? out_row[2] : out_row[3]));
                const uint32_t m_t2 = t2 == 0 ? m[0] : (t2 == 1 ? m[1] : (t2 == 2 ? m[2] : m[3]));
                if (!got) continue;
                const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + set * SET_COLS + t2 * COUT;
                if constexpr (STAGED)
                    store_tile_staged<COUT>(taddr, any && m_t2, epi, relu, s_stage + warp * STAGE_BYTES, lane, pos, row, n, b, max_voxels, out);
                else
                    store_tile<COUT>(taddr, any && m_t2, epi, relu, pos, row, n, b, max_voxels, out, wide, nullptr, nullptr, 0, 0, 0);
            }
            if (any && got) {
                tc_fence_before();
                mbar_arrive(smem_u32(&ctl->acc_empty[set]));   // the set may be overwritten
            }
        } else if (warp < WEIGHT_WARP) {
            // ---------------- MMA issuers ----------------
            // Issuer t owns tile t: its accumulator, the items (t, g) and their slots. All four wait for every
            // weight block and release it, also one with nothing to do for the stage: each of its waits and
            // arrivals must count for this use of the weight slot, not for an earlier one (a slot refilled while
            // an issuer has not yet tested its previous use would leave that issuer waiting on the wrong phase).
            // The schedule of the group is worked out once, lane g for stage g (which weight slot and phase, whether tile t takes
            // part, which A slot its item sits in). With 64 input channels it is left in shared memory for one elected thread, which
            // goes through it alone; with fewer the warp goes through it together and hands it round with shuffles, and the elected
            // lane issues (always the same one: commits count the instructions of their own thread). Calls, warp and thread, in us:
            // 64 -> 64 32 x 120,000 points 1008 and 989, 32 x 20,000 378 and 369; 16 -> 32 1262 and 1295, 417 and 425; 32 -> 64
            // 1327 and 1347, 411 and 417. Looking at the next stage's barriers ahead of time is slower for either.
            if (any) {
                const int t = warp - EPI_WARPS;
                const uint32_t bits = lane < nstages ? active_tiles<KG>(m, lane) : 0u;
                int blocks_before = 0;
                const int items_before = items_before_stage(bits, lane, &blocks_before);
                const uint32_t pos = a_it + (uint32_t)items_before + (uint32_t)__popc(bits & ((1u << t) - 1u));
                const uint32_t my_b = b_it + (uint32_t)blocks_before;
                const uint32_t info = ((bits >> t) & 1u) | ((my_b % B_STAGES) << 1) | (((my_b / B_STAGES) & 1u) << 3) | ((pos % NSLOT) << 4);
                const uint32_t d_tmem = tmem + set * SET_COLS + t * COUT;
                bool started = false;
                auto weights_landed = [&](uint32_t inf, int j) {
                    return mbar_wait<false, true>(smem_u32(&ctl->b_full[(inf >> 1) & 3u]), (inf >> 3) & 1u, abort_flag,
                                                  5 | (int)((b_it + j) << 4));
                };
                auto rows_landed = [&](uint32_t inf, int j) {   // the issuer's next use of the slot is the next phase
                    const uint32_t sa = (inf >> 4) & 15u, phase = (full_phase >> sa) & 1u;
                    full_phase ^= 1u << sa;
                    return mbar_wait<false, true>(smem_u32(&ctl->a_full[t][sa]), phase, abort_flag, 6 | (int)((b_it + j) << 4));
                };
                auto issue = [&](uint32_t inf) {
                    const uint32_t sb = (inf >> 1) & 3u, sa = (inf >> 4) & 15u;
                    fence_proxy_async();       // the gathered rows were written through the generic proxy
                    tc_fence_after();
                    const uint64_t adesc = umma_desc(smem_u32(sA + sa * A_BYTES));
                    const uint64_t bdesc = umma_desc(smem_u32(sB + sb * B_BYTES));
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16(d_tmem, adesc + 2 * kk, bdesc + 2 * kk, IDESC, (started || kk > 0) ? 1u : 0u);
                    umma_commit(smem_u32(&ctl->a_empty[sa]));   // frees the A slot once these MMAs have read it
                    umma_commit(smem_u32(&ctl->b_empty[sb]));   // and this issuer's hold on the weight block
                };
                auto pass = [&](uint32_t inf) { mbar_arrive(smem_u32(&ctl->b_empty[(inf >> 1) & 3u])); };   // nothing to read from this block
                // the epilogue must have read this set's previous contents (two groups back)
                auto set_free = [&]() {
                    return mbar_wait<false, true>(smem_u32(&ctl->acc_empty[set]), set_phase ^ 1u, abort_flag, 4 | (int)(acc_it << 4));
                };
                auto report = [&]() {
                    if (started) umma_commit(smem_u32(&ctl->acc_full[set]));
                    else mbar_arrive(smem_u32(&ctl->acc_full[set]));
                };
                if constexpr (CIN == 64) {
                    if (bits) ctl->issue[t][blocks_before] = (uint8_t)info;
                    __syncwarp();
                    if (leader) {
                        bool ok = set_free();
                        if (early) {
                            pdl_enter();
                            early = false;
                        }
                        tc_fence_after();
#pragma unroll 2
                        for (int j = 0; j < n_b; ++j) {
                            if (!ok) break;
                            const uint32_t inf = ctl->issue[t][j];
                            ok = weights_landed(inf, j);
                            if (!ok) break;
                            if (inf & 1u) {
                                ok = rows_landed(inf, j);
                                if (!ok) break;
                                issue(inf);
                                started = true;
                            } else {
                                pass(inf);
                            }
                        }
                        if (ok) report();
                    }
                } else {
                    bool ok = __all_sync(0xFFFFFFFFu, set_free());
                    if (early) {
                        pdl_enter();
                        early = false;
                    }
                    tc_fence_after();
                    uint32_t left = __ballot_sync(0xFFFFFFFFu, bits != 0u);
                    for (int j = 0; left && ok; ++j, left &= left - 1u) {
                        const uint32_t inf = __shfl_sync(0xFFFFFFFFu, info, __ffs((int)left) - 1);
                        ok = weights_landed(inf, j);
                        if (inf & 1u) ok = ok && rows_landed(inf, j);
                        ok = __all_sync(0xFFFFFFFFu, ok);
                        if (!ok) break;
                        if (inf & 1u) {
                            if (leader) issue(inf);
                            started = true;
                        } else if (leader) {
                            pass(inf);
                        }
                    }
                    if (ok && leader) report();
                }
            }
            __syncwarp();
        } else if (warp == INDEX_WARP) {
            // ---------------- neighbour-index loader ----------------
            // Copies, for every item in consumption order, the KG x 128 neighbour indices into the next block of
            // the index ring, two to three slot cycles ahead of the gather warp that will use them. The map is
            // tile-major and spaces a tile's offsets like the index block does, so an item is one bulk copy that
            // reports to the block's barrier by byte count; the lanes of the warp work on IDX_BATCH consecutive
            // items at once (one dependent chain of wait, expect and copy per lane instead of one per item). The
            // gather warps ignore the indices of rows past the frame's row count (stale) and of offsets past kvol
            // (not loaded).
            {
                uint8_t* list = ctl->idx_list;
                {
                    const uint32_t bits = lane < nstages ? active_tiles<KG>(m, lane) : 0u;
                    int at = items_before_stage(bits, lane);
#pragma unroll
                    for (int tt = 0; tt < TILES; ++tt)
                        if ((bits >> tt) & 1u) list[at++] = (uint8_t)((lane << 2) | tt);
                    __syncwarp();
                }
                // The lanes step through the batches together: an item's wait tests the parity of the previous use
                // of its block, which is only meaningful once the lane that handled that use (a lane of an earlier
                // batch) has passed its own wait. A lane running batches ahead of the others would break that.
                bool live = true;
                for (int base = 0; base < n_a; base += IDX_BATCH) {
                    const int e = base + lane;
                    if (live && lane < IDX_BATCH && e < n_a) {
                        const uint32_t q = a_it + (uint32_t)e;
                        const uint32_t j = q % NIDX;
                        const int code = list[e];
                        const int g = code >> 2, t = code & 3;
                        if (early && q >= (uint32_t)NIDX) {
                            pdl_enter();
                            early = false;
                        }
                        live = mbar_wait(smem_u32(&ctl->i_empty[j]), ((q / NIDX) & 1u) ^ 1u, abort_flag, 7 | (int)(q << 4));
                        if (live) {
                            // the map is tile-major with the block's own spacing between offsets: the stage's
                            // offsets of this tile are one contiguous run
                            int nk = kvol - g * KG;
                            nk = nk > KG ? KG : nk;
                            const uint32_t bar = smem_u32(&ctl->i_full[j]);
                            ctl->idx_uses[j] = q / NIDX + 1u;
                            mbar_arrive_expect_tx(bar, (uint32_t)(nk * TAP_WORDS * 4));
                            bulk_load(smem_u32(&s_idx[j * IDX_WORDS]),
                                      nbr + nbr_index(kvol, max_voxels, b, g * KG, row0 + t * TILE_M),
                                      (uint32_t)(nk * TAP_WORDS * 4), bar);
                        }
                    }
                    live = __all_sync(0xFFFFFFFFu, live);   // also the batch boundary: no lane starts the next batch early
                    if (!live) break;
                }
            }
        } else {
            // ---------------- weight streamer ----------------
            if (lane == 0 && !withhold_weights) {
                uint32_t my_b = b_it;
                for (int g = 0; g < nstages; ++g) {
                    if (!active_tiles<KG>(m, g)) continue;
                    const uint32_t sb = my_b % B_STAGES;
                    if (early && my_b >= B_STAGES) {
                        pdl_enter();
                        early = false;
                    }
                    if (!mbar_wait(smem_u32(&ctl->b_empty[sb]), ((my_b / B_STAGES) & 1u) ^ 1u, abort_flag,
                                   8 | (int)(my_b << 4)))
                        break;
                    const uint32_t bar = smem_u32(&ctl->b_full[sb]);
                    mbar_arrive_expect_tx(bar, B_BYTES);
                    bulk_load(smem_u32(sB + sb * B_BYTES), wtiles + (size_t)g * B_BYTES, B_BYTES, bar);
                    ++my_b;
                    b_issued = my_b;
                }
            }
            __syncwarp();
        }
        a_it += n_a;
        b_it += n_b;
        if (any) ++acc_it;
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        // An aborting CTA must not return while its own copies are still writing shared memory or its MMAs tensor
        // memory: the gather and index warps wait for their cp.async copies, the issuers commit to a barrier that
        // warp 4 waits on (bounded) before it frees the tensor memory, the weight streamer waits (bounded) for
        // its last bulk copies.
        if (warp >= FIRST_GATHER_WARP || warp == INDEX_WARP) asm volatile("cp.async.wait_all;" ::: "memory");
        if (warp >= EPI_WARPS && warp < WEIGHT_WARP && leader) umma_commit(smem_u32(&ctl->mma_drain));
        if (warp == INDEX_WARP) {
            for (int j = lane; j < NIDX; j += 32) {
                const uint32_t uses = ctl->idx_uses[j];
                if (!uses) continue;
                const uint32_t bar = smem_u32(&ctl->i_full[j]);
                const long long t0 = clock64();
                while (!mbar_try_wait(bar, (uses - 1u) & 1u) && clock64() - t0 < WAIT_LIMIT_CYCLES) {}
            }
        }
        auto settle = [&](const unsigned long long* bar, uint32_t parity) {
            const long long t0 = clock64();
            while (!mbar_try_wait(smem_u32(bar), parity) && clock64() - t0 < WAIT_LIMIT_CYCLES) {}
        };
        if (warp == WEIGHT_WARP && lane == 0)
            for (uint32_t j = b_issued > B_STAGES ? b_issued - B_STAGES : 0u; j < b_issued; ++j)
                settle(&ctl->b_full[j % B_STAGES], (j / B_STAGES) & 1u);
        if (few_uses) settle(&ctl->a_full[0][few_slot(warp)], (few_uses - 1u) & 1u);
    }
    __syncthreads();
    if (tid == 0 && *abort_flag) {
        atomicOr(status, SESSD_STATUS_TIMEOUT);
        atomicCAS(status + 1, 0, ctl->abort_where);   // first report wins: which wait, at which ring position
    }
    if (warp == EPI_WARPS) {
        if (*abort_flag && lane == 0) {
            // the tensor memory is given back only when no MMA of this CTA can still write to it
            const long long t0 = clock64();
            while (!mbar_try_wait(smem_u32(&ctl->mma_drain), 0u) && clock64() - t0 < WAIT_LIMIT_CYCLES) {}
        }
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

template <int CIN, int COUT, bool STAGED = false>
int launch_one(const ConvLaunch& c, cudaStream_t stream) {
    static const std::string name = "conv_umma<f16," + std::to_string(CIN) + "," + std::to_string(COUT) + ">";
    const int smem = umma_smem_bytes<CIN, COUT, STAGED>();
    static_assert(umma_smem_bytes<CIN, COUT, STAGED>() <= 227 * 1024, "ring does not fit the shared memory of one SM");
    // the attribute belongs to the device's context: set it once per device (repeating it is harmless, so a
    // race between two host threads only costs a second call)
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    SESSD_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        SESSD_CUDA(cudaFuncSetAttribute(conv_umma_kernel<CIN, COUT, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured.fetch_or(bit, std::memory_order_release);
    }
    if (!c.scale_host || !c.shift_host) return SESSD_ERR_PARAM;
    EpiConst epi;
    memcpy(epi.scale, c.scale_host, sizeof epi.scale);
    memcpy(epi.shift, c.shift_host, sizeof epi.shift);
    SESSD_LAUNCH_NAMED(name.c_str(), (conv_umma_kernel<CIN, COUT, STAGED>), persistent_grid(1), Ring<CIN>::THREADS, smem, stream,
                       static_cast<const __half*>(c.in), static_cast<__half*>(c.out), c.nbr, c.order, c.tile_mask, c.out_num,
                       static_cast<const uint8_t*>(c.umma_weights), epi, c.relu, c.batch, c.max_voxels,
                       c.kvol, static_cast<__half*>(c.dense), reinterpret_cast<const int4*>(c.out_coors), c.D, c.H, c.W,
                       c.status, c.tile_counter, few_tiles(CIN, COUT, c.subm != 0, c.order != nullptr), c.maps_ready, c.debug_withhold_weights);
    return SESSD_OK;
}

}  // namespace

bool conv_umma_supported(int cin, int cout) {
    return (cin == 16 || cin == 32 || cin == 64) && (cout == 16 || cout == 32 || cout == 64);
}

// Weight tiles in the order the kernel consumes them: for stage g (a group of 64/Cin kernel offsets) a
// block of Cout rows x 128 bytes, row n holding K index kk = j*Cin + ci -> W[g*KG + j][ci][n], stored
// K-major with the 128-byte swizzle (16-byte chunk index XOR row index mod 8), zero beyond kvol.
int conv_umma_pack_weights(const float* weights, int kvol, int cin, int cout, void** device_out) {
    *device_out = nullptr;
    if (!conv_umma_supported(cin, cout)) return SESSD_OK;
    const int kg = 64 / cin, nstages = (kvol + kg - 1) / kg;
    std::vector<__half> img((size_t)nstages * cout * 64, __float2half_rn(0.f));
    for (int g = 0; g < nstages; ++g)
        for (int n = 0; n < cout; ++n)
            for (int kk = 0; kk < 64; ++kk) {
                const int k = g * kg + kk / cin, ci = kk % cin;
                if (k >= kvol) continue;
                const int chunk = kk / 8;
                const size_t pos = ((size_t)g * cout + n) * 64 + (size_t)((chunk ^ (n & 7)) * 8) + (kk % 8);
                img[pos] = __float2half_rn(weights[((size_t)k * cin + ci) * cout + n]);
            }
    void* d = nullptr;
    cudaError_t e = cudaMalloc(&d, img.size() * sizeof(__half));
    if (e == cudaSuccess) e = cudaMemcpy(d, img.data(), img.size() * sizeof(__half), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        set_cuda_error(e, "conv_umma_pack_weights");
        if (d) cudaFree(d);
        return SESSD_ERR_CUDA;
    }
    *device_out = d;
    return SESSD_OK;
}

int launch_conv_umma(const ConvLaunch& c, cudaStream_t stream) {
    if (c.dtype != SESSD_F16 || !c.umma_weights || !c.tile_mask || !c.tile_counter || c.kvol > KVOL_MAX) return SESSD_ERR_UNSUPPORTED;
#define SESSD_CASE(CI, CO) \
    if (c.cin == CI && c.cout == CO) return launch_one<CI, CO>(c, stream);
    SESSD_CASE(16, 16)
    SESSD_CASE(16, 32)
    SESSD_CASE(32, 32)
    SESSD_CASE(32, 64)
    // (a layer with the scatter has no groups: it takes the kernel whose code the layers before it have fetched, front end of 1 x 20,000
    // points 190.2 and 188.8 us)
    if (c.cin == 64 && c.cout == 64 && (c.kvol > STAGED_KVOL || c.dense)) return launch_one<64, 64, true>(c, stream);
    SESSD_CASE(64, 64)
#undef SESSD_CASE
    return SESSD_ERR_UNSUPPORTED;
}

}  // namespace sessd
