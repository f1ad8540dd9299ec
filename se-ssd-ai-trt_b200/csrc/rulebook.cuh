// Device pieces of the rulebook that more than one kernel uses: the x-grouped coordinate table and the marking of
// candidate outputs in an occupancy grid.
#pragma once

#include "common.cuh"

namespace sessd {

// Integer helpers for the candidate geometry. Strides and candidate spans are 1, 2 or 3; a division by a
// run-time divisor costs some 25 instructions on the GPU and these kernels are bound by instruction issue,
// so the common divisors get shifts.
__device__ __forceinline__ int div_trunc(int a, int s) {   // C division (rounds toward zero)
    if (s == 1) return a;
    if (s == 2) return (a + (a < 0 ? 1 : 0)) >> 1;
    return a / s;
}
__device__ __forceinline__ void split_small(int e, int m, int* q, int* r) {   // e = q * m + r, e >= 0
    if (m == 1) {
        *q = e;
        *r = 0;
    } else if (m == 2) {
        *q = e >> 1;
        *r = e & 1;
    } else {
        *q = e / m;
        *r = e - *q * m;
    }
}

__device__ __forceinline__ unsigned long long rec_bits(const uint4& r) {
    return (unsigned long long)r.x | ((unsigned long long)r.y << 32);
}

// Position of the n-th set bit of v (n < popcount).
__device__ __forceinline__ int nth_bit(unsigned long long v, int n) {
    uint32_t x = (uint32_t)v;
    int pos = 0, c = __popc(x);
    if (n >= c) n -= c, x = (uint32_t)(v >> 32), pos = 32;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        c = __popc(x & ((1u << s) - 1u));
        if (n >= c) n -= c, x >>= s, pos += s;
    }
    return pos;
}

// Writes the coordinates of the cells of a warp's 32 words: lane's word `word` (of a grid with xw words per line and Y lines
// per plane) has `bits`, its cells the rows id, id + 1, .. of frame b, consecutive over the lanes. A lane per cell: it finds
// its word by bisection over the lanes. (A lane per cell of one word at a time keeps most lanes idle: words have some four
// cells.)
__device__ __forceinline__ void write_cells(int4* __restrict__ coors, int b, int xw, int Y, int word, unsigned long long bits,
                                            int id) {
    const int lane = threadIdx.x & 31;
    const int line = word / xw, z0 = line / Y, y0 = line - z0 * Y, x0 = (word - line * xw) << 6;   // of the word's first cell
    const int first = __shfl_sync(0xFFFFFFFFu, id, 0);
    const int end = __shfl_sync(0xFFFFFFFFu, id + __popcll(bits), 31);
    for (int r0 = first; r0 < end; r0 += 32) {
        const int r = r0 + lane;
        int src = 0;                                     // the last lane whose rows start at or before r
#pragma unroll
        for (int s = 16; s; s >>= 1)
            if (__shfl_sync(0xFFFFFFFFu, id, src + s) <= r) src += s;
        const int id0 = __shfl_sync(0xFFFFFFFFu, id, src);
        const unsigned long long v = __shfl_sync(0xFFFFFFFFu, bits, src);
        const int z = __shfl_sync(0xFFFFFFFFu, z0, src), y = __shfl_sync(0xFFFFFFFFu, y0, src), x = __shfl_sync(0xFFFFFFFFu, x0, src);
        if (r < end) coors[r] = make_int4(b, z, y, x + nth_bit(v, r - id0));
    }
}

// Enters row i of the cell with linear index `key` into a frame's x-grouped table; false when the table is full.
__device__ __forceinline__ bool bucket_insert(uint32_t* __restrict__ base, uint32_t cap, int shift, uint32_t key, int i) {
    const uint32_t gkey = key >> 2;
    uint32_t h = hash_slot(gkey, shift);
    for (uint32_t probe = 0; probe < cap; ++probe) {
        uint32_t* bk = base + (size_t)h * 8;
        uint32_t cur = bk[4];
        if (cur == kEmpty) cur = atomicCAS(&bk[4], kEmpty, gkey);
        if (cur == kEmpty || cur == gkey) {
            atomicMax(reinterpret_cast<int32_t*>(&bk[key & 3u]), i);  // duplicates: highest row wins
            return true;
        }
        h = (h + 1) & (cap - 1);
    }
    return false;
}

// Marks the candidate outputs of the input row at c4 = (b, z, y, x) in frame b's grid: the reference's enumeration
// (sparseConv3dlayer.cu:339-383). Per axis the row has up to three candidate output positions (one or two for the
// stride-2 layers); the x candidates of one (z, y) pair are neighbouring bits, mostly of one 64-bit word, so they are
// tested and set together, and all words are read before any is updated (the reads are independent; most of them find
// their bits already set by a neighbouring row and nothing is written).
__device__ __forceinline__ void mark_row(const int4& c4, int b, const ConvGeom& g, const BitGrid& out) {
    constexpr int MAXS = 3;   // span_max never exceeds the kernel size (<= 3)
    const int c[3] = {c4.y, c4.z, c4.w};
    // candidate positions per axis, upper corner downward; pos[j][e] < 0 marks an unusable candidate
    int pos[3][MAXS];
    bool in_ok = true;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        // C integer division, as in the reference (sparseConv3dlayer.cu:339-348); dilation is 1
        const int lo = div_trunc(c[j] - (g.K[j] - 1) - 1 + g.S[j] + g.P[j], g.S[j]);
        const int hi = div_trunc(c[j] + g.P[j], g.S[j]);
        in_ok = in_ok && c[j] >= 0 && c[j] < g.in_shape[j];
#pragma unroll
        for (int e = 0; e < MAXS; ++e) {
            const int o = hi - e;
            const int k = c[j] - o * g.S[j] + g.P[j];   // the offset this pair would get (:366)
            const bool ok = e < g.span_max[j] && e <= hi - lo && o >= 0 && o < g.out_shape[j] && k >= 0 && k < g.K[j];
            pos[j][e] = ok ? o : -1;
        }
    }
    if (!in_ok) return;
    // the x candidates as bits of at most two neighbouring words
    int w0 = -1;
    unsigned long long bits0 = 0ull, bits1 = 0ull;
#pragma unroll
    for (int e = 0; e < MAXS; ++e) {
        const int ox = pos[2][e];
        if (ox < 0) continue;
        if (w0 < 0) w0 = ox >> 6;            // candidates descend, so the first valid one has the highest word
        if ((ox >> 6) == w0) bits0 |= 1ull << (ox & 63);
        else bits1 |= 1ull << (ox & 63);     // the word below (spans are at most three cells)
    }
    if (w0 < 0) return;
    unsigned long long* base = reinterpret_cast<unsigned long long*>(out.rec + (size_t)b * out.words);
    unsigned long long cur0[MAXS * MAXS], cur1[MAXS * MAXS];
    size_t rec[MAXS * MAXS];
#pragma unroll
    for (int ez = 0; ez < MAXS; ++ez)
#pragma unroll
        for (int ey = 0; ey < MAXS; ++ey) {
            const int q = ez * MAXS + ey;
            const bool ok = pos[0][ez] >= 0 && pos[1][ey] >= 0;
            rec[q] = ok ? ((size_t)pos[0][ez] * out.Y + pos[1][ey]) * out.xw + w0 : (size_t)-1;
            // a record is 16 bytes: its bits are the first 8
            cur0[q] = ok ? *reinterpret_cast<volatile unsigned long long*>(base + 2 * rec[q]) : ~0ull;
            cur1[q] = (ok && bits1) ? *reinterpret_cast<volatile unsigned long long*>(base + 2 * (rec[q] - 1)) : ~0ull;
        }
#pragma unroll
    for (int q = 0; q < MAXS * MAXS; ++q) {
        if (rec[q] == (size_t)-1) continue;
        if ((cur0[q] & bits0) != bits0) atomicOr(base + 2 * rec[q], bits0);
        if (bits1 && (cur1[q] & bits1) != bits1) atomicOr(base + 2 * (rec[q] - 1), bits1);
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

// Last word of word w's record: the first two cells of the next word of the line, whose low bits (before any row is dropped)
// are `low` and whose rows begin at next_row.
__device__ __forceinline__ uint32_t next_cells(uint32_t low, int w, const BitGrid& g, int next_row, int max_voxels) {
    uint32_t c = low & 3u;
    if (next_row + 2 > max_voxels) c = next_row < max_voxels ? c & (0u - c) : 0u;
    return c && w + 1 < g.words && (w + 1) % g.xw != 0 ? c : 0u;
}

// Sets the bits `lo` of the grid word at rec[0] and `hi` of the next one, for up to four words. The words are read first,
// side by side and through L1: a stale copy only costs an atomic that changes nothing, and most bits have been set by a
// neighbouring word long before.
__device__ __forceinline__ void set_bits(uint4* const (&rec)[4], unsigned long long lo, unsigned long long hi) {
    unsigned long long cur[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) cur[i] = rec[i] ? *reinterpret_cast<const unsigned long long*>(rec[i]) : ~0ull;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if ((cur[i] & lo) != lo) atomicOr(reinterpret_cast<unsigned long long*>(rec[i]), lo);
    if (!hi) return;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (rec[i]) atomicOr(reinterpret_cast<unsigned long long*>(rec[i] + 1), hi);
}

// Marks, in the grids of all levels of a chain, the outputs of the cells of word (z, y, wx) of the voxeliser's level,
// given its bits. Per axis the outputs of a range of input cells are a range of output cells (sparseConv3dlayer.cu:339-348
// enumerates the same cells), so a word reaches at most two or three lines per axis of every level; in x the layers are
// those of derivable_in_x: kernel 1 and stride 1 (outputs are the cells themselves) or kernel 3, stride 2, padding 1
// (output x has the inputs 2x - 1, 2x, 2x + 1).
__device__ __forceinline__ void mark_levels(unsigned long long bits, int z, int y, int wx, int b, const LevelChain& chain) {
    int z0 = z, z1 = z, y0 = y, y1 = y, off = wx << 6;   // lines, and the cell of the lowest bit (even before every halving)
    for (int l = 0; l < chain.count && bits; ++l) {
        const ConvGeom& g = chain.geom[l];
        const BitGrid& out = chain.grid[l];
        z0 = div_trunc(max(z0 + g.P[0] - g.K[0] + g.S[0], 0), g.S[0]), z1 = min(div_trunc(z1 + g.P[0], g.S[0]), out.Z - 1);
        y0 = div_trunc(max(y0 + g.P[1] - g.K[1] + g.S[1], 0), g.S[1]), y1 = min(div_trunc(y1 + g.P[1], g.S[1]), out.Y - 1);
        if (z0 > z1 || y0 > y1) return;   // no output of this level, so none of the levels below (which an empty range would not say)
        if (g.K[2] == 3) {
            const unsigned long long even = even_bits(bits), odd = even_bits(bits >> 1);
            bits = even | odd | (odd << 1);
            off >>= 1;
        }
        if (off + 64 > out.X) bits &= off < out.X ? (1ull << (out.X - off)) - 1ull : 0ull;
        const int sh = off & 63;
        const unsigned long long lo = bits << sh, hi = sh ? bits >> (64 - sh) : 0ull;
        uint4* rec = out.rec + (size_t)b * out.words + (off >> 6);
        for (int oz = z0; oz <= z1; oz += 2)             // (rarely more than 2 x 2 lines)
            for (int oy = y0; oy <= y1; oy += 2) {
                uint4* at = rec + (oz * out.Y + oy) * out.xw;
                const bool z2 = oz < z1, y2 = oy < y1;
                uint4* const lines[4] = {at, y2 ? at + out.xw : nullptr, z2 ? at + out.Y * out.xw : nullptr,
                                         z2 && y2 ? at + (out.Y + 1) * out.xw : nullptr};
                set_bits(lines, lo, hi);
            }
    }
}

}  // namespace sessd
