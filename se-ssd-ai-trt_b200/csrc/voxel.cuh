// Device pieces of the voxelisers: cell of a point, a cell's list of its first points, the mean of the listed points.
#pragma once

#include "common.cuh"

namespace sessd {

constexpr int kMaxPointsPerVoxel = 8;   // largest max_points_per_voxel the parameter check accepts

struct VoxGeom {
    float x_min, x_max, y_min, y_max, z_min, z_max;
    float vx, vy, vz;
    int gx, gy, gz;
};
inline VoxGeom voxel_geom(const sessd_voxel_params& p) {
    return VoxGeom{p.x_min, p.x_max, p.y_min, p.y_max, p.z_min, p.z_max, p.voxel_x, p.voxel_y, p.voxel_z,
                   p.grid_x, p.grid_y, p.grid_z};
}

// Cell of a point, false outside the range: the tests and fp32 arithmetic of voxelGenerator.cu:363-375.
__device__ __forceinline__ bool voxel_cell(const VoxGeom& g, const float4& pt, int* ix, int* iy, int* iz) {
    if (!(pt.x >= g.x_min && pt.x < g.x_max && pt.y >= g.y_min && pt.y < g.y_max && pt.z >= g.z_min && pt.z < g.z_max))
        return false;
    *ix = (int)floorf(__fdiv_rn(__fsub_rn(pt.x, g.x_min), g.vx));
    *iy = (int)floorf(__fdiv_rn(__fsub_rn(pt.y, g.y_min), g.vy));
    *iz = (int)floorf(__fdiv_rn(__fsub_rn(pt.z, g.z_min), g.vz));
    return *ix >= 0 && *ix < g.gx && *iy >= 0 && *iy < g.gy && *iz >= 0 && *iz < g.gz;
}

// Keeps the max_pts smallest point indices of a cell, ascending, free places (kEmpty) at the end: offers the index to
// position 0; whatever loses a position (the larger value) is offered to the next.
__device__ __forceinline__ void list_push(uint32_t* list, int max_pts, uint32_t p) {
    uint32_t carry = p;
    for (int j = 0; j < max_pts; ++j) {
        const uint32_t old = atomicMin(&list[j], carry);
        if (old == kEmpty) break;
        carry = old > carry ? old : carry;
    }
}
__device__ __forceinline__ void list_load(const uint32_t* list, int max_pts, uint32_t (&pi)[kMaxPointsPerVoxel]) {
#pragma unroll
    for (int j = 0; j < kMaxPointsPerVoxel; ++j) pi[j] = j < max_pts ? list[j] : kEmpty;
}

// Mean as generateAverage_kernel (voxelGenerator.cu:274-296): left-to-right sum over all max_pts slots (unused slots
// contribute +0), divided by the number of listed points.
__device__ __forceinline__ float4 voxel_mean(const float4* __restrict__ points, int max_pts,
                                             const uint32_t (&pi)[kMaxPointsPerVoxel], int* count) {
    float4 v[kMaxPointsPerVoxel];
    int cnt = 0;
#pragma unroll
    for (int j = 0; j < kMaxPointsPerVoxel; ++j) {
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (pi[j] != kEmpty) {
            v[j] = __ldg(&points[pi[j]]);
            ++cnt;
        }
    }
    float sx = v[0].x, sy = v[0].y, sz = v[0].z, sw = v[0].w;
#pragma unroll
    for (int j = 1; j < kMaxPointsPerVoxel; ++j) {
        if (j >= max_pts) break;
        sx = __fadd_rn(sx, v[j].x);
        sy = __fadd_rn(sy, v[j].y);
        sz = __fadd_rn(sz, v[j].z);
        sw = __fadd_rn(sw, v[j].w);
    }
    const float fn = (float)cnt;
    *count = cnt;
    return make_float4(__fdiv_rn(sx, fn), __fdiv_rn(sy, fn), __fdiv_rn(sz, fn), __fdiv_rn(sw, fn));
}

__device__ __forceinline__ void store_voxel(float* voxels, size_t row, float x, float y, float z, float w) {
    reinterpret_cast<float4*>(voxels)[row] = make_float4(x, y, z, w);
}
__device__ __forceinline__ void store_voxel(__half* voxels, size_t row, float x, float y, float z, float w) {
    __half2 lo = __floats2half2_rn(x, y), hi = __floats2half2_rn(z, w);
    uint2 packed;
    packed.x = *reinterpret_cast<uint32_t*>(&lo);
    packed.y = *reinterpret_cast<uint32_t*>(&hi);
    reinterpret_cast<uint2*>(voxels)[row] = packed;
}

// Calls fn(frame, point) for every point of the batch, `blocks` blocks of kThreads threads sharing them.
template <class Fn>
__device__ __forceinline__ void for_points(const int32_t* __restrict__ points_size, int batch, int max_points, int block,
                                           int blocks, Fn fn) {
    const int chunks = (max_points + kThreads - 1) / kThreads;
    const int items = batch * chunks;
    for (int it = block; it < items; it += blocks) {
        const int b = it / chunks;
        const int p = (it - b * chunks) * kThreads + threadIdx.x;
        int n = __ldg(points_size + b);
        n = n > max_points ? max_points : n;
        if (p < n) fn(b, p);
    }
}

// Number of the record of an occupied word of a two-level grid.
__device__ __forceinline__ int word_id(const BitGrid& grid, int b, uint32_t word) {
    const uint4 t = load_late(grid.top + (size_t)b * grid.top_words + (word >> 6));
    const unsigned long long bits = (unsigned long long)t.x | ((unsigned long long)t.y << 32);
    return (int)t.z + __popcll(bits & ((1ull << (word & 63)) - 1ull));
}

// Pushes every point into the list of its row.
__device__ __forceinline__ void push_points(const PointLists& l, int batch, int block, int blocks) {
    for_points(l.points_size, batch, l.max_points, block, blocks, [&](int b, int p) {
        const uint32_t key = __ldg(l.pt_key + (size_t)b * l.max_points + p);
        if (key == kEmpty) return;
        const uint4 r = load_late(l.grid.rec + (size_t)b * l.grid.words + word_id(l.grid, b, key >> 6));
        const unsigned long long bits = (unsigned long long)r.x | ((unsigned long long)r.y << 32);
        const int row = (int)r.z + __popcll(bits & ((1ull << (key & 63)) - 1ull));
        list_push(l.lists + ((size_t)b * l.max_points + row) * l.max_pts, l.max_pts, (uint32_t)p);
    });
}

}  // namespace sessd
