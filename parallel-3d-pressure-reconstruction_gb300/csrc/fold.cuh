// Between the row-major volumes and the walks' skewed copies (Layout).
//
// A plane of a skewed copy is a diagonal of every z slice, so a kernel that writes or reads the
// copies voxel by voxel touches a sector per voxel and copy.  These work on tiles of 32 x 32
// voxels of one z slice in shared memory: the row-major side goes row by row, the skewed side
// diagonal by diagonal (i + j or i - j constant), whose voxels are contiguous in the copy.  The
// tile's pitch of 32 keeps rows and both kinds of diagonals free of bank conflicts.
#pragma once

#include <cuda_runtime.h>

#include "omni3d_internal.h"
#include "walk.cuh"

namespace omni3d {

constexpr int kTile = 32, kTileThreads = 256;

// The tiles' rounds through shared memory take 15 us of latency until their blocks fill the SMs:
// smaller volumes are written and read voxel by voxel.  A selected sweep (field packed, pressure
// spread, sums folded) with tiles and by voxels, 162 directions: 28^3 156 and 135 us, 64^3 396 and
// 376, 80^3 631 and 629, 96^3 943 and 1006, 128^3 1966 and 2130.
constexpr long long kTileVoxels = 1LL << 19;
inline bool by_tiles(const Grid &g, const Layout &lay) { return lay.wrap && g.V >= kTileVoxels; }
inline unsigned voxel_blocks(const Grid &g) { return (unsigned)((g.V + kTileThreads - 1) / kTileThreads); }

inline unsigned tile_blocks(const Grid &g)
{
    const long long tx = (g.X + kTile - 1) / kTile, ty = (g.Y + kTile - 1) / kTile;
    return (unsigned)(tx * ty * g.Z);
}

// The tile of this block: its first voxel (i0, j0) and its slice k.
struct TileAt {
    int i0, j0, k;
    __device__ __forceinline__ TileAt(const Grid &g)
    {
        const unsigned tx = (unsigned)(g.X + kTile - 1) / kTile, ty = (unsigned)(g.Y + kTile - 1) / kTile;
        const unsigned b = blockIdx.x, row = b / tx;
        i0 = (int)(b - row * tx) * kTile;
        k = (int)(row / ty);
        j0 = (int)(row - (unsigned)k * ty) * kTile;
    }
    // Runs f(place in the tile, voxel, i, j) for the tile's voxels, row by row.
    template <typename F>
    __device__ __forceinline__ void rows(const Grid &g, F &&f) const
    {
        const int i = i0 + (threadIdx.x & 31);
        for (int r = threadIdx.x >> 5; r < kTile; r += kTileThreads / 32) {
            const int j = j0 + r;
            if (i < g.X && j < g.Y) f(32 * r + (threadIdx.x & 31), (long long)i + (long long)j * g.X + (long long)k * g.XY, i, j);
        }
    }
    // Runs f(place in the tile, index in a copy of class c) for the tile's voxels, diagonal by
    // diagonal (classes c and c ^ 2 have the same diagonals).
    template <typename F>
    __device__ __forceinline__ void diagonals(const Grid &g, const Layout &lay, int c, F &&f) const
    {
        const int lane = threadIdx.x & 31, i = i0 + lane;
        for (int d = threadIdx.x >> 5; d < 2 * kTile - 1; d += kTileThreads / 32) {
            const int r = (c & 1) ? lane - (d - (kTile - 1)) : d - lane;  // i - j or i + j constant
            const int j = j0 + r;
            if (r >= 0 && r < kTile && i < g.X && j < g.Y) f(32 * r + lane, layout_index(lay, g.X, g.Y, c, i, j, k));
        }
    }
};

__device__ __forceinline__ void fold_add(float &a, const float &b) { a += b; }
__device__ __forceinline__ void fold_add(double &a, const double &b) { a += b; }
__device__ __forceinline__ void fold_add(long long &a, const long long &b) { a += b; }
__device__ __forceinline__ void fold_add(float2 &a, const float2 &b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ void fold_add(double2 &a, const double2 &b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ void fold_add(uint32_t &a, const uint32_t &b) { a += b; }

template <typename T>
__device__ __forceinline__ T fold_load(const T *in, size_t i)
{
    return __ldg(in + i);
}

// f(voxel, sum of the copies' entries of it) for every voxel; the copies are added in the order
// of their classes.  256^3, float2: 0.45 -> 0.33 ms against one gather per voxel and copy.
template <typename IN, typename F>
__global__ void __launch_bounds__(kTileThreads) k_fold(Grid g, Layout lay, IN in, F f)
{
    using T = decltype(fold_load(in, 0));
    __shared__ T tile[kTile * kTile];
    const TileAt at(g);
    for (int c = 0; c < 4; c++) {
        const size_t copy = (size_t)c * (size_t)lay.stride;
        at.diagonals(g, lay, c, [&](int p, uint32_t q) {
            T x = fold_load(in, copy + q);
            if (c) {
                T s = tile[p];
                fold_add(s, x);
                x = s;
            }
            tile[p] = x;
        });
        __syncthreads();
    }
    at.rows(g, [&](int p, long long v, int, int) { f(v, tile[p]); });
}
template <typename IN, typename F>
__global__ void __launch_bounds__(kTileThreads) k_fold_voxels(Grid g, Layout lay, IN in, F f)
{
    const long long v = (long long)blockIdx.x * kTileThreads + threadIdx.x;
    if (v >= g.V) return;
    if (!lay.wrap) {
        f(v, fold_load(in, (size_t)v));
        return;
    }
    const VoxelAt at(g, v);
    auto x = fold_load(in, layout_index(lay, g.X, g.Y, 0, at.i, at.j, at.k));
#pragma unroll
    for (int c = 1; c < 4; c++)
        fold_add(x, fold_load(in, (size_t)c * (size_t)lay.stride + layout_index(lay, g.X, g.Y, c, at.i, at.j, at.k)));
    f(v, x);
}
template <typename IN, typename F>
cudaError_t fold_copies(const Grid &g, const Layout &lay, const IN &in, const F &f, cudaStream_t st)
{
    if (by_tiles(g, lay)) k_fold<<<tile_blocks(g), kTileThreads, 0, st>>>(g, lay, in, f);
    else k_fold_voxels<<<voxel_blocks(g), kTileThreads, 0, st>>>(g, lay, in, f);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

}  // namespace omni3d
