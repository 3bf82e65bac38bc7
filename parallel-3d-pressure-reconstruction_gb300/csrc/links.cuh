// Rows of the anchor operator and of its transpose, as the iterations read them.
//
// A row's links are (index, weight) pairs, one load each, or for unit weights (plain method)
// 16-byte vectors, the row's start aligned, of four 32-bit indices or of eight 16-bit ones.  The
// gathered vector is kept in shared memory where it fits: the links of a row point all over the
// volume's faces, so every lane's 4-byte gather is a sector of its own through L2 (293 G gathers/s)
// but at worst a bank conflict in shared memory.  Up to kIterSplitMax anchors the columns are
// split into two panels that fit one after the other, a row being two rows of 16-bit links, one
// per panel, each with room for all of the row's links (as many bytes as 32-bit links take).
// 128^3 / 642 directions (97 K anchors, 61 M links): 96 us an iteration with 32-bit links through
// L1, 76 us with two panels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace omni3d {

enum LinkKind { kLinkPair = 0, kLink32 = 1, kLink16 = 2 };

// Links per load of a row.
__host__ __device__ constexpr int links_per_vector(int kind) { return kind == kLinkPair ? 1 : (kind == kLink32 ? 4 : 8); }

// Bytes of a link.
__host__ __device__ constexpr size_t link_size(int kind) { return kind == kLinkPair ? 8 : (kind == kLink32 ? 4 : 2); }

// Lanes that share a row: a row of the 642-direction operators (about 640 links) is then 10 to
// 20 loads per lane, four of them in flight, and a warp works on several rows at once.
__host__ __device__ constexpr int lanes_per_row(int kind) { return kind == kLinkPair ? 32 : (kind == kLink32 ? 16 : 8); }

// add(index, weight, i) for the links of this lane (of lanes_per_row) of a row of m links at
// `links` (entry j0, aligned); i: the link's place in its unrolled load, known at compile time.
template <int KIND, typename F>
__device__ __forceinline__ void row_links(const void *links, unsigned long long j0, uint32_t m, int lane, F &&add)
{
    constexpr uint32_t S = lanes_per_row(KIND);
    uint32_t v = lane;
    if constexpr (KIND == kLinkPair) {
        const uint2 *q = static_cast<const uint2 *>(links) + j0;
        for (; v < m; v += 4 * S) {
            uint2 x[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (v + u * S < m) x[u] = __ldg(q + v + u * S);
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (v + u * S < m) add(x[u].x, __uint_as_float(x[u].y), u);
        }
    } else {
        constexpr uint32_t W = links_per_vector(KIND);
        const uint4 *q = static_cast<const uint4 *>(links) + j0 / W;
        auto at = [](const uint4 &x, uint32_t k) {
            const uint32_t a[4] = {x.x, x.y, x.z, x.w};
            return KIND == kLink32 ? a[k] : (a[k / 2] >> (16 * (k & 1))) & 0xffffu;
        };
        const uint32_t full = m / W;  // whole vectors
        for (; v + 3 * S < full; v += 4 * S) {
            uint4 x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = __ldg(q + v + u * S);
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (uint32_t k = 0; k < W; k++) add(at(x[u], k), 1.0f, (int)k);
        }
        for (; v < full; v += S) {
            const uint4 x = __ldg(q + v);
#pragma unroll
            for (uint32_t k = 0; k < W; k++) add(at(x, k), 1.0f, (int)k);
        }
        if (v == full && W * full < m) {  // the slots past the row's links hold nothing
            const uint4 x = __ldg(q + full);
#pragma unroll
            for (uint32_t k = 0; k < W; k++)
                if (W * full + k < m) add(at(x, k), 1.0f, (int)k);
        }
    }
}

// Store link `slot`.
template <int KIND>
__device__ __forceinline__ void store_link(void *links, unsigned long long slot, uint32_t index, float weight)
{
    if (KIND == kLinkPair) static_cast<uint2 *>(links)[slot] = make_uint2(index, __float_as_uint(weight));
    else if (KIND == kLink32) static_cast<uint32_t *>(links)[slot] = index;
    else static_cast<uint16_t *>(links)[slot] = (uint16_t)index;
}

// The vector an iteration gathers from: copied into shared memory (SMEM) or read through L1.
constexpr int kIterSmemMax = 216 * 1024;  // bytes of it: beside the rows' sums, what an SM gives one CTA
constexpr long long kIterPanelMax = kIterSmemMax / 4, kIterSplitMax = 2 * kIterPanelMax;
template <bool SMEM>
__device__ __forceinline__ const float *gather_vector(const float *x, long long n, float *sh)
{
    if (!SMEM) return x;
    const long long n4 = n / 4;  // (the iterates' buffers are 256-byte aligned)
    for (long long i = threadIdx.x; i < n4; i += blockDim.x)
        reinterpret_cast<float4 *>(sh)[i] = __ldg(reinterpret_cast<const float4 *>(x) + i);
    for (long long i = 4 * n4 + threadIdx.x; i < n; i += blockDim.x) sh[i] = __ldg(x + i);
    __syncthreads();
    return sh;
}

// Launch shape of an iteration over n rows: CTAs of 256 threads, or with the vector in shared
// memory one CTA of 1024 per SM, and rows per warp.  alone: the iteration does not
// share the GPU with others, as it does in a batch's graph, where kernels that fill the SMs'
// shared memory keep the members apart (16 plain snapshots: 15.6 ms so, 13.8 without).
// Vectors below kIterSmemMin stay in L1 anyway: 642 directions, 54^3 (17 K rows) 16.4 us through L1,
// 12.3 from shared memory, 72^3 26.7 and 18.5; 162 directions 9.7 and 8.4, 12.3 with either (60^3 to
// 68^3 10.3 and 12.3: a second row for some warps).
constexpr long long kIterSmemMin = 16384;
// (paired links always gather through L1: their stream takes longer than the gathers; 25 K anchors, 40^3
// selected: 44 us an iteration from shared memory, 32 through L1)
struct IterShape {
    bool smem;
    int threads, rows;
    unsigned blocks;
    size_t bytes;
};
// Rows per warp at most.  In shared memory enough for a single wave over kIterSplitMax rows; else
// more blocks end more evenly (paired links, 112^3 selected: 0.77 ms of iterations at 16, 0.81 at 24).
__host__ __device__ constexpr int iter_rows_max(bool smem) { return smem ? 24 : 16; }

// Columns of a panel of an operator of n anchors (whole 16-byte vectors), 0: not split.
inline uint32_t link_split(long long n, bool unit)
{
    return unit && n > kIterPanelMax && n <= kIterSplitMax ? (uint32_t)((n + 7) / 8 * 4) : 0u;
}
inline int link_kind(long long n, bool unit)
{
    return !unit ? kLinkPair : (n <= kIterSplitMax ? kLink16 : kLink32);
}

// uneven: the lines of the minimum-curl methods run together, and with them the links in a few rows; with
// paired links a block for every 8 rows then evens them out (96^3 / 642 directions, 54 K rows, 58 M
// links: 206 -> 121 us an iteration; unit links 120 us so, 98 from shared memory as ever).
inline IterShape iter_shape(long long n, bool alone, int kind, uint32_t split, bool uneven)
{
    IterShape s{};
    s.bytes = sizeof(float) * (split ? (size_t)split : (size_t)n);
    s.smem = alone && kind == kLink16 && n >= kIterSmemMin;
    s.threads = s.smem ? 1024 : 256;
    // with the vector in shared memory one CTA per SM (1024 threads at 48 to 64 registers): a shape for two
    // took 60^3 to 68^3 / 642 directions, 21 to 27 K rows, 22.6 instead of 18.5 us in two rounds
    // at least as many rows as a warp takes at once: fewer blocks then hand in fewer change sums (32^3
    // / 162 directions: 15.2 -> 12.3 us an iteration with its test)
    const long long warps = 152LL * (s.smem ? 32 : 48);
    const long long rows = (n + warps - 1) / warps, least = 32 / lanes_per_row(kind);
    s.rows = (int)(rows < least || (uneven && kind == kLinkPair) ? least : (rows > iter_rows_max(s.smem) ? iter_rows_max(s.smem) : rows));
    const long long per = (long long)s.rows * (s.threads / 32);
    s.blocks = (unsigned)((n + per - 1) / per);
    if (!s.smem) s.bytes = 0;
    return s;
}

}  // namespace omni3d
