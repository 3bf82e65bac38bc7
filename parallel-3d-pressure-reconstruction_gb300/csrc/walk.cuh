// The walk along one line's staircase, shared by the sweep, operator and adjoint kernels,
// and the volume layouts it can address.
//
// A warp walks one group: up to 32 lines of one direction through one tile of lattice points,
// all at the same level.  The level of a voxel is the signed sum s_x i + s_y j + s_z k over
// the direction's step signs; every step raises it by one, so lines that start together stay
// together.  The group's step words begin with idle codes on the lanes whose lines enter at a
// higher level, and end with them on the lanes whose lines leave earlier.
//
// Over a row-major volume a level brings nothing: no two of its voxels share a row.  There every lane
// starts at its own entry (OWN), its step words shifted past the idle codes: neighbouring lines
// that enter by one face then read and write its rows together, and the warp is done after its
// longest line.  64^3 / 642 directions, a row-major sweep: 1.41 -> 1.18 ms (1.12 before groups were
// aligned by level, with warps of any 32 lines).
//
// A line's voxel addresses follow from its 2-bit steps alone, not from the values loaded
// along it.  The walk therefore decodes a batch of B steps, issues the B gathers (and, with
// AUX, B loads of an int32 per voxel from `aux`) before using any of them.  Without the batch
// each step's gather waits for the previous step's arithmetic, and a warp spends most of its
// time waiting on L2 latency.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "omni3d_internal.h"
#include "sums.cuh"

namespace omni3d {

constexpr int kIdle = 3;  // step code of a lane that takes no step

// What a walk gathers per step: nothing; the voxel's float4 (ax, ay, az, curl); or its edge
// record, the trapezoid increments by which a line of the octant enters the voxel along x, y
// and z, and the curl (k_pack).
enum WalkGrad { kNoGrad = 0, kGradVoxel = 1, kGradEdge = 2 };

// The arrays a walk gathers from.
struct WalkField {
    const float4 *voxel = nullptr;  // the float4 field (row-major layout)
    const float4 *edge = nullptr;   // 8 octants x V edge records (skewed layout)
};

// The lines a walking kernel runs over.
struct WalkLines {
    const GroupRec *groups;
    long long n_groups;
    const LineRec *lines;
    const uint32_t *desc;
};

// Coordinates of a row-major voxel index.
struct VoxelAt {
    int i, j, k;
    __device__ __forceinline__ VoxelAt(const Grid &g, long long v)
    {
        const uint32_t u = (uint32_t)v, row = u / (uint32_t)g.X;
        i = (int)(u - row * (uint32_t)g.X);
        k = (int)(row / (uint32_t)g.Y);
        j = (int)(row - (uint32_t)k * (uint32_t)g.Y);
    }
};

// Idle steps before a lane's line enters, which bring the group's lines to one level: sg its step
// signs, ds its direction's.  A line that moves against its direction's signs (directions with k3 = 0
// have some, see om_cross2point) starts at once.  Every lane of the warp calls it.
__device__ __forceinline__ int line_lag(int ie, int je, int ke, int sg, int ds)
{
    const bool regular = sg == (ds & 7);
    const int level = ((ds & 1) ? ie : -ie) + ((ds & 2) ? je : -je) + ((ds & 4) ? ke : -ke);
    const int low = __reduce_min_sync(0xffffffffu, regular ? level : 0x7fffffff);
    return regular ? level - low : 0;
}

// One lane of a group: its line (none on the lanes beyond the group's lines) and where and
// how it steps in the layout's copy for its step signs.
struct LineWalk {
    uint32_t v;           // index of the current voxel in the copy
    uint32_t wv;          // added when a step leaves the copy's range (see Layout)
    int d0, d1, d2;       // index strides of a step along x, y, z
    float h0, h1, h2;     // -rho * sign * spacing / 2 per axis (K:1816, 1825, 1834; in the edge records already)
    uint32_t e;           // entry voxel, row-major
    uint32_t span;        // steps of the group, idle ones included
    size_t copy;          // first entry of the copy
    int oct;              // step-sign octant: 2 x class + (upward)
    bool on;              // the lane has a line of its own (the lanes beyond the group's repeat the last one)
    uint32_t line;        // that line
    const uint32_t *dp;   // this lane's first step word
    uint32_t m;           // steps of the line
    uint32_t words;       // OWN: words at dp,
    uint32_t shift;       // bits of the first one before the line's first step

    // False when the warp has no group (whole warps).  OWN: the lane starts at its own entry.
    template <bool OWN = false>
    __device__ __forceinline__ bool init(const Grid &g, const Layout &lay, const WalkLines &W)
    {
        const long long gi = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        if (gi >= W.n_groups) return false;
        const int lane = threadIdx.x & 31;
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(W.groups) + gi);
        const uint32_t count = q.w & kGroupCount;
        on = (uint32_t)lane < count;
        line = q.x + min((uint32_t)lane, count - 1u);
        const uint4 r = __ldg(reinterpret_cast<const uint4 *>(W.lines) + line);
        span = q.z;
        dp = W.desc + 32ull * q.y + lane;
        e = r.x;
        const uint32_t X = (uint32_t)g.X, Y = (uint32_t)g.Y;
        const int ie = (int)(r.x % X), je = (int)((r.x / X) % Y), ke = (int)(r.x / (uint32_t)g.XY);
        const int ix = (int)(r.y % X), jx = (int)((r.y / X) % Y), kx = (int)(r.y / (uint32_t)g.XY);
        const int ds = (int)(q.w >> kGroupSigns), sg = line_signs(ie, je, ke, ix, jx, kx, ds);
        m = r.w;
        if (OWN) {
            const uint32_t lag = (uint32_t)line_lag(ie, je, ke, sg, ds);
            words = ((span + 15u) >> 4) - (lag >> 4);
            dp += 32u * (lag >> 4);
            shift = 2u * (lag & 15u);
            span = __reduce_max_sync(0xffffffffu, m);
        }
        const int si = (sg & 1) ? 1 : -1, sj = (sg & 2) ? 1 : -1, sk = (sg & 4) ? 1 : -1;
        // the reference forms -rho*s*dl in float and halves it in double (exact)
        h0 = __fmul_rn(-g.rho * (float)si, g.dx) * 0.5f;
        h1 = __fmul_rn(-g.rho * (float)sj, g.dy) * 0.5f;
        h2 = __fmul_rn(-g.rho * (float)sk, g.dz) * 0.5f;
        if (lay.wrap) {  // skewed copies: every step moves one plane up or down
            const int up = si * lay.XZ;
            d0 = up + si;
            d1 = up;
            d2 = up + sk * g.X;
            wv = si > 0 ? 0u - lay.wrap : lay.wrap;
            const int c = layout_class(sg);
            copy = (size_t)c * (size_t)lay.stride;
            oct = 2 * c + (sg & 1);
            v = layout_index(lay, g.X, g.Y, c, ie, je, ke);
        } else {
            d0 = si;
            d1 = sj * g.X;
            d2 = sk * (int)g.XY;
            wv = 0u;
            copy = 0;
            oct = 0;
            v = r.x;
        }
        return true;
    }

    // Word i of the lane's stored steps, OWN (idle past them), and the codes of its own steps 16 i on.
    __device__ __forceinline__ uint32_t stored(uint32_t i) const { return i < words ? __ldg(dp + 32u * i) : 0xffffffffu; }
    __device__ __forceinline__ uint32_t own(uint32_t i) const { return __funnelshift_r(stored(i), stored(i + 1), shift); }

    // The next voxel along axis code a (0, 1, 2).
    __device__ __forceinline__ void step(int a)
    {
        v += (uint32_t)(a == 0 ? d0 : (a == 1 ? d1 : d2));
        v = min(v, v + wv);
    }
};

// Steps of a batch as predicates: bits 2q, 2q + 1 of `c` hold the code of step q, bit 2q of
// `idle` tells that the lane does not take it.
__device__ __forceinline__ bool is_x(uint32_t c, int q) { return (c & (3u << (2 * q))) == 0u; }
__device__ __forceinline__ bool is_y(uint32_t c, int q) { return (c & (3u << (2 * q))) == (1u << (2 * q)); }
template <bool MASK>
__device__ __forceinline__ bool taken(uint32_t idle, int q)
{
    return !MASK || (idle & (1u << (2 * q))) == 0u;
}

// x, y or z by the axis of step q.  Written as selections by the code's two bits: from
// conditional expressions the compiler makes a three-way branch, which diverges at almost every
// step.
__device__ __forceinline__ uint32_t by_axis(uint32_t c, int q, uint32_t x, uint32_t y, uint32_t z)
{
    uint32_t r;
    asm("{\n\t.reg .pred py, pz;\n\t.reg .b32 t, u;\n\t"
        "and.b32 t, %4, %5;\n\t"
        "setp.ne.u32 pz, t, 0;\n\t"
        "and.b32 u, %4, %6;\n\t"
        "setp.ne.u32 py, u, 0;\n\t"
        "selp.b32 t, %2, %1, py;\n\t"
        "selp.b32 %0, %3, t, pz;\n\t}"
        : "=r"(r)
        : "r"(x), "r"(y), "r"(z), "r"(c), "r"(2u << (2 * q)), "r"(1u << (2 * q)));
    return r;
}
__device__ __forceinline__ float by_axis(uint32_t c, int q, float x, float y, float z)
{
    return __uint_as_float(by_axis(c, q, __float_as_uint(x), __float_as_uint(y), __float_as_uint(z)));
}

// Address of entry v of an array, as one wide multiply-add: the shifted add that the compiler
// takes is two instructions on the ALU, the busiest unit of a selected sweep.
template <typename T>
__device__ __forceinline__ T *entry(T *base, uint32_t v)
{
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(v), "n"(sizeof(T)), "l"((uint64_t)base));
    return reinterpret_cast<T *>(r);
}

// Least and greatest of a batch's curls (the magnitudes with ABS), NaN when one of them is NaN.
// One pair of comparisons then decides for the batch what would take a pair for every step.
__device__ __forceinline__ float min_nan(float a, float b, float c)
{
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b, float c)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
template <bool ABS, int B>
__device__ __forceinline__ void curl_range(const float4 (&g)[B], float &lo, float &hi)
{
    auto w = [&](int q) { return ABS ? fabsf(g[q].w) : g[q].w; };
    lo = hi = w(0);
#pragma unroll
    for (int q = 1; q < B; q += 2) {
        lo = min_nan(lo, w(q), w(q + 1 < B ? q + 1 : q));
        hi = max_nan(hi, w(q), w(q + 1 < B ? q + 1 : q));
    }
}

// The trapezoid increment of step q, gv the sample of the voxel it enters and gl that of the
// voxel before (an edge record holds the increments of the octant's steps).  Its roundings are
// named, as are those of the sums it enters: an expression that the compiler may fuse with the next
// addition would give other bits than the stored product of an edge record.
template <int GRAD>
__device__ __forceinline__ float step_increment(const LineWalk &L, uint32_t c, int q, const float4 &gv, const float4 &gl)
{
    if (GRAD == kGradEdge) return by_axis(c, q, gv.x, gv.y, gv.z);
    return __fmul_rn(by_axis(c, q, L.h0, L.h1, L.h2),
                     by_axis(c, q, __fadd_rn(gv.x, gl.x), __fadd_rn(gv.y, gl.y), __fadd_rn(gv.z, gl.z)));
}

// The curl sum of the selected method after a voxel of curl cn.
__device__ __forceinline__ float add_curl(float csum, float cn) { return __fmaf_rn(cn, 1.0e-4f, csum); }

// The array a walk gathers from, at the lane's copy.
template <int GRAD>
__device__ __forceinline__ const float4 *lane_field(const WalkField &f, const Layout &lay, const LineWalk &L)
{
    if (GRAD == kGradEdge) return f.edge + (size_t)L.oct * (size_t)lay.stride;
    return f.voxel;  // row-major layouts only
}
template <int GRAD>
__device__ __forceinline__ float4 sample(const float4 *field, uint32_t v)
{
    return GRAD == kNoGrad ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(field + v);
}

// State of the selected method along a line (K:2280-2537): inside a segment (run), or before
// the first one or between two (a good voxel then starts one).  The decisions of a step depend
// on the curl of the voxel it enters alone.  One integer instead of two flags, which the compiler
// packs into bits and unpacks at every step: 64^3 sweep 1.29 -> 1.25 ms.
struct SelectState {
    int phase;  // 0 before the first segment, 1 inside one, 2 between two
    __device__ __forceinline__ void enter(float curl, float thr) { phase = (curl == 0.0f || curl > thr) ? 0 : 1; }
    __device__ __forceinline__ bool run() const { return phase == 1; }
    // A step along x, y or z into a voxel of curl cn, taken when `on`: `add`, it adds to the
    // segment; `start`, a segment (re)starts at the voxel; `clear`, that start also clears the
    // running curl sum and count (a restart on a z step keeps them).
    __device__ __forceinline__ void step(bool x, bool y, bool on, float cn, float thr, bool &add, bool &start, bool &clear)
    {
        const bool nz = cn != 0.0f;
        const bool good = (cn < thr) & nz;
        const bool pause = (cn >= thr) | (x & !nz);
        const bool inside = phase == 1, fresh = phase == 0;
        add = on & inside & good;
        start = on & !inside & (good | (fresh & nz & !x));
        clear = start & (fresh | x | y);
        phase = start ? 1 : (on & inside & pause ? 2 : phase);
    }
    // Whether the step after a voxel of curl cn can start a segment (it cannot after a voxel
    // that is good: that one is in a segment or starts one).
    static __device__ __forceinline__ bool may_start_after(float cn, float thr) { return !((cn < thr) & (cn != 0.0f)); }
};

// Walks the group's lines in batches of B steps (aux points at the lane's copy).  Each batch
// goes to f in one of three forms:
//   f.batch<false>(codes, 0, voxels, samples, aux values) when every lane takes all B steps and
//     f.quick<false>(0, samples, aux values) holds on every lane: no line enters, leaves or
//     changes its state, so that code needs no branches;
//   f.batch<true>(codes, idle, ...) when some lane takes only some of the steps and
//     f.quick<true>(idle, ...) holds on every lane (the ends of the groups: a third of the
//     batches at 96^3, an eighth at 256^3);
//   f.general<false or true>(...) otherwise.
// The lanes beyond the group's lines take no steps.  OWN: as L was initialised; a lane then gathers
// nothing for a step that it does not take (1.18 -> 1.11 ms; over skewed copies it gathers its last
// voxel again: the selected method's walks, bound by the ALU, were 2 % slower with the tests).
template <int B, int GRAD, bool AUX, bool OWN, typename F>
__device__ __forceinline__ void walk_steps(LineWalk &L, const float4 *field, const int32_t *aux, F &f)
{
    static_assert(16 % B == 0, "a batch may not straddle step words");
    constexpr uint32_t kOnes = 0x55555555u & ((1u << (2 * B)) - 1u);
    const uint32_t off = L.on ? 0u : 0xffffffffu;
    uint32_t next = L.span ? __ldg(L.dp) : 0u, after = OWN ? L.stored(1) : 0u;
    for (uint32_t s0 = 0; s0 < L.span; s0 += 16) {
        uint32_t w = (OWN ? __funnelshift_r(next, after, L.shift) : next) | off;
        if (OWN) {
            next = after;
            after = L.stored((s0 >> 4) + 2);
        } else if (s0 + 16 < L.span) {
            next = __ldg(L.dp + 2 * s0 + 32);
        }
        const uint32_t n = min(16u, L.span - s0);  // codes past the span are idle
        for (uint32_t t0 = 0; t0 < n; t0 += B) {
            const uint32_t c = w;
            w >>= 2 * B;
            uint32_t vv[B];
            float4 g[B];
            int32_t xw[B];
            const uint32_t idle = c & (c >> 1) & kOnes;
            const bool all = __all_sync(0xffffffffu, idle == 0u);
            if (all) {
#pragma unroll
                for (int q = 0; q < B; q++) {
                    L.v += by_axis(c, q, (uint32_t)L.d0, (uint32_t)L.d1, (uint32_t)L.d2);
                    L.v = min(L.v, L.v + L.wv);
                    vv[q] = L.v;
                }
            } else {
#pragma unroll
                for (int q = 0; q < B; q++) {
                    const uint32_t d = by_axis(c, q, (uint32_t)L.d0, (uint32_t)L.d1, (uint32_t)L.d2);
                    L.v += taken<true>(idle, q) ? d : 0u;
                    L.v = min(L.v, L.v + L.wv);
                    vv[q] = L.v;
                }
            }
            if (all | !OWN) {
#pragma unroll
                for (int q = 0; q < B; q++) {
                    g[q] = sample<GRAD>(field, vv[q]);
                    xw[q] = AUX ? __ldg(aux + vv[q]) : 0;
                }
            } else {
#pragma unroll
                for (int q = 0; q < B; q++) {
                    g[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    xw[q] = -1;
                    if (taken<true>(idle, q)) {
                        g[q] = sample<GRAD>(field, vv[q]);
                        if (AUX) xw[q] = __ldg(aux + vv[q]);
                    }
                }
            }
            if (all) {
                if (__all_sync(0xffffffffu, f.template quick<false>(0u, g, xw))) f.template batch<false>(c, 0u, vv, g, xw);
                else f.template general<false>(c, 0u, vv, g, xw);
            } else {
                if (__all_sync(0xffffffffu, f.template quick<true>(idle, g, xw))) f.template batch<true>(c, idle, vv, g, xw);
                else f.template general<true>(c, idle, vv, g, xw);
            }
        }
    }
}

}  // namespace omni3d
