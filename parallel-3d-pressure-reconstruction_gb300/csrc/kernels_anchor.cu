// Anchor operator: the reference iteration restricted to the voxels whose values feed back.
//
// In one iteration of the reference (K:8840-8861) a voxel v receives, from every line
// segment through it, w * (p[start] + I(v)) in pn and w in count (w = 1 for the plain
// method; the start is the line entry, K:1760-1761; for the weighted method the start is
// the entry and w = n / sum(curl/1e4) along the line, K:2086-2130; for the selected method
// the start is the voxel where the segment began or restarted, K:2301-2411, and
// w = n / sum(curl/1e4) along the segment).
// I(v) and w depend only on the gradient field, so
//     p_new(v) = (b(v) + sum_j w_j p_old(start_j)) / c(v),  b = sum w I,  c = sum w.
// Only the start voxels ("anchors") are ever read, so the iteration closes on the anchors:
// iterate p_a <- (b_a + M p_a) / c_a on them alone, then evaluate every voxel once from
// the final anchor values with one full sweep.  This gives the reference's iterate exactly
// (up to the order of floating-point sums) at a fraction of the cost.
//
// The operator is built from the same line descriptors as the sweep: a marking pass finds
// the anchors, the geometry's line counts size each anchor's row, a filling pass writes
// (column = start anchor, weight) pairs and accumulates b and c.  The filling pass learns
// whether a visited voxel is an anchor from the field gather itself: for the duration of
// the pass the anchors' field records carry a flag in a bit no value uses (the sign
// of the curl in .w, curl being non-negative), so a step costs one gather.  A field with a
// negative curl value gathers the anchor id beside it.
//
// The filling pass sums each line's integral in plain FP32 in step order, as the reference
// does (K:1816-1834); the final sweep, whose integrals reach every voxel directly, keeps
// compensated sums (the compensation took 2.7 ms of the pass's 52.7 ms at 256^3 / 642 directions).
//
// What bounds the filling pass (160^3, 642 directions, ncu): the plain method's the L1 data pipe
// (82-86 %: the 16-byte gathers), the selected method's the same pipe (73 %) beside the
// half-rate integer and selection pipe (62 %, 47 instructions per step).  256^3 / 642 directions,
// selected method, with the pass's setup: 44.3 -> 33.8 ms against the row-major walk.
#include <algorithm>

#include "fixed.cuh"
#include "links.cuh"
#include "omni3d_internal.h"
#include "walk.cuh"

namespace omni3d {

// Steps whose gathers a walk issues together: 4 beat 8 and 2 by 6 and 2 ms at 256^3 / 642
// directions.
constexpr int kWalkBatch = 4;
// Launch shape of the operator passes: 64 registers hold a batch with its records; at 48 (20
// CTAs) the selected method's pass spills 90 bytes and took 39.5 instead of 36.9 ms.  Small CTAs
// free their slots as soon as their own few lines end.
constexpr int kFillBlocks = 16;
constexpr int kFillThreads = 64;  // threads per CTA (whole warps: one line per thread)
constexpr uint32_t kAllIdle = 0x55555555u & ((1u << (2 * kWalkBatch)) - 1u);  // no step of the batch is the lane's

namespace {

// Whether a gathered voxel is an anchor: with FB the sign bit of its curl (the flag the filling
// pass sets in the field), else its anchor id gathered beside it.
template <bool FB>
__device__ __forceinline__ bool anchor_of(const float4 &gv, int32_t id)
{
    return FB ? (__float_as_uint(gv.w) >> 31) != 0u : id >= 0;
}

// Curl of a gathered voxel: under FB its sign bit is the anchor flag.
template <bool FB>
__device__ __forceinline__ float curl_of(const float4 &gv)
{
    return FB ? fabsf(gv.w) : gv.w;
}

enum Pass { kMark = 0, kFill = 2, kRhs = 3 };

struct Sink {
    const int32_t *id;   // the walks' copies of the anchor ids (-1: no anchor)
    uint8_t *flag;       // row-major (the marking pass walks the row-major layout)
    unsigned long long *next;  // per row: the next free link slot (starts at the row's first slot)
    void *links;     // per link the start anchor, and its weight in weighted operators (links.cuh)
    int kind;        // LinkKind
    uint32_t split;  // columns of a panel (links.cuh), 0: one panel
    float2 *bc;      // per row: (b, c)
    long long *bc64; // bit-reproducible mode: per row the fixed-point (b, c) instead of bc
    const double *fix;  // its scales (fixed.cuh)
};

// Record one contribution of weight wt and integral I into the anchor row `row` (-1: none) from
// the segment whose start anchor is scol (its id, loaded once per segment).  A link costs one
// row lookup, one 64-bit slot atomic, one store and one vector reduction of (b, c); UNIT
// operators (every weight 1) store no weight.
//
// take_slot reserves the link's slot (the row's next), put_link fills it.
template <bool UNIT>
__device__ __forceinline__ bool upper_panel(const Sink &S, uint32_t scol)
{
    return UNIT && S.split && scol >= S.split;
}
template <bool UNIT>
__device__ __forceinline__ unsigned long long take_slot(const Sink &S, int row, uint32_t scol)
{
    return atomicAdd(S.next + (UNIT && S.split ? 2u * (uint32_t)row + (upper_panel<UNIT>(S, scol) ? 1u : 0u) : (uint32_t)row), 1ull);
}
template <bool UNIT>
__device__ __forceinline__ void put_link(const Sink &S, int row, unsigned long long slot, uint32_t scol, float wt, float I)
{
    if (upper_panel<UNIT>(S, scol)) scol -= S.split;
    const float bt = UNIT ? I : wt * I, ct = UNIT ? 1.0f : wt;
    if (!UNIT) store_link<kLinkPair>(S.links, slot, scol, wt);
    else if (S.kind == kLink16) store_link<kLink16>(S.links, slot, scol, wt);
    else store_link<kLink32>(S.links, slot, scol, wt);
    if (S.bc64) {  // bit-reproducible: exact, order-independent fixed-point row sums
        fix_add(S.bc64 + 2 * row, bt, fix_scale(S.fix[kFixB]));
        fix_add(S.bc64 + 2 * row + 1, ct, fix_scale(S.fix[kFixC]));
    } else {
        atomicAdd(S.bc + row, make_float2(bt, ct));
    }
}
// Plain method, operator cached: only b = sum I is field-dependent.
__device__ __forceinline__ void put_rhs(const Sink &S, int row, float I)
{
    if (S.bc64) fix_add(S.bc64 + 2 * row, I, fix_scale(S.fix[kFixB]));
    else atomicAdd(&S.bc[row].x, I);
}
template <int PASS, bool UNIT>
__device__ __forceinline__ void emit_w(const Sink &S, int row, uint32_t scol, float wt, float I)
{
    if (row < 0) return;  // not an anchor after all: nothing to index
    if (PASS == kRhs) {
        put_rhs(S, row, I);
        return;
    }
    if (PASS == kFill && (int)scol < 0) return;  // a start that is no anchor: no column to link
    put_link<UNIT>(S, row, take_slot<UNIT>(S, row, scol), scol, wt, I);
}

// The contributions of a batch's steps `todo` (bits 2q) into the anchors they enter, unit weights:
// the row lookups of all steps wait together, then their slots (128^3: 3.02 -> 2.98 ms against a
// step at a time; the weighted forms have no registers for it and spill: 29.0 -> 32.4 ms at 256^3).
template <int PASS>
__device__ __forceinline__ void emit_units(const Sink &S, uint32_t todo, const uint32_t (&v)[kWalkBatch], uint32_t scol,
                                           const float (&I)[kWalkBatch])
{
    int rows[kWalkBatch];
    unsigned long long slot[kWalkBatch];
#pragma unroll
    for (int q = 0; q < kWalkBatch; q++) {
        rows[q] = -1;
        if (todo & (1u << (2 * q))) rows[q] = __ldg(S.id + v[q]);
        if (PASS == kFill && (int)scol < 0) rows[q] = -1;
    }
    if (PASS == kFill) {
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++)
            if (rows[q] >= 0) slot[q] = take_slot<true>(S, rows[q], scol);
    }
#pragma unroll
    for (int q = 0; q < kWalkBatch; q++) {
        if (rows[q] < 0) continue;
        if (PASS == kFill) put_link<true>(S, rows[q], slot[q], scol, 1.0f, I[q]);
        else put_rhs(S, rows[q], I[q]);
    }
}

// The anchor id of a segment's start voxel, for the filling pass's links.
template <int PASS>
__device__ __forceinline__ uint32_t start_col(const Sink &S, uint32_t start)
{
    return PASS == kFill ? (uint32_t)__ldg(S.id + start) : 0u;
}

// Element q of a batch's registers, q not known at compile time.
template <typename T>
__device__ __forceinline__ T pick(const T (&x)[kWalkBatch], int q)
{
    T r = x[0];
#pragma unroll
    for (int i = 1; i < kWalkBatch; i++) r = q == i ? x[i] : r;
    return r;
}

// Bits 2q of the batch's steps that enter an anchor.
template <bool FB>
__device__ __forceinline__ uint32_t anchor_steps(uint32_t idle, const float4 (&g)[kWalkBatch], const int32_t (&id)[kWalkBatch])
{
    uint32_t m = 0u;
#pragma unroll
    for (int q = 0; q < kWalkBatch; q++)
        m += (FB ? __float_as_uint(g[q].w) >> 31 : (uint32_t)~id[q] >> 31) << (2 * q);
    return m & ~idle;
}

// Whether any lane's batch may enter an anchor (an idle step's sample counts too: a false alarm
// costs the slower form, no record).
template <bool FB>
__device__ __forceinline__ bool any_anchor(const float4 (&g)[kWalkBatch], const int32_t (&id)[kWalkBatch])
{
    uint32_t m = 0u;
#pragma unroll
    for (int q = 0; q < kWalkBatch; q++) m |= FB ? __float_as_uint(g[q].w) : ~(uint32_t)id[q];
    return __any_sync(0xffffffffu, (int32_t)m < 0);
}

// What every operator pass keeps along a line.  A batch without an anchor only sums; in one
// with anchors the sums at its steps stay in registers and the lanes then record their
// contributions together, each lane its next one per round (unit weights: all at once), instead
// of step by step with the few lanes that enter an anchor at that step (three of 32 on average):
// a record waits for a row lookup and an atomic, and a round of them waits once.
template <int GRAD>
struct FillLine {
    const LineWalk &L;
    const Sink S;      // ids of the lane's copy
    float4 gl;         // sample of the last voxel
    float I = 0.0f;

    // I += the trapezoid increment of step q of a batch, or 0 on a lane that does not take it
    __device__ __forceinline__ void integrate(uint32_t c, int q, const float4 &gv, bool t)
    {
        const float x = step_increment<GRAD>(L, c, q, gv, gl);
        I = __fadd_rn(I, t ? x : 0.0f);
        if (GRAD != kGradEdge) gl = gv;
    }
};

// Plain method: anchors are the entries; every voxel of a line takes (p[entry] + I, 1).
template <int GRAD, int PASS, bool FB>
struct PlainFill : FillLine<GRAD> {
    uint32_t ecol;
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t, const float4 (&)[kWalkBatch], const int32_t (&)[kWalkBatch]) const
    {
        return true;
    }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                          const float4 (&g)[kWalkBatch], const int32_t (&id)[kWalkBatch])
    {
        if (!any_anchor<FB>(g, id)) {
#pragma unroll
            for (int q = 0; q < kWalkBatch; q++) this->integrate(c, q, g[q], taken<MASK>(idle, q));
            return;
        }
        float Is[kWalkBatch];
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            this->integrate(c, q, g[q], taken<MASK>(idle, q));
            Is[q] = this->I;
        }
        emit_units<PASS>(this->S, anchor_steps<FB>(idle, g, id), v, ecol, Is);
    }
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t, uint32_t, const uint32_t (&)[kWalkBatch],
                                            const float4 (&)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
    }
};

// SELF = false leaves the entry's own term out (the minimum-curl plain variant).
template <int GRAD, int PASS, bool SELF, bool FB>
__global__ void __launch_bounds__(kFillThreads, kFillBlocks)
k_anchor_plain(Grid g, Layout lay, WalkLines W, WalkField F, Sink S)
{
    LineWalk L;
    if (!L.init<GRAD != kGradEdge>(g, lay, W)) return;
    if (PASS == kMark) {
        if (L.on) S.flag[L.e] = 1;
        return;
    }
    const float4 *field = lane_field<GRAD>(F, lay, L);
    S.id += L.copy;
    PlainFill<GRAD, PASS, FB> f{{L, S, sample<GRAD>(field, L.v)}, start_col<PASS>(S, L.v)};
    if (SELF && L.on) emit_w<PASS, true>(S, __ldg(S.id + L.v), f.ecol, 1.0f, 0.0f);
    walk_steps<kWalkBatch, GRAD, !FB, GRAD != kGradEdge>(L, field, S.id, f);
}

// Weighted methods: the walks of k_sweep_weighted (K:1993-2135, RAW: K:2937-3085); anchors are
// the entries (the marking pass is the plain method's).  The entry itself receives nothing, or
// with RAW its own term.
template <int GRAD, bool RAW, bool FB>
struct WeightedFill : FillLine<GRAD> {
    uint32_t ecol;
    float csum, nseg;
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t, const float4 (&)[kWalkBatch], const int32_t (&)[kWalkBatch]) const
    {
        return true;
    }
    template <bool FLAGS>  // FLAGS: the curl may carry an anchor flag
    __device__ __forceinline__ void step(uint32_t c, int q, const float4 &gv, bool t)
    {
        const float cn = t ? curl_of<FLAGS>(gv) : 0.0f;
        csum += RAW ? cn : __fdiv_rn(cn, 1.0e4f);
        this->integrate(c, q, gv, t);
        nseg += t ? 1.0f : 0.0f;
    }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                          const float4 (&g)[kWalkBatch], const int32_t (&id)[kWalkBatch])
    {
        if (!any_anchor<FB>(g, id)) {
#pragma unroll
            for (int q = 0; q < kWalkBatch; q++) step<false>(c, q, g[q], taken<MASK>(idle, q));
            return;
        }
        uint32_t todo = anchor_steps<FB>(idle, g, id);
        float Is[kWalkBatch], ws[kWalkBatch];
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            step<FB>(c, q, g[q], taken<MASK>(idle, q));
            Is[q] = this->I;
            ws[q] = __fdividef(nseg, csum);
            if (!RAW) todo &= csum == 0.0f ? ~(1u << (2 * q)) : ~0u;
        }
        for (; todo; todo &= todo - 1u) {
            const int q = (__ffs(todo) - 1) >> 1;
            emit_w<kFill, false>(this->S, __ldg(this->S.id + pick(v, q)), ecol, pick(ws, q), pick(Is, q));
        }
    }
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t, uint32_t, const uint32_t (&)[kWalkBatch],
                                            const float4 (&)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
    }
};

template <int GRAD, bool RAW, bool FB>
__global__ void __launch_bounds__(kFillThreads, kFillBlocks)
k_anchor_weighted(Grid g, Layout lay, WalkLines W, WalkField F, Sink S)
{
    LineWalk L;
    if (!L.init<GRAD != kGradEdge>(g, lay, W)) return;
    const float4 *field = lane_field<GRAD>(F, lay, L);
    S.id += L.copy;
    WeightedFill<GRAD, RAW, FB> f{{L, S, sample<GRAD>(field, L.v)}, start_col<kFill>(S, L.v), 0.0f, 0.0f};
    if (RAW) {
        f.csum = curl_of<FB>(f.gl);
        f.nseg = 1.0f;
        if (L.on) emit_w<kFill, false>(S, __ldg(S.id + L.v), f.ecol, __frcp_rn(f.csum), 0.0f);
    }
    walk_steps<kWalkBatch, GRAD, !FB, GRAD != kGradEdge>(L, field, S.id, f);
}

// Selected method: the state machine of k_sweep_select (K:2280-2537); anchors are the
// segment starts.  The marking pass reads the curl alone, row-major.
template <int GRAD, int PASS, bool FB>
struct SelectFill : FillLine<GRAD> {
    const float *curl;
    float thr;
    SelectState st;
    uint32_t scol;
    float csum = 0.0f, nseg = 0.0f;

    // every step adds to a running segment
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t idle, const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch]) const
    {
        if (PASS == kMark) return false;
        if (!MASK && FB) {
            float lo, hi;
            curl_range<true>(g, lo, hi);
            return st.run() & (lo > 0.0f) & (hi < thr);
        }
        bool ok = st.run();
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            const float cn = curl_of<FB>(g[q]);
            ok = ok & (((cn < thr) & (cn != 0.0f)) | !taken<MASK>(idle, q));
        }
        return ok | (MASK & (idle == kAllIdle));
    }
    template <bool FLAGS>  // FLAGS: the curl may carry an anchor flag
    __device__ __forceinline__ void step(uint32_t c, int q, const float4 &gv, bool t)
    {
        csum = add_curl(csum, t ? curl_of<FLAGS>(gv) : 0.0f);  // the weights as in k_sweep_select
        this->integrate(c, q, gv, t);
        nseg += t ? 1.0f : 0.0f;
    }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                          const float4 (&g)[kWalkBatch], const int32_t (&id)[kWalkBatch])
    {
        if (!any_anchor<FB>(g, id)) {
#pragma unroll
            for (int q = 0; q < kWalkBatch; q++) step<false>(c, q, g[q], taken<MASK>(idle, q));
            return;
        }
        float Is[kWalkBatch], ws[kWalkBatch];
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            step<FB>(c, q, g[q], taken<MASK>(idle, q));
            Is[q] = this->I;
            ws[q] = __fdividef(nseg, csum);
        }
        for (uint32_t todo = anchor_steps<FB>(idle, g, id); todo; todo &= todo - 1u) {
            const int q = (__ffs(todo) - 1) >> 1;
            emit_w<PASS, false>(this->S, __ldg(this->S.id + pick(v, q)), scol, pick(ws, q), pick(Is, q));
        }
    }
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                            const float4 (&g)[kWalkBatch], const int32_t (&id)[kWalkBatch])
    {
        if (PASS == kMark) {
            float cn[kWalkBatch];
#pragma unroll
            for (int q = 0; q < kWalkBatch; q++) cn[q] = __ldg(curl + v[q]);
#pragma unroll
            for (int q = 0; q < kWalkBatch; q++) {
                bool add, start, clear;
                st.step(is_x(c, q), is_y(c, q), taken<MASK>(idle, q), cn[q], thr, add, start, clear);
                if (start) this->S.flag[v[q]] = 1;
            }
            return;
        }
        // the ids of the voxels that are anchors or may start a segment, loaded together
        int32_t rows[kWalkBatch];
        bool open = !st.run();
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            rows[q] = -1;
            if ((open | anchor_of<FB>(g[q], id[q])) & taken<MASK>(idle, q)) rows[q] = __ldg(this->S.id + v[q]);
            open = st.may_start_after(curl_of<FB>(g[q]), thr) | !taken<MASK>(idle, q);
        }
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            bool add, start, clear;
            st.step(is_x(c, q), is_y(c, q), taken<MASK>(idle, q), curl_of<FB>(g[q]), thr, add, start, clear);
            if (add) {
                step<FB>(c, q, g[q], true);
                if (rows[q] >= 0) emit_w<PASS, false>(this->S, rows[q], scol, __fdividef(nseg, csum), this->I);
            }
            if (GRAD != kGradEdge) this->gl = g[q];
            scol = start ? (uint32_t)rows[q] : scol;
            this->I = start ? 0.0f : this->I;
            nseg = clear ? 0.0f : nseg;
            csum = clear ? 0.0f : csum;
        }
    }
};

template <int GRAD, int PASS, bool FB>
__global__ void __launch_bounds__(kFillThreads, kFillBlocks)
k_anchor_select(Grid g, Layout lay, WalkLines W, WalkField F, const float *__restrict__ curl, Sink S)
{
    LineWalk L;
    if (!L.init<GRAD != kGradEdge>(g, lay, W)) return;
    const float4 *field = lane_field<GRAD>(F, lay, L);
    const float4 gl = sample<GRAD>(field, L.v);
    if (PASS == kFill) S.id += L.copy;
    SelectState st;
    st.enter(PASS == kFill ? curl_of<FB>(gl) : __ldg(curl + L.v), g.thr);
    if (PASS == kMark && st.run() && L.on) S.flag[L.v] = 1;
    SelectFill<GRAD, PASS, FB> f{{L, S, gl}, curl, g.thr, st, st.run() ? start_col<PASS>(S, L.v) : 0u};
    walk_steps<kWalkBatch, GRAD, PASS == kFill && !FB, GRAD != kGradEdge>(L, field, S.id, f);
}

// Selected method: a voxel can start a segment only if it is on the boundary (a line entry)
// or if the voxel before it on some line is "bad" (curl == 0 or curl >= thr): a start
// before the first good voxel follows a voxel that failed the start test, and a restart
// follows a voxel that paused or kept the pause (K:2300-2506); and every start voxel has
// curl != 0.  Flags that superset and counts it into *count.
__global__ void k_select_candidates(Grid g, const float *__restrict__ curl, uint8_t *flag,
                                    unsigned long long *count)
{
    const long long X = g.X, Y = g.Y, Z = g.Z, XY = g.XY;
    unsigned long long local = 0;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < g.V;
         v += (long long)gridDim.x * blockDim.x) {
        long long i = v % X, j = (v / X) % Y, k = v / XY;
        bool c = i == 0 || i == X - 1 || j == 0 || j == Y - 1 || k == 0 || k == Z - 1;
        if (!c) {
            const long long nb[6] = {v - 1, v + 1, v - X, v + X, v - XY, v + XY};
#pragma unroll
            for (int q = 0; q < 6; q++) {
                float cu = __ldg(curl + nb[q]);
                c |= (cu == 0.0f || cu >= g.thr);
            }
        }
        // every start rule needs curl != 0 at the start voxel (the masked interior drops out)
        c = c && __ldg(curl + v) != 0.0f;
        flag[v] = c ? 1 : 0;
        local += c ? 1 : 0;
    }
    for (int o = 16; o; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(count, local);
}

__global__ void k_flag_to_u32(long long V, const uint8_t *flag, uint32_t *out)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        out[v] = flag[v];
}

// id[v] = position among anchors or -1; vox[id] = v; the walks' copies of id (set to -1
// before) at the anchors.
__global__ void k_assign_ids(Grid g, Layout lay, const uint8_t *flag, const uint32_t *pos, int32_t *id, uint32_t *vox,
                             int32_t *wid)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < g.V;
         v += (long long)gridDim.x * blockDim.x) {
        if (!flag[v]) {
            id[v] = -1;
            continue;
        }
        const int32_t a = (int32_t)pos[v];
        id[v] = a;
        vox[a] = (uint32_t)v;
        if (!lay.wrap) continue;
        const VoxelAt q(g, v);
#pragma unroll
        for (int c = 0; c < 4; c++)
            wid[(size_t)c * (size_t)lay.stride + layout_index(lay, g.X, g.Y, c, q.i, q.j, q.k)] = a;
    }
}

// Link slots of every row: the lines through its voxel (each contributes at most once), in whole
// loads of `per` links; *total: the slots before rounding.
__global__ void k_row_capacity(long long n, const uint32_t *vox, const uint32_t *lines_through, unsigned per, int panels,
                               unsigned long long *out, unsigned long long *total)
{
    unsigned long long t = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t c = lines_through[vox[i]];
        for (int p = 0; p < panels; p++) out[i * panels + p] = (c + per - 1) / per * per;
        t += c;
    }
    for (int o = 16; o; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd(total, t);
}

// Row sums of the anchor iteration.  A row gathers about as many terms as lines cross its voxel
// (~1000 at 642 directions); plain FP32 sums of that many terms leave a rounding floor near 1e-6 in
// the iteration's relative change, above the tolerances the solver is asked for.  A lane's links are
// summed with their errors (sums.cuh), the lane sums added as unevaluated pairs (hi, lo), and the
// row's update is in FP64.
template <int LANES>
__device__ __forceinline__ void warp_sum_pair(float &hi, float &lo)
{
#pragma unroll
    for (int o = LANES / 2; o; o >>= 1)
        add_pair(hi, lo, __shfl_xor_sync(0xffffffffu, hi, o), __shfl_xor_sync(0xffffffffu, lo, o));
}

// The exact sum of fixed-point lane sums (integer additions: order-independent).
template <int LANES>
__device__ __forceinline__ long long warp_sum_fixed(long long t)
{
#pragma unroll
    for (int o = LANES / 2; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

__device__ __forceinline__ double warp_sum_double(double x)
{
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// The convergence measure of an iteration (tolerance-driven solves): the gauged squared change
// and norm over all anchors, sum (d - sd)^2 and sum (p - sp)^2 with d = pn - pc.  The shifts
// (the reference entry's change and value, the means, or 0) are not known before every row is
// done, so the sums are taken about the last iteration's shifts (`about`, 0 in the first) and
// moved to this one's at the end, where little is left to cancel.
struct ChangeOut {
    double *red2;        // {change, norm} (null: no measure)
    double *about;       // 2: the shifts of the last iteration
    unsigned *arrived;   // blocks done (wraps to 0)
    double *part;        // 4 per block
    int gauge;
    long long ref;
    double tol;          // with stop: the chunk's test, see iterate_chunk
    int step;
    int *stop;
    double *rel_out;
};

// One anchor iteration, p_next = (b + seed p_init + M p_cur) / c; KIND: the links; FIX: the
// bit-reproducible mode's exact fixed-point sums, whatever the entries' order; SMEM: p_cur in
// shared memory.  The FP64 work of a row -- its update, one division among it -- is done for a
// block's rows together, a thread each, since this GPU's FP64 units take 16 cycles per warp
// instruction and SM: with a row per warp and FP64 lane sums they alone took 0.1 ms of the
// 0.165 of an iteration at 128^3 / 642 directions (97 K rows).  96^3 / 642 directions (54 K rows,
// 34 M links): 80 us, 48 with the rows' FP64 work together, 35 with 16-bit links, 28 with
// p_cur in shared memory; six CTAs of 256 threads per SM at 40 registers (five: 10 to 25 % more).
template <int KIND, bool FIX, bool SMEM>
__global__ void __launch_bounds__(SMEM ? 1024 : 256, SMEM ? 1 : 6) k_anchor_iterate(
    long long n, int rows, uint32_t split, const unsigned long long *__restrict__ rowptr,
    const uint32_t *__restrict__ rowlen, const void *__restrict__ links, const float2 *__restrict__ bc,
    const uint32_t *__restrict__ vox, const float *__restrict__ p_init, int seed, const float *__restrict__ pc, float *pn,
    const int *stop, const double *__restrict__ fix, ChangeOut C)
{
    extern __shared__ float4 sh_vector[];
    if (stop && *stop) return;  // a graph-captured chunk that has met its tolerance
    constexpr int kWarps = (SMEM ? 1024 : 256) / 32, kLanes = lanes_per_row(KIND), kRows = 32 / kLanes;
    __shared__ double row_sum[kWarps * iter_rows_max(SMEM)];  // (hi, lo) pairs, or the exact integers
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long base = (long long)blockIdx.x * kWarps * rows;  // the block's first row
    const long long row0 = base + (long long)warp * rows;
    const FixScale sr = FIX ? fix_scale(fix[kFixRow]) : FixScale{};
    const int panels = KIND == kLink16 && split ? 2 : 1;
    for (int p = 0; p < panels; p++) {
        if (SMEM && p) __syncthreads();  // the first panel has been read
        const long long c0 = p ? (long long)split : 0;
        const float *x = gather_vector<SMEM>(pc + c0, panels == 1 ? n : min((long long)split, n - c0), reinterpret_cast<float *>(sh_vector));
        unsigned long long ptr = 0ull;
        uint32_t len = 0u;
        if (lane < rows && row0 + lane < n) {
            ptr = rowptr[(row0 + lane) * panels + p];
            len = rowlen[(row0 + lane) * panels + p];
        }
        for (int r = 0; r < rows; r += kRows) {
            if (row0 + r >= n) break;  // whole warps
            const int mine = r + lane / kLanes;  // (lanes past the last row have length 0)
            const unsigned long long j0 = __shfl_sync(0xffffffffu, ptr, mine & 31);
            const uint32_t m = __shfl_sync(0xffffffffu, len, mine & 31);
            float s = 0.0f, comp = 0.0f;
            long long t = 0;
            row_links<KIND>(links, j0, mine < rows ? m : 0u, lane % kLanes, [&](uint32_t c, float w, int) {
                const float y = SMEM ? x[c] : __ldg(x + c);
                if (FIX) t += (long long)fix_term(KIND == kLinkPair ? w * y : y, sr);
                else if (KIND == kLinkPair) kahan_add_product(s, comp, w, y);
                else two_sum_add(s, comp, y);
            });
            __syncwarp();
            if (FIX) {
                t = warp_sum_fixed<kLanes>(t);
                if (p && mine < rows) t += __double_as_longlong(row_sum[warp * rows + mine]);
            } else {
                float h = s, l = KIND == kLinkPair ? -comp : comp;
                warp_sum_pair<kLanes>(h, l);
                if (p && mine < rows) {  // the first panel's pair
                    const unsigned long long f = (unsigned long long)__double_as_longlong(row_sum[warp * rows + mine]);
                    add_pair(h, l, __uint_as_float((uint32_t)(f >> 32)), __uint_as_float((uint32_t)f));
                }
                t = (long long)(((unsigned long long)__float_as_uint(h) << 32) | __float_as_uint(l));
            }
            if (lane % kLanes == 0 && mine < rows) row_sum[warp * rows + mine] = __longlong_as_double(t);
        }
    }
    __syncthreads();
    // the block's rows, a thread each
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const double ad = C.about ? C.about[0] : 0.0, ap = C.about ? C.about[1] : 0.0;
    for (int i = threadIdx.x; i < kWarps * rows; i += 32 * kWarps) {
        const long long mine = base + i;
        if (mine >= n) break;
        const unsigned long long t = (unsigned long long)__double_as_longlong(row_sum[i]);
        const double sum = FIX ? (double)(long long)t / fix[kFixRow]
                               : (double)__uint_as_float((uint32_t)(t >> 32)) + (double)__uint_as_float((uint32_t)t);
        const float2 q = bc[mine];
        const float old = pc[mine];
        double numer = (double)q.x + sum;
        if (seed && p_init) numer += (double)p_init[vox[mine]];
        const float now = q.y > 0.0f ? (float)(numer / (double)q.y) : old;
        pn[mine] = now;
        if (C.red2) {
            const double d = (double)now - (double)old - ad, p = (double)now - ap;
            v[0] += d;
            v[1] += d * d;
            v[2] += p;
            v[3] += p * p;
        }
    }
    if (!C.red2) return;
    __shared__ double sh[4][kWarps];
    __shared__ bool last;
    if (warp * 32 < kWarps * rows) {  // whole warps: the others have no rows
        for (int i = 0; i < 4; i++) v[i] = warp_sum_double(v[i]);
    }
    if (lane == 0)
        for (int i = 0; i < 4; i++) sh[i][warp] = v[i];
    __syncthreads();
    if (threadIdx.x < 4) {
        double t = 0.0;
        for (int w = 0; w < kWarps; w++) t += sh[threadIdx.x][w];
        C.part[4ull * blockIdx.x + threadIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(C.arrived, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;  // the last block adds the blocks' sums in their order
    __threadfence();
    const int i = threadIdx.x & 3;
    double t = 0.0;
#pragma unroll 4
    for (unsigned b = threadIdx.x >> 2; b < gridDim.x; b += 8 * kWarps) t += __ldcg(C.part + 4ull * b + i);
    for (int o = 16; o >= 4; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);  // lanes 0..3: this warp's four sums
    if (lane < 4) sh[lane][warp] = t;
    __syncthreads();
    if (warp != 0) return;
    t = 0.0;  // lanes 0..3 (and those that repeat them): the block's four
    for (int w = 0; w < kWarps; w++) t += sh[i][w];
    double S[4];
    for (int k = 0; k < 4; k++) S[k] = __shfl_sync(0xffffffffu, t, k);
    if (lane != 0) return;
    const double N = (double)n;
    double ed = -ad, ep = -ap;  // the shifts about the old ones (none: 0)
    if (C.gauge == OMNI3D_GAUGE_POINT && C.ref >= 0) {
        const volatile float *now = pn;
        const double at = (double)now[C.ref];
        ep = at - ap;
        ed = at - (double)pc[C.ref] - ad;
    } else if (C.gauge == OMNI3D_GAUGE_MEAN) {
        ed = S[0] / N;
        ep = S[2] / N;
    }
    // sum (x - shift)^2 from sum x^2 and sum x: infinite and NaN sums stay so
    auto moved = [&](double square, double linear, double shift) {
        if (shift == 0.0 || (isfinite(shift) && !isfinite(square))) return square;
        const double r = square - 2.0 * shift * linear + N * shift * shift;
        return r < 0.0 ? 0.0 : r;
    };
    const double change = moved(S[1], S[0], ed), norm = moved(S[3], S[2], ep);
    C.red2[0] = change;
    C.red2[1] = norm;
    if (C.about) {
        C.about[0] = ad + ed;
        C.about[1] = ap + ep;
    }
    if (C.stop) {  // the chunk's convergence test: the host loop's formula
        const double rel = norm > 0 ? sqrt(change / norm) : 0.0;
        C.rel_out[C.step] = rel;
        if (rel < C.tol) *C.stop = C.step + 1;
    }
}

constexpr int kRedBlocks = 256, kRedThreads = 256;

__device__ __forceinline__ double block_sum(double x, double *sh)
{
    for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += sh[i];
    __syncthreads();
    return s;
}

// Sums of (d, p, 1) over the selected entries (for the mean gauge).
__global__ void k_sum_dp(long long n, const float *pc, const float *pn, const uint8_t *mask, double *part)
{
    __shared__ double sh[32];
    double sd = 0.0, sp = 0.0, cn = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (mask && !mask[i]) continue;
        sd += (double)pn[i] - (double)pc[i];
        sp += (double)pn[i];
        cn += 1.0;
    }
    double a = block_sum(sd, sh), bb = block_sum(sp, sh), cc = block_sum(cn, sh);
    if (threadIdx.x == 0) {
        part[3 * blockIdx.x] = a;
        part[3 * blockIdx.x + 1] = bb;
        part[3 * blockIdx.x + 2] = cc;
    }
}

__global__ void k_finish(const double *part, int nblk, int width, double *out)
{
    if ((int)threadIdx.x < width) {
        double s = 0.0;
        for (int i = 0; i < nblk; i++) s += part[width * i + threadIdx.x];
        out[threadIdx.x] = s;
    }
}

// Gauged squared change and squared norm over the selected entries: sum (d - sd)^2 and
// sum (p - sp)^2.  The shifts are the reference entry's change and value (point gauge),
// the means (mean gauge: sums[0..2] = sum d, sum p, count) or 0.
__global__ void k_change(long long n, const float *pc, const float *pn, const uint8_t *mask, int gauge,
                         long long ref, const double *sums, double *part)
{
    __shared__ double sh[32];
    double sd = 0.0, sp = 0.0;
    if (gauge == OMNI3D_GAUGE_POINT && ref >= 0) {
        sp = (double)pn[ref];
        sd = sp - (double)pc[ref];
    } else if (gauge == OMNI3D_GAUGE_MEAN && sums[2] > 0) {
        sd = sums[0] / sums[2];
        sp = sums[1] / sums[2];
    }
    double a = 0.0, bb = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        if (mask && !mask[i]) continue;
        double d = (double)pn[i] - (double)pc[i] - sd;
        double q = (double)pn[i] - sp;
        a += d * d;
        bb += q * q;
    }
    double ta = block_sum(a, sh), tb = block_sum(bb, sh);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = ta; part[2 * blockIdx.x + 1] = tb; }
}

// The anchor values into the walks' copies of the pressure.
__global__ void k_scatter(Grid g, Layout lay, long long n, const uint32_t *vox, const float *pa, float *vol)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t v = vox[i];
        const float x = pa[i];
        if (!lay.wrap) {
            vol[v] = x;
            continue;
        }
        const VoxelAt q(g, v);
#pragma unroll
        for (int c = 0; c < 4; c++)
            vol[(size_t)c * (size_t)lay.stride + layout_index(lay, g.X, g.Y, c, q.i, q.j, q.k)] = x;
    }
}

__global__ void k_gather(long long n, const uint32_t *vox, const float *vol, float *pa)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        pa[i] = vol[vox[i]];
}

unsigned grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    if (b > 152LL * 64) b = 152LL * 64;
    if (b < 1) b = 1;
    return (unsigned)b;
}

// b = 0 on every row, c kept (the cached plain operator's refresh).
__global__ void k_clear_b(long long n, float2 *bc)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        bc[i].x = 0.0f;
}

// After the filling pass: each row's length from its next free slot.
__global__ void k_row_lengths(long long n, const unsigned long long *__restrict__ rowptr,
                              const unsigned long long *__restrict__ next, uint32_t *rowlen)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        rowlen[i] = (uint32_t)(next[i] - rowptr[i]);
}

// Set (set = 1) or clear the anchor flag, the sign bit of the curl, in the n anchors' field
// records that the walks read.
__global__ void k_field_flags(Grid g, Layout lay, long long n, const uint32_t *__restrict__ vox, float4 *field, int set)
{
    const int per = lay.wrap ? 8 : 1;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n * per; i += (long long)gridDim.x * blockDim.x) {
        const uint32_t v = vox[i / per];
        size_t at = v;
        if (lay.wrap) {
            const int oct = (int)(i % per);
            const VoxelAt q(g, v);
            at = (size_t)oct * (size_t)lay.stride + layout_index(lay, g.X, g.Y, oct >> 1, q.i, q.j, q.k);
        }
        uint32_t *u = reinterpret_cast<uint32_t *>(&field[at].w);
        *u = set ? (*u | 0x80000000u) : (*u & 0x7fffffffu);
    }
}

// *any = 1 when some curl value has its sign bit set (negative, or -0).
__global__ void k_sign_any(long long V, const float *__restrict__ curl, uint32_t *any)
{
    bool neg = false;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        neg |= (__float_as_uint(curl[v]) >> 31) != 0u;
    if (__any_sync(0xffffffffu, neg) && (threadIdx.x & 31) == 0) *any = 1u;
}

// Launch the pass for the method's accumulation kind.  FB: the anchors are flagged in the
// field.
template <int GRAD, int PASS, bool FB>
void launch_pass(int acc, const Geometry &geo, const Field &f, const Sink &S, cudaStream_t st)
{
    const unsigned blocks = group_blocks(geo, kFillThreads);
    const Grid &g = geo.grid;
    const Layout lay = PASS == kMark ? row_major_layout(g) : f.lay;
    const WalkLines W{geo.d_groups, geo.n_groups, geo.d_lines, geo.d_desc};
    const WalkField F{f.f32, f.edge};
    OM_COUNT_LAUNCH();
    if constexpr (PASS == kFill) {
        if (acc == kAccWeightedRawCurl) {
            k_anchor_weighted<GRAD, true, FB><<<blocks, kFillThreads, 0, st>>>(g, lay, W, F, S);
            return;
        }
        if (acc == kAccWeighted) {
            k_anchor_weighted<GRAD, false, FB><<<blocks, kFillThreads, 0, st>>>(g, lay, W, F, S);
            return;
        }
        if (acc == kAccPlainNoEntry) {
            k_anchor_plain<GRAD, kFill, false, FB><<<blocks, kFillThreads, 0, st>>>(g, lay, W, F, S);
            return;
        }
    }
    if constexpr (PASS != kRhs) {
        if (acc == kAccSelect) {
            k_anchor_select<GRAD, PASS, FB><<<blocks, kFillThreads, 0, st>>>(g, lay, W, F, f.curl, S);
            return;
        }
    }
    // plain method, and the marking pass of every method whose anchors are the entries
    k_anchor_plain<GRAD, PASS, true, FB><<<blocks, kFillThreads, 0, st>>>(g, lay, W, F, S);
}

// fb: the anchors' field entries carry the anchor flag (k_field_flags): possible when no
// curl value has its sign bit set.
template <int PASS>
cudaError_t run_pass(const Geometry &geo, const Field &f, int method, bool fb, const Sink &S, cudaStream_t st)
{
    if (geo.n_lines == 0) return cudaSuccess;
    // every pointer the pass dereferences must be set: refuse to launch otherwise
    const bool need_field = PASS == kFill || PASS == kRhs;
    bool ok = geo.d_lines && geo.d_groups && geo.d_desc;
    if (PASS == kMark) ok = ok && S.flag;
    else ok = ok && S.id && S.bc;
    const bool unit_links = method_accum(method) == kAccPlain || method_accum(method) == kAccPlainNoEntry;
    if (PASS == kFill) ok = ok && S.next && S.links && (unit_links == (S.kind != kLinkPair));
    if (need_field) ok = ok && (f.lay.wrap ? f.edge != nullptr : f.f32 != nullptr);
    const int acc = method_accum(method);
    const bool weighted = acc == kAccWeighted || acc == kAccWeightedRawCurl;
    if (acc == kAccSelect || (weighted && PASS == kFill)) ok = ok && f.curl;
    if (PASS == kRhs && acc != kAccPlain) ok = false;  // only the plain operator is cached
    if (!ok) return cudaErrorInvalidValue;
    if constexpr (PASS == kMark) launch_pass<kNoGrad, kMark, false>(acc, geo, f, S, st);  // reads no packed field
    else if (f.lay.wrap) fb ? launch_pass<kGradEdge, PASS, true>(acc, geo, f, S, st)
                            : launch_pass<kGradEdge, PASS, false>(acc, geo, f, S, st);
    else fb ? launch_pass<kGradVoxel, PASS, true>(acc, geo, f, S, st) : launch_pass<kGradVoxel, PASS, false>(acc, geo, f, S, st);
    return cudaGetLastError();
}

}  // namespace

#define AN_TRY(x)                                                              \
    do {                                                                       \
        cudaError_t e_ = (x);                                                  \
        if (e_ != cudaSuccess) {                                               \
            if (err) *err = std::string(#x) + ": " + cudaGetErrorString(e_);   \
            return e_;                                                         \
        }                                                                      \
    } while (0)

size_t change_scratch_doubles();

// Grow-only device buffer: reallocates only when `bytes` exceeds the recorded capacity.
template <typename T>
cudaError_t grow(T *&p, size_t &cap, size_t bytes)
{
    if (bytes == 0) bytes = 1;
    if (bytes <= cap && p) return cudaSuccess;
    cudaFree(p);
    p = nullptr;
    cap = 0;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaSuccess) cap = bytes;
    return e;
}

void anchor_free(Anchor *A)
{
    cudaFree(A->flag); cudaFree(A->wid); cudaFree(A->id); cudaFree(A->vox); cudaFree(A->rowptr);
    cudaFree(A->links); cudaFree(A->bc); cudaFree(A->pa); cudaFree(A->pb);
    cudaFree(A->red); cudaFree(A->rowlen); cudaFree(A->u); cudaFree(A->pos); cudaFree(A->tmp); cudaFree(A->cnt64); cudaFree(A->tmp64);
    cudaFree(A->neg); cudaFree(A->next);
    *A = Anchor();
}

cudaError_t anchor_build(Geometry &geo, const Field &f, int method, long long ref_voxel,
                         long long max_nnz, Anchor *A, cudaStream_t st, std::string *err, Fixed *fx, uint32_t *scratch)
{
    const long long V = geo.grid.V;
    size_t *cap = A->cap;
    const Layout &lay = f.lay;
    const int acc = method_accum(method);
    const bool unit_links = acc == kAccPlain || acc == kAccPlainNoEntry;
    Sink S{};
    // the field carries curl in .w: its sign bit can flag the anchors unless a curl value
    // already has it set
    const bool check_sign = f.curl != nullptr;
    AN_TRY(grow(A->neg, cap[18], sizeof(uint32_t)));
    AN_TRY(cudaMemsetAsync(A->neg, 0, sizeof(uint32_t), st));
    if (check_sign) {
        k_sign_any<<<grid_for(V), 256, 0, st>>>(V, f.curl, A->neg);
        OM_COUNT_LAUNCH();
        AN_TRY(cudaGetLastError());
    }
    uint32_t n = (uint32_t)A->n, neg = 0;
    // The anchors and their rows' capacities.  Those of the methods whose anchors are the lines'
    // entries follow from the geometry's walks alone: a later field finds them in place (40^3 /
    // 642 directions, weighted: 0.95 -> 0.84 ms a solve).
    if (A->placed == geo.walk_generation + 1 && acc != kAccSelect) {
        AN_TRY(cudaMemcpyAsync(&neg, A->neg, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        AN_TRY(cudaStreamSynchronize(st));
    } else {
        A->placed = 0;
        AN_TRY(grow(A->flag, cap[0], (size_t)V));
        if (lay.wrap) {
            AN_TRY(grow(A->wid, cap[1], sizeof(int32_t) * (size_t)lay.copies * (size_t)V));
            AN_TRY(cudaMemsetAsync(A->wid, 0xff, sizeof(int32_t) * (size_t)lay.copies * (size_t)V, st));
        }
        AN_TRY(grow(A->id, cap[2], sizeof(int32_t) * (size_t)V));
        AN_TRY(grow(A->u, cap[3], sizeof(uint32_t) * (size_t)V));
        AN_TRY(grow(A->pos, cap[4], sizeof(uint32_t) * (size_t)(V + 1)));
        AN_TRY(grow(A->tmp, cap[5], sizeof(uint32_t) * scan_tmp_elems(V)));
        S.flag = A->flag;
        bool marked = false;
        if (acc == kAccSelect) {
            // cheap superset of the segment starts; used when it stays small
            AN_TRY(grow(A->cnt64, cap[8], sizeof(unsigned long long) * 1));
            unsigned long long *dcount = A->cnt64;
            AN_TRY(cudaMemsetAsync(dcount, 0, sizeof(unsigned long long), st));
            k_select_candidates<<<grid_for(V), 256, 0, st>>>(geo.grid, f.curl, A->flag, dcount);
            OM_COUNT_LAUNCH();
            AN_TRY(cudaGetLastError());
            unsigned long long nc = 0;
            AN_TRY(cudaMemcpyAsync(&nc, dcount, sizeof(nc), cudaMemcpyDeviceToHost, st));
            AN_TRY(cudaStreamSynchronize(st));
            marked = (long long)nc <= V / 16;
        }
        if (!marked) {
            AN_TRY(cudaMemsetAsync(A->flag, 0, (size_t)V, st));
            AN_TRY(run_pass<kMark>(geo, f, method, false, S, st));
        }
        if (ref_voxel >= 0 && ref_voxel < V) AN_TRY(cudaMemsetAsync(A->flag + ref_voxel, 1, 1, st));
        k_flag_to_u32<<<grid_for(V), 256, 0, st>>>(V, A->flag, A->u);
        OM_COUNT_LAUNCH();
        AN_TRY(cudaGetLastError());
        AN_TRY(exclusive_scan_u32(A->u, A->pos, V, A->tmp, st));
        AN_TRY(cudaMemcpyAsync(&n, A->pos + V, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        AN_TRY(cudaMemcpyAsync(&neg, A->neg, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        AN_TRY(cudaStreamSynchronize(st));
        A->n = n;
        AN_TRY(grow(A->vox, cap[7], sizeof(uint32_t) * (size_t)n));
        k_assign_ids<<<grid_for(V), 256, 0, st>>>(geo.grid, lay, A->flag, A->pos, A->id, A->vox, A->wid);
        OM_COUNT_LAUNCH();
        AN_TRY(cudaGetLastError());

        // rows: a voxel receives at most one contribution per line through it, so the
        // geometry-only line counts size the rows and no counting pass is needed
        AN_TRY(ensure_lines_through(&geo, f.lay, scratch, st));
        A->kind = link_kind(n, unit_links);
        A->split = link_split(n, unit_links);
        const long long rows = (long long)n * A->panels();
        AN_TRY(grow(A->cnt64, cap[8], sizeof(unsigned long long) * (size_t)(rows + 1)));
        AN_TRY(grow(A->tmp64, cap[9], sizeof(unsigned long long) * scan_tmp_elems(rows)));
        AN_TRY(grow(A->rowptr, cap[10], sizeof(unsigned long long) * (size_t)(rows + 1)));
        AN_TRY(cudaMemsetAsync(A->cnt64 + rows, 0, sizeof(unsigned long long), st));
        k_row_capacity<<<grid_for(n), 256, 0, st>>>(n, A->vox, geo.d_lines_through, (unsigned)links_per_vector(A->kind),
                                                    A->panels(), A->cnt64, A->cnt64 + rows);
        OM_COUNT_LAUNCH();
        AN_TRY(cudaGetLastError());
        AN_TRY(exclusive_scan_u64(A->cnt64, A->rowptr, rows, A->tmp64, st));
        unsigned long long nnz = 0;
        AN_TRY(cudaMemcpyAsync(&A->slots, A->rowptr + rows, sizeof(A->slots), cudaMemcpyDeviceToHost, st));
        AN_TRY(cudaMemcpyAsync(&nnz, A->cnt64 + rows, sizeof(nnz), cudaMemcpyDeviceToHost, st));
        AN_TRY(cudaStreamSynchronize(st));
        A->nnz = (long long)nnz;
        if (acc != kAccSelect) A->placed = geo.walk_generation + 1;
    }
    const bool fb = neg == 0u;
    const long long subrows = (long long)n * A->panels();
    const size_t link_bytes = link_size(A->kind);
    long long limit = max_nnz;
    if (max_nnz == 0) {  // links that fit in place always pass (asking takes 23 us)
        size_t fr = 0, tot = 0;
        if (link_bytes * (size_t)A->slots <= cap[11]) limit = -1;
        else if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) limit = anchor_link_limit(fr);
    }
    if (limit >= 0 && A->nnz > limit) {
        if (err) *err = "anchor operator larger than its limit";
        return cudaErrorNotSupported;
    }

    AN_TRY(grow(A->links, cap[11], link_bytes * (size_t)A->slots));
    AN_TRY(grow(A->bc, cap[13], sizeof(float2) * (size_t)n));
    A->uneven = geo.walk_rule == 3;
    const long long n1 = std::max<long long>(n, 1);
    AN_TRY(grow(A->red, cap[6], sizeof(double) * (4 + 4 * (size_t)std::max(iter_shape(n1, true, A->kind, A->split, A->uneven).blocks,
                                                                           iter_shape(n1, false, A->kind, A->split, A->uneven).blocks))));
    AN_TRY(grow(A->pa, cap[15], sizeof(float) * (size_t)n));
    AN_TRY(grow(A->pb, cap[16], sizeof(float) * (size_t)n));
    AN_TRY(grow(A->rowlen, cap[17], sizeof(uint32_t) * (size_t)subrows));
    AN_TRY(grow(A->next, cap[19], sizeof(unsigned long long) * (size_t)std::max<long long>(subrows, 1)));
    if (n) AN_TRY(cudaMemcpyAsync(A->next, A->rowptr, sizeof(unsigned long long) * (size_t)subrows, cudaMemcpyDeviceToDevice, st));
    AN_TRY(cudaMemsetAsync(A->bc, 0, sizeof(float2) * (size_t)std::max<long long>(n, 1), st));
    S.id = lay.wrap ? A->wid : A->id;
    S.next = A->next;
    S.links = A->links;
    S.kind = A->kind;
    S.split = A->split;
    S.bc = A->bc;
    if (fx) {  // bit-reproducible: the rows' (b, c) in fixed point (scales set by the caller)
        AN_TRY(grow(fx->bc64, fx->cap_bc64, sizeof(long long) * 2 * (size_t)std::max<long long>(n, 1)));
        AN_TRY(cudaMemsetAsync(fx->bc64, 0, sizeof(long long) * 2 * (size_t)std::max<long long>(n, 1), st));
        S.bc64 = fx->bc64;
        S.fix = fx->scale;
    }
    if (fb && n) {
        k_field_flags<<<grid_for(n * 8), 256, 0, st>>>(geo.grid, f.lay, n, A->vox, f.lay.wrap ? f.edge : f.f32, 1);
        OM_COUNT_LAUNCH();
        AN_TRY(cudaGetLastError());
    }
    AN_TRY(run_pass<kFill>(geo, f, method, fb, S, st));
    if (fx) AN_TRY(fix_rows_to_float(n, *fx, A->bc, false, st));
    if (n) {
        k_row_lengths<<<grid_for(subrows), 256, 0, st>>>(subrows, A->rowptr, A->next, A->rowlen);
        OM_COUNT_LAUNCH();
        if (fb) {  // the sweeps read the field unflagged
            k_field_flags<<<grid_for(n * 8), 256, 0, st>>>(geo.grid, f.lay, n, A->vox, f.lay.wrap ? f.edge : f.f32, 0);
            OM_COUNT_LAUNCH();
        }
        AN_TRY(cudaGetLastError());
    }
    return cudaGetLastError();
}

size_t change_scratch_doubles() { return 8 + 3 * kRedBlocks; }

cudaError_t change_sums(long long n, const float *pc, const float *pn, int gauge, long long ref, double *scratch,
                        double *out2, cudaStream_t st, const uint8_t *mask)
{
    double *part = scratch + 8;
    if (gauge == OMNI3D_GAUGE_MEAN) {
        k_sum_dp<<<kRedBlocks, kRedThreads, 0, st>>>(n, pc, pn, mask, part);
        OM_COUNT_LAUNCH();
        k_finish<<<1, 32, 0, st>>>(part, kRedBlocks, 3, scratch + 4);
        OM_COUNT_LAUNCH();
    }
    k_change<<<kRedBlocks, kRedThreads, 0, st>>>(n, pc, pn, mask, gauge, ref, scratch + 4, part);
    OM_COUNT_LAUNCH();
    k_finish<<<1, 32, 0, st>>>(part, kRedBlocks, 2, out2);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

cudaError_t anchor_mark(const Geometry &geo, const Field &f, int method, long long ref_voxel,
                        uint8_t *flag, unsigned long long *count1, cudaStream_t st)
{
    const long long V = geo.grid.V;
    cudaError_t e;
    bool marked = false;
    if (method_accum(method) == kAccSelect) {
        e = cudaMemsetAsync(count1, 0, sizeof(unsigned long long), st);
        if (e != cudaSuccess) return e;
        k_select_candidates<<<grid_for(V), 256, 0, st>>>(geo.grid, f.curl, flag, count1);
        OM_COUNT_LAUNCH();
        unsigned long long nc = 0;
        e = cudaMemcpyAsync(&nc, count1, sizeof(nc), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        marked = (long long)nc <= V / 16;
    }
    if (!marked) {
        e = cudaMemsetAsync(flag, 0, (size_t)V, st);
        if (e != cudaSuccess) return e;
        Sink S{};
        S.flag = flag;
        e = run_pass<kMark>(geo, f, method, false, S, st);
        if (e != cudaSuccess) return e;
    }
    if (ref_voxel >= 0 && ref_voxel < geo.grid.V) e = cudaMemsetAsync(flag + ref_voxel, 1, 1, st);
    return e;
}

cudaError_t anchor_step(const Anchor &A, const float *p_init, bool seed, bool first, int gauge, long long ref_anchor,
                        const float *p_cur, float *p_next, double *red2, cudaStream_t st, const ChunkTest *test,
                        const Fixed *fx, bool alone)
{
    if (A.n == 0) return cudaSuccess;
    const int *stop = test ? test->stop : nullptr;
    const double *fix = nullptr;
    if (fx) {  // bit-reproducible: the row sums' scale from this iterate's largest value
        cudaError_t e = fix_row_scale(A.n, p_cur, *fx, st, stop);
        if (e != cudaSuccess) return e;
        fix = fx->scale;
    }
    ChangeOut C{};
    if (red2) {
        C.red2 = red2;
        C.about = A.red;
        C.arrived = reinterpret_cast<unsigned *>(A.red + 2);
        C.part = A.red + 4;
        C.gauge = gauge;
        C.ref = ref_anchor;
        if (first) {  // nothing to take the sums about
            cudaError_t e = cudaMemsetAsync(A.red, 0, sizeof(double) * 4, st);
            if (e != cudaSuccess) return e;
        }
        if (test) {
            C.tol = test->tol;
            C.step = test->step;
            C.stop = test->stop;
            C.rel_out = test->rel_out;
        }
    }
    const IterShape I = iter_shape(A.n, alone, A.kind, A.split, A.uneven);
    auto launch = [&](auto kernel) {
        if (I.bytes > 48 * 1024) {  // (a host-side attribute of the kernel: cheap, and safe while capturing)
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kIterSmemMax);
            if (e != cudaSuccess) return e;
        }
        kernel<<<I.blocks, I.threads, I.bytes, st>>>(A.n, I.rows, A.split, A.rowptr, A.rowlen, A.links, A.bc, A.vox, p_init, seed ? 1 : 0,
                                                     p_cur, p_next, stop, fix, C);
        OM_COUNT_LAUNCH();
        return cudaGetLastError();
    };
#define OM_LAUNCH_ITERATE(KIND, SMEM) (fix ? launch(k_anchor_iterate<KIND, true, SMEM>) : launch(k_anchor_iterate<KIND, false, SMEM>))
    switch (A.kind) {
    case kLink16: return I.smem ? OM_LAUNCH_ITERATE(kLink16, true) : OM_LAUNCH_ITERATE(kLink16, false);
    case kLink32: return OM_LAUNCH_ITERATE(kLink32, false);
    default: return OM_LAUNCH_ITERATE(kLinkPair, false);
    }
#undef OM_LAUNCH_ITERATE
}

cudaError_t anchor_refresh_rhs(const Geometry &geo, const Field &f, Anchor *A, cudaStream_t st,
                               const Fixed *fx)
{
    if (A->n == 0) return cudaSuccess;
    if (fx && (!fx->bc64 || fx->cap_bc64 < sizeof(long long) * 2 * (size_t)A->n)) return cudaErrorInvalidValue;
    k_clear_b<<<grid_for(A->n), 256, 0, st>>>(A->n, A->bc);
    OM_COUNT_LAUNCH();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    Sink S{};
    S.id = f.lay.wrap ? A->wid : A->id;
    S.bc = A->bc;
    if (fx) {
        if ((e = cudaMemsetAsync(fx->bc64, 0, sizeof(long long) * 2 * (size_t)A->n, st)) != cudaSuccess) return e;
        S.bc64 = fx->bc64;
        S.fix = fx->scale;
    }
    // the plain method's field carries no curl (.w = +0), so the anchors can be flagged in it
    const bool fb = f.curl == nullptr;
    if (fb) {
        k_field_flags<<<grid_for(A->n * 8), 256, 0, st>>>(geo.grid, f.lay, A->n, A->vox, f.lay.wrap ? f.edge : f.f32, 1);
        OM_COUNT_LAUNCH();
    }
    e = run_pass<kRhs>(geo, f, OMNI3D_METHOD_PLAIN, fb, S, st);
    if (e == cudaSuccess && fx) e = fix_rows_to_float(A->n, *fx, A->bc, true, st);
    if (e != cudaSuccess || !fb) return e;
    k_field_flags<<<grid_for(A->n * 8), 256, 0, st>>>(geo.grid, f.lay, A->n, A->vox, f.lay.wrap ? f.edge : f.f32, 0);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

cudaError_t anchor_scatter(const Grid &g, const Layout &lay, const Anchor &A, const float *pa, float *vol,
                           cudaStream_t st)
{
    if (A.n == 0) return cudaSuccess;
    k_scatter<<<grid_for(A.n), 256, 0, st>>>(g, lay, A.n, A.vox, pa, vol);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

cudaError_t anchor_gather(const Anchor &A, const float *vol, float *pa, cudaStream_t st)
{
    if (A.n == 0) return cudaSuccess;
    k_gather<<<grid_for(A.n), 256, 0, st>>>(A.n, A.vox, vol, pa);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

}  // namespace omni3d
