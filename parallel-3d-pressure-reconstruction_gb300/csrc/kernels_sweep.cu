// Omni sweep over the traced lines: the accumulation half of bodyIntegralInner
// (K:1743-1863), bodyIntegralInnerWeighted (K:1993-2135) and bodyIntegralInnerSelect
// (K:2280-2537), the normalisation
// devidecountInner (K:6746-6759), the curl indicator (K:8352-8378) and the gauge.
//
// One thread walks one line by decoding its 2-bit staircase; a warp holds a group (walk.cuh):
// the lines of one direction through a lattice tile, all at the same level of the volume.  The
// edge record of each visited voxel is one 16-byte gather; contributions go to an interleaved
// (pn, count) pair with one vector reduction (red.global.add.v2.f32) per visited voxel.  The
// trapezoid prefix integral along the line is a compensated (Kahan) FP32 sum.
//
// What bounds the full sweep (selected method, 160^3, 642 directions, ncu): the L1 data pipe, 82 %
// busy -- eight cycles to write back a warp's 16-byte gather, four wavefronts for its lines, and
// about eight for the reduction -- and, with 0.48 reduction sectors per visit, the L2's atomic
// rate (the chip takes about 200 G sector operations per second whatever their width).  In the
// row-major volume the same sweep had 0.76 sectors per visit and 14 wavefronts for gather and
// reduction instead of 7.5; 256^3 / 642 directions: 73.6 -> 44.2 ms.  With the gathers taken out it would
// take 32 ms, with the reductions taken out 34.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "fixed.cuh"
#include "fold.cuh"
#include "omni3d_internal.h"
#include "walk.cuh"

namespace omni3d {

// Steps whose gathers a walk issues together, and the launch shape: 32 warps per SM at 64
// registers, in small CTAs that free their slots as soon as their own lines end.  256^3 / 642
// directions: batches of 4 in 16 CTAs of 64 threads 44.7 ms, 4 CTAs of 256 46.2, 20 of 64 (48
// registers) 51.9; batches of 2 45.3, of 8 49.1 or more (fewer warps, or spills).
constexpr int kWalkBatch = 4;
constexpr int kSweepThreads = 64, kSweepBlocks = 16;  // threads per CTA, CTAs per SM

namespace {

// Contributions into the accumulators.  ACC float2: (pn, count), one FP32 vector reduction;
// double2: the FP64 defect-correction sweep's, two FP64 reductions; long long: the
// bit-reproducible mode's, two 64-bit fixed-point additions; float, double, unsigned long long:
// the same with pn alone.  All are stated as reductions: entry() hides from the compiler that the
// address is global, and of an atomicAdd it would make an atomic with a result (a plain sweep at
// 128^3: 6.4 ms so with pn alone, 5.0 as a reduction; 5.6 with the counts).
template <typename ACC>
struct Scales {};
template <>
struct Scales<long long> {
    FixScale pn, cnt;
    long long *counts;  // the lane's copy
};
template <>
struct Scales<unsigned long long> {
    FixScale pn;
};
template <typename ACC>
__device__ __forceinline__ Scales<ACC> load_scales(const double *fix, ACC *copy, size_t n)
{
    if constexpr (std::is_same<ACC, long long>::value)
        return {fix_scale(fix[kFixPn]), fix_scale(fix[kFixCnt]), copy + n};
    else if constexpr (std::is_same<ACC, unsigned long long>::value) return {fix_scale(fix[kFixPn])};
    else return {};
}
__device__ __forceinline__ void acc_add(const Scales<float2> &, float2 *acc, uint32_t v, float x, float y)
{
    float2 *a = entry(acc, v);
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(__cvta_generic_to_global(a)), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void acc_add(const Scales<double2> &, double2 *acc, uint32_t v, float x, float y)
{
    double2 *a = entry(acc, v);
    const size_t g = __cvta_generic_to_global(a);
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(g), "d"((double)x) : "memory");
    asm volatile("red.global.add.f64 [%0 + 8], %1;" ::"l"(g), "d"((double)y) : "memory");
}
__device__ __forceinline__ void acc_add(const Scales<long long> &s, long long *acc, uint32_t v, float x, float y)
{
    fix_add(entry(acc, v), x, s.pn);
    fix_add(entry(s.counts, v), y, s.cnt);
}

__device__ __forceinline__ void acc_add(const Scales<float> &, float *acc, uint32_t v, float x, float)
{
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(entry(acc, v))), "f"(x) : "memory");
}
__device__ __forceinline__ void acc_add(const Scales<double> &, double *acc, uint32_t v, float x, float)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(entry(acc, v))), "d"((double)x) : "memory");
}
__device__ __forceinline__ void acc_add(const Scales<unsigned long long> &s, unsigned long long *acc, uint32_t v, float x, float)
{
    fix_add(reinterpret_cast<long long *>(entry(acc, v)), x, s.pn);
}

// n / csum for a batch of the walk (f.quick has seen csum far from the subnormal range): the
// reciprocal's and the product's rounding, as __fdividef's within 2 ulp, without its scaling.
__device__ __forceinline__ float quick_div(float n, float csum)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(csum));
    return n * r;
}
// n / csum of a batch's contribution.  The fixed-point sums take the division of the general form:
// which form a batch takes depends on all of a warp's lines, and the bits of the bit-reproducible mode
// must not depend on the line order.
template <typename ACC>
__device__ __forceinline__ float batch_weight(float n, float csum)
{
    constexpr bool kFixed = std::is_same<ACC, long long>::value || std::is_same<ACC, unsigned long long>::value;
    return kFixed ? __fdividef(n, csum) : quick_div(n, csum);
}
constexpr float kQuickMin = 1e-30f;  // least csum of a batch that uses quick_div
constexpr float kQuickCurl = 1e-25f; // least curl of one that starts a sum
constexpr uint32_t kAllIdle = 0x55555555u & ((1u << (2 * kWalkBatch)) - 1u);  // no step of the batch is the lane's

// What every accumulation keeps along a line.
template <int GRAD, typename ACC>
struct LineSum {
    const LineWalk &L;
    ACC *acc;          // the lane's copy
    const Scales<ACC> scales;
    float4 gl;         // sample of the last voxel
    float I = 0.0f, comp = 0.0f;

    __device__ __forceinline__ void add(uint32_t v, float x, float y) const
    {
        acc_add(scales, acc, v, x, y);
    }
    // I += the trapezoid increment of step q of a batch, or 0 on a lane that does not take it
    // (`t` false: the lane's line is not in the volume, so that its sums are still zero or not
    // read again).  No branch: the lanes of a step mostly agree, and selections cost less.
    __device__ __forceinline__ void integrate(uint32_t c, int q, const float4 &gv, bool t)
    {
        const float x = step_increment<GRAD>(L, c, q, gv, gl);
        kahan_add(I, comp, t ? x : 0.0f);
        if (GRAD != kGradEdge) gl = gv;
    }
};

// Plain method: every voxel of the line, the entry included, receives p[entry] + I(v).
template <int GRAD, typename ACC>
struct PlainWalk : LineSum<GRAD, ACC> {
    float pe;
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t, const float4 (&)[kWalkBatch], const int32_t (&)[kWalkBatch]) const
    {
        return true;
    }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                          const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++)
        {
            const bool t = taken<MASK>(idle, q);
            this->integrate(c, q, g[q], t);
            if (t) this->add(v[q], pe + this->I, 1.0f);
        }
    }
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t, uint32_t, const uint32_t (&)[kWalkBatch],
                                            const float4 (&)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
    }
};

// SELF = false leaves the entry out (the minimum-curl plain variant, K:2797-2936).
template <int GRAD, bool SELF, typename ACC>
__global__ void __launch_bounds__(kSweepThreads, kSweepBlocks)
k_sweep_plain(Grid g, Layout lay, WalkLines W,
              WalkField F, const float *__restrict__ p, ACC *pncnt, const double *__restrict__ fix)
{
    LineWalk L;
    if (!L.init<GRAD == kGradVoxel>(g, lay, W)) return;
    const float4 *field = lane_field<GRAD>(F, lay, L);
    PlainWalk<GRAD, ACC> f{{L, pncnt + L.copy, load_scales(fix, pncnt + L.copy, (size_t)lay.copies * (size_t)g.V), sample<GRAD>(field, L.v)}, __ldg(p + L.copy + L.v)};
    if (SELF && L.on) f.add(L.v, f.pe, 1.0f);
    walk_steps<kWalkBatch, GRAD, false, GRAD == kGradVoxel>(L, field, nullptr, f);
}

// Weighted methods.  RAW = false (K:1993-2135): the entry receives nothing; step s of the line
// (s = 1..m) adds w_s (p[entry] + I_s) and w_s, w_s = s / sum_{t<=s} curl_t/1e4, once that sum
// is nonzero.  Each curl/1e4 term is the reference's correctly rounded float division, so the
// "sum != 0" decision (all curls so far zero) is the reference's.
// RAW = true (the minimum-curl variant, K:2937-3085): the sum starts at the entry's curl and the
// entry receives (p[entry], 1) / C; step s adds its curl (not divided by 1e4) and contributes
// w (p[entry] + I), w = (s + 1) / C, with no test for a zero sum: a zero sum gives infinities,
// as in the reference.
template <int GRAD, bool RAW, typename ACC>
struct WeightedWalk : LineSum<GRAD, ACC> {
    float pe;
    float csum, nseg;
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t idle, const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch]) const
    {
        if (!MASK) {
            float lo, hi;
            curl_range<false>(g, lo, hi);
            return (csum >= kQuickMin) & (lo >= 0.0f);
        }
        bool ok = csum >= kQuickMin;
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) ok = ok & ((g[q].w >= 0.0f) | !taken<MASK>(idle, q));
        return ok | (MASK & (idle == kAllIdle));
    }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                          const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++)
        {
            const bool t = taken<MASK>(idle, q);
            const float cn = t ? g[q].w : 0.0f;
            csum += RAW ? cn : __fdiv_rn(cn, 1.0e4f);
            this->integrate(c, q, g[q], t);
            nseg += t ? 1.0f : 0.0f;
            const float w = batch_weight<ACC>(nseg, csum);
            if (t) this->add(v[q], (pe + this->I) * w, w);
        }
    }
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                            const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++)
        {
            const bool t = taken<MASK>(idle, q);
            const float cn = t ? g[q].w : 0.0f;
            csum += RAW ? cn : __fdiv_rn(cn, 1.0e4f);
            this->integrate(c, q, g[q], t);
            nseg += t ? 1.0f : 0.0f;
            const float w = __fdividef(nseg, csum);
            if (t & (RAW | (csum != 0.0f))) this->add(v[q], (pe + this->I) * w, w);
        }
    }
};

template <int GRAD, bool RAW, typename ACC>
__global__ void __launch_bounds__(kSweepThreads, kSweepBlocks)
k_sweep_weighted(Grid g, Layout lay, WalkLines W,
                 WalkField F, const float *__restrict__ p, ACC *pncnt, const double *__restrict__ fix)
{
    LineWalk L;
    if (!L.init<GRAD == kGradVoxel>(g, lay, W)) return;
    const float4 *field = lane_field<GRAD>(F, lay, L);
    WeightedWalk<GRAD, RAW, ACC> f{{L, pncnt + L.copy, load_scales(fix, pncnt + L.copy, (size_t)lay.copies * (size_t)g.V), sample<GRAD>(field, L.v)},
                                   __ldg(p + L.copy + L.v), 0.0f, 0.0f};
    if (RAW) {
        f.csum = f.gl.w;
        f.nseg = 1.0f;
        const float w0 = __frcp_rn(f.csum);
        if (L.on) f.add(L.v, f.pe * w0, w0);
    }
    walk_steps<kWalkBatch, GRAD, false, GRAD == kGradVoxel>(L, field, nullptr, f);
}

// Selected method (K:2280-2537), state machine and asymmetries included: the entry is a
// segment start when 0 < curl <= thr; before the first start an x step needs
// 0 < curl < thr, a y/z step only curl != 0; a bad voxel pauses the segment (an x step
// also pauses on curl == 0, a y/z step walks through it without adding that step's
// increment); a good voxel after a pause restarts the segment at that voxel; the z
// branch keeps the running curl/count sums on restart.
template <int GRAD, typename ACC>
struct SelectWalk : LineSum<GRAD, ACC> {
    const float *p;    // the lane's copy
    float thr;
    SelectState st;
    float p0;
    float csum = 0.0f, nseg = 0.0f;

    // every step adds to a running segment
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t idle, const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch]) const
    {
        if (!MASK) {
            float lo, hi;
            curl_range<false>(g, lo, hi);
            return st.run() & (csum >= kQuickMin) & (lo > 0.0f) & (hi < thr);
        }
        bool ok = st.run() & ((csum >= kQuickMin) | (nseg == 0.0f));
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++)
            ok = ok & (((g[q].w >= kQuickCurl) & (g[q].w < thr)) | !taken<true>(idle, q));
        return ok | (idle == kAllIdle);
    }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                          const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++)
        {
            const bool t = taken<MASK>(idle, q);
            csum = add_curl(csum, t ? g[q].w : 0.0f);
            this->integrate(c, q, g[q], t);
            nseg += t ? 1.0f : 0.0f;
            const float w = batch_weight<ACC>(nseg, csum);
            if (t) this->add(v[q], (p0 + this->I) * w, w);
        }
    }
    // The p values of the voxels that may start a segment are loaded together, before the sums
    // that wait for them: a segment starts only after a voxel that is not good.
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t c, uint32_t idle, const uint32_t (&v)[kWalkBatch],
                                            const float4 (&g)[kWalkBatch], const int32_t (&)[kWalkBatch])
    {
        float ps[kWalkBatch];
        bool open = !st.run();
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            ps[q] = 0.0f;
            if (open & taken<MASK>(idle, q)) ps[q] = __ldg(p + v[q]);
            open = st.may_start_after(g[q].w, thr) | !taken<MASK>(idle, q);
        }
#pragma unroll
        for (int q = 0; q < kWalkBatch; q++) {
            bool add, start, clear;
            st.step(is_x(c, q), is_y(c, q), taken<MASK>(idle, q), g[q].w, thr, add, start, clear);
            if (add) {
                // weight n / sum(curl / 1e4) of the reference (K:2390-2392), as one fast
                // division (within 2 ulp) instead of its two correctly rounded ones: the
                // weights only scale averages, and the FP64-oracle bars hold
                csum = add_curl(csum, g[q].w);
                nseg += 1.0f;
                this->integrate(c, q, g[q], true);
                const float w = __fdividef(nseg, csum);
                this->add(v[q], (p0 + this->I) * w, w);
            }
            if (GRAD != kGradEdge) this->gl = g[q];
            p0 = start ? ps[q] : p0;
            this->I = start ? 0.0f : this->I;
            this->comp = start ? 0.0f : this->comp;
            nseg = clear ? 0.0f : nseg;
            csum = clear ? 0.0f : csum;
        }
    }
};

template <int GRAD, typename ACC>
__global__ void __launch_bounds__(kSweepThreads, kSweepBlocks)
k_sweep_select(Grid g, Layout lay, WalkLines W,
               WalkField F, const float *__restrict__ p, ACC *pncnt, const double *__restrict__ fix)
{
    LineWalk L;
    if (!L.init<GRAD == kGradVoxel>(g, lay, W)) return;
    const float4 *field = lane_field<GRAD>(F, lay, L);
    p += L.copy;
    const float4 gl = sample<GRAD>(field, L.v);
    SelectState st;
    st.enter(gl.w, g.thr);
    SelectWalk<GRAD, ACC> f{{L, pncnt + L.copy, load_scales(fix, pncnt + L.copy, (size_t)lay.copies * (size_t)g.V), gl}, p, g.thr, st,
                            st.run() ? __ldg(p + L.v) : 0.0f};
    walk_steps<kWalkBatch, GRAD, false, GRAD == kGradVoxel>(L, field, nullptr, f);
}

// p = pn / count where count > 0, else the kept value; a pair of sums in FP32 or FP64.
template <typename ACC>
struct Normalize {
    const float *p_keep;
    float *p_out, *cnt_out;
    __device__ __forceinline__ void operator()(long long v, const ACC &a) const
    {
        const float pk = p_keep ? p_keep[v] : 0.0f;
        if (p_out) p_out[v] = a.y > 0 ? quotient(a) : pk;
        if (cnt_out) cnt_out[v] = (float)a.y;
    }
    static __device__ __forceinline__ float quotient(const float2 &a) { return __fdiv_rn(a.x, a.y); }
    static __device__ __forceinline__ float quotient(const double2 &a) { return (float)(a.x / a.y); }
};

// f(v, (pn, count)) of sums of pn alone, the counts known.
template <typename ACC, typename F>
struct Counted {
    F f;
    const uint32_t *through;
    template <typename T>
    __device__ __forceinline__ void operator()(long long v, T pn) const
    {
        ACC a;
        a.x = pn;
        a.y = (T)through[v];
        f(v, a);
    }
};

struct AddTo {
    float *pn, *cnt;
    __device__ __forceinline__ void operator()(long long v, const float2 &a) const
    {
        pn[v] += a.x;
        cnt[v] += a.y;
    }
};

__device__ __forceinline__ float &pn_of(float &a) { return a; }
__device__ __forceinline__ float &pn_of(float2 &a) { return a.x; }
__device__ __forceinline__ double &pn_of(double &a) { return a; }
__device__ __forceinline__ double &pn_of(double2 &a) { return a.x; }

// The seed of a sweep that accumulates on top of p_init: into the first copy.
template <typename ACC>
__global__ void k_seed_accum(Grid g, Layout lay, const float *__restrict__ p_init, ACC *pncnt)
{
    const long long V = g.V;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V;
         v += (long long)gridDim.x * blockDim.x) {
        size_t at = (size_t)v;
        if (lay.wrap) {
            const VoxelAt q(g, v);
            at = layout_index(lay, g.X, g.Y, 0, q.i, q.j, q.k);
        }
        pn_of(pncnt[at]) = p_init[v];
    }
}

// out = the copies of the row-major volume in.
__global__ void __launch_bounds__(kTileThreads) k_spread(Grid g, Layout lay, const float *__restrict__ in, float *out)
{
    __shared__ float tile[kTile * kTile];
    const TileAt at(g);
    at.rows(g, [&](int p, long long v, int, int) { tile[p] = in[v]; });
    __syncthreads();
    for (int c = 0; c < 4; c++)
        at.diagonals(g, lay, c, [&](int p, uint32_t q) { out[(size_t)c * (size_t)lay.stride + q] = tile[p]; });
}

__global__ void __launch_bounds__(kTileThreads) k_spread_voxels(Grid g, Layout lay, const float *__restrict__ in, float *out)
{
    const long long v = (long long)blockIdx.x * kTileThreads + threadIdx.x;
    if (v >= g.V) return;
    const VoxelAt at(g, v);
    const float x = in[v];
#pragma unroll
    for (int c = 0; c < 4; c++) out[(size_t)c * (size_t)lay.stride + layout_index(lay, g.X, g.Y, c, at.i, at.j, at.k)] = x;
}

__device__ __forceinline__ uint32_t to_bf16(float x)
{
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// BF16 pattern of a curl value.  Round to nearest even, except that a nonzero curl never
// rounds to zero and, for a thresholded method (g.curl_map), every decision of the selected
// method is kept: the kernels then compare against the BF16 stand-in g.thr of the threshold
// g.thr_src (its truncation), and a positive curl below g.thr_src maps below g.thr, one equal
// to it maps to g.thr, one above it maps above g.thr (positive BF16 patterns order like their
// values).  The decisions (curl == 0, curl < thr, curl > thr) are then those of the FP32 curl.
__device__ __forceinline__ uint32_t curl_bf16(float c, const Grid &g)
{
    if (c == 0.0f) return __float_as_uint(c) >> 16;  // +0 and -0 stay as they are
    uint32_t v = to_bf16(c);
    if ((v & 0x7fffu) == 0u) v |= 1u;  // no underflow to zero
    if (g.curl_map && c > 0.0f && g.thr_src > 0.0f) {
        const uint32_t t = __float_as_uint(g.thr) >> 16;
        if (c < g.thr_src) {
            if (v >= t) v = t - 1u;
        } else if (c == g.thr_src) {
            v = t;
        } else if (v <= t) {
            v = t + 1u;
        }
    }
    return v;
}

// The packed field, float4 (ax, ay, az, curl), row-major, and for skewed layouts the walks'
// edge records: per step-sign octant a copy of float4 (ex, ey, ez, curl) in the octant's class,
// e_a(v) the trapezoid increment of a step of the octant into v along a, -rho sign h_a / 2 times
// the sum of component a at both its ends (0 where the voxel it leaves lies outside).  A step
// then needs the one record of the voxel it enters.  With the coefficient in the record a step
// selects it no more (256^3 / 642 directions: operator pass 29.9 -> 27.4 ms; 64^3 selected
// sweep, which the ALU bounds, 1.25 -> 1.15 ms).
// With BF16 storage every component and the curl (curl_bf16) is rounded to BF16 first, and
// curl_out (which may be the curl array itself) receives the rounded curl: every pass sees the
// same field.
// The records of a tile are put together in shared memory and written diagonal by diagonal
// (fold.cuh): 256^3, 2.46 -> 0.50 ms against eight scattered records per voxel.
struct PackIn {
    const float *ax, *ay, *az, *curl;
    int round16;
    // a component as stored
    __device__ __forceinline__ float at(const float *a, long long v) const
    {
        const float x = a[v];
        return round16 ? __uint_as_float(to_bf16(x) << 16) : x;
    }
};
// The sums of the components over a voxel's two edges along each axis (lower, upper), and its curl.
struct VoxelEdges {
    float xl, xu, yl, yu, zl, zu, c;
};
// Packs voxel v into f32 and curl_out; its edges' sums where a layout needs them.
__device__ __forceinline__ VoxelEdges pack_voxel(const Grid &g, const PackIn &in, long long v, int i, int j, int k, bool edges,
                                                 float4 *f32, float *curl_out)
{
    VoxelEdges E{};
    const float x = in.at(in.ax, v), y = in.at(in.ay, v), z = in.at(in.az, v);
    E.c = in.curl ? in.curl[v] : 0.0f;
    if (in.round16) {
        E.c = __uint_as_float(curl_bf16(E.c, g) << 16);
        if (curl_out) curl_out[v] = E.c;
    }
    f32[v] = make_float4(x, y, z, E.c);
    if (!edges) return E;
    if (i > 0) E.xl = x + in.at(in.ax, v - 1);
    if (i < g.X - 1) E.xu = x + in.at(in.ax, v + 1);
    if (j > 0) E.yl = y + in.at(in.ay, v - g.X);
    if (j < g.Y - 1) E.yu = y + in.at(in.ay, v + g.X);
    if (k > 0) E.zl = z + in.at(in.az, v - g.XY);
    if (k < g.Z - 1) E.zu = z + in.at(in.az, v + g.XY);
    return E;
}
// The edge records of a voxel in class c: entry q of its two octants' copies.
__device__ __forceinline__ void store_edges(const Grid &g, const Layout &lay, int c, uint32_t q, const VoxelEdges &E, float4 *edge)
{
    // the coefficients of the octant that steps upward along x
    const float hx = __fmul_rn(-g.rho, g.dx) * 0.5f, h1 = __fmul_rn(-g.rho, g.dy) * 0.5f, h2 = __fmul_rn(-g.rho, g.dz) * 0.5f;
    const float hy = (c & 1) ? -h1 : h1, hz = (c & 2) ? -h2 : h2;
    // a step upward along an axis crosses the voxel's lower edge
    const float yd = (c & 1) ? E.yl : E.yu, yu = (c & 1) ? E.yu : E.yl, zd = (c & 2) ? E.zl : E.zu, zu = (c & 2) ? E.zu : E.zl;
    edge[(size_t)(2 * c) * (size_t)lay.stride + q] = make_float4(-hx * E.xu, -hy * yd, -hz * zd, E.c);
    edge[(size_t)(2 * c + 1) * (size_t)lay.stride + q] = make_float4(hx * E.xl, hy * yu, hz * zu, E.c);
}

__global__ void __launch_bounds__(kTileThreads) k_pack(Grid g, PackIn in, float4 *f32, Layout lay, float4 *edge, float *curl_out)
{
    __shared__ float sums[7][kTile * kTile];
    const TileAt at(g);
    at.rows(g, [&](int p, long long v, int i, int j) {
        const VoxelEdges E = pack_voxel(g, in, v, i, j, at.k, true, f32, curl_out);
        sums[0][p] = E.xl; sums[1][p] = E.xu; sums[2][p] = E.yl; sums[3][p] = E.yu;
        sums[4][p] = E.zl; sums[5][p] = E.zu; sums[6][p] = E.c;
    });
    __syncthreads();
    for (int c = 0; c < 4; c++)
        at.diagonals(g, lay, c, [&](int p, uint32_t q) {
            store_edges(g, lay, c, q, VoxelEdges{sums[0][p], sums[1][p], sums[2][p], sums[3][p], sums[4][p], sums[5][p], sums[6][p]}, edge);
        });
}
// p, pw: as k_spread_voxels (null: not given); a launch less for a small sweep.
__global__ void __launch_bounds__(kTileThreads) k_pack_voxels(Grid g, PackIn in, float4 *f32, Layout lay, float4 *edge, float *curl_out,
                                                              const float *__restrict__ p, float *pw)
{
    const long long v = (long long)blockIdx.x * kTileThreads + threadIdx.x;
    if (v >= g.V) return;
    const VoxelAt at(g, v);
    const VoxelEdges E = pack_voxel(g, in, v, at.i, at.j, at.k, lay.wrap != 0, f32, curl_out);
    if (!lay.wrap) return;
    const float pv = p ? p[v] : 0.0f;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t q = layout_index(lay, g.X, g.Y, c, at.i, at.j, at.k);
        store_edges(g, lay, c, q, E, edge);
        if (p) pw[(size_t)c * (size_t)lay.stride + q] = pv;
    }
}

// |curl a| x mask with the reference's stencil and evaluation order (K:8352-8378).
__global__ void k_curl(Grid g, const float *__restrict__ au, const float *__restrict__ av,
                       const float *__restrict__ aw, const float *__restrict__ mask, float *out)
{
    const long long X = g.X, Y = g.Y, Z = g.Z, XY = g.XY;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < g.V;
         v += (long long)gridDim.x * blockDim.x) {
        long long i = v % X, j = (v / X) % Y, k = v / XY;
        long long i0 = i - 1 >= 0 ? i - 1 : i, j0 = j - 1 >= 0 ? j - 1 : j, k0 = k - 1 >= 0 ? k - 1 : k;
        long long ie = i + 1 <= X - 1 ? i + 1 : i, je = j + 1 <= Y - 1 ? j + 1 : j, ke = k + 1 <= Z - 1 ? k + 1 : k;
        float dj = (float)(je - j0), dk = (float)(ke - k0), di = (float)(ie - i0);
        float cx = __fdiv_rn(__fdiv_rn(__fsub_rn(aw[i + je * X + k * XY], aw[i + j0 * X + k * XY]), dj), g.dy);
        cx = __fadd_rn(cx, __fdiv_rn(__fdiv_rn(-__fsub_rn(av[i + j * X + ke * XY], av[i + j * X + k0 * XY]), dk), g.dz));
        float cy = __fdiv_rn(__fdiv_rn(-__fsub_rn(aw[ie + j * X + k * XY], aw[i0 + j * X + k * XY]), di), g.dx);
        cy = __fadd_rn(cy, __fdiv_rn(__fdiv_rn(__fsub_rn(au[i + j * X + ke * XY], au[i + j * X + k0 * XY]), dk), g.dz));
        float cz = __fdiv_rn(__fdiv_rn(__fsub_rn(av[ie + j * X + k * XY], av[i0 + j * X + k * XY]), di), g.dx);
        cz = __fadd_rn(cz, __fdiv_rn(__fdiv_rn(-__fsub_rn(au[i + je * X + k * XY], au[i + j0 * X + k * XY]), dj), g.dy));
        float s = __fadd_rn(__fadd_rn(__fmul_rn(cx, cx), __fmul_rn(cy, cy)), __fmul_rn(cz, cz));
        out[v] = __fmul_rn(__fsqrt_rn(s), mask ? mask[v] : 1.0f);
    }
}

// Deterministic FP64 sums: fixed grid, per-block partials, one block adds them in order.
constexpr int kRedBlocks = 256, kRedThreads = 256;

__device__ __forceinline__ double block_sum(double x, double *sh)
{
    for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[w];
    __syncthreads();
    return s;
}

__global__ void k_masked_sum(long long V, const float *__restrict__ p, const float *__restrict__ cnt,
                             double *part)
{
    __shared__ double sh[32];
    double s = 0.0, n = 0.0;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V;
         v += (long long)gridDim.x * blockDim.x) {
        if (cnt[v] > 0.0f) { s += (double)p[v]; n += 1.0; }
    }
    double bs = block_sum(s, sh);
    double bn = block_sum(n, sh);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = bs; part[2 * blockIdx.x + 1] = bn; }
}

__global__ void k_finish_sums(const double *part, int nblk, int width, double *out)
{
    if (threadIdx.x < width) {
        double s = 0.0;
        for (int b = 0; b < nblk; b++) s += part[width * b + threadIdx.x];
        out[threadIdx.x] = s;
    }
}

// p -= sums[0] / sums[1] (the mean, or the reference value with sums[1] = 1).
__global__ void k_shift(long long V, const double *sums, float *p)
{
    const double sub = sums[1] > 0 ? sums[0] / sums[1] : 0.0;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V;
         v += (long long)gridDim.x * blockDim.x)
        p[v] = (float)((double)p[v] - sub);
}

__global__ void k_read_point(const float *p, long long ref, double *out) { out[0] = (double)p[ref]; out[1] = 1.0; }

// One wavefront of the centre integration (initialIntegration.cpp:9-407): every voxel at L1
// distance L = a + b + c from the centre (X/2, Y/2, Z/2), thread (a, b) taking the up to
// eight voxels (+-a, +-b, +-c).  A voxel's value is the mean over its off-centre axes, in
// x, y, z order, of (the neighbour one step nearer the centre, at distance L - 1) + or -
// rho * 0.5 * (a[voxel] + a[neighbour]) * spacing, + on the low side of the centre; FP64
// with explicit rounding in the reference's C evaluation order.
__global__ void k_centre_level(Grid g, int L, const float *__restrict__ au, const float *__restrict__ av,
                               const float *__restrict__ aw, int stride, double *pn)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long w1 = (long long)L + 1;
    if (t >= w1 * w1) return;
    const int a = (int)(t / w1), b = (int)(t % w1);
    if (a + b > L) return;
    const int c = L - a - b;
    const int cx = g.X / 2, cy = g.Y / 2, cz = g.Z / 2;
    const double rho = (double)g.rho, dx = (double)g.dx, dy = (double)g.dy, dz = (double)g.dz;
    for (int o = 0; o < 8; o++) {
        const int sx = (o & 1) ? 1 : -1, sy = (o & 2) ? 1 : -1, sz = (o & 4) ? 1 : -1;
        if ((a == 0 && sx > 0) || (b == 0 && sy > 0) || (c == 0 && sz > 0)) continue;  // each voxel once
        const int i = cx + sx * a, j = cy + sy * b, k = cz + sz * c;
        if (i < 0 || i >= g.X || j < 0 || j >= g.Y || k < 0 || k >= g.Z) continue;
        const long long ind = i + (long long)j * g.X + (long long)k * g.XY;
        double v = 0.0;
        int n = 0;
        if (a) {
            const long long nb = ind - sx;
            const double tr = __dmul_rn(__dmul_rn(__dmul_rn(0.5, __dadd_rn((double)au[ind * stride], (double)au[nb * stride])), dx), rho);
            v = sx < 0 ? __dadd_rn(pn[nb], tr) : __dsub_rn(pn[nb], tr);
            n = 1;
        }
        if (b) {
            const long long nb = ind - (long long)sy * g.X;
            const double tr = __dmul_rn(__dmul_rn(__dmul_rn(0.5, __dadd_rn((double)av[ind * stride], (double)av[nb * stride])), dy), rho);
            const double w = sy < 0 ? __dadd_rn(pn[nb], tr) : __dsub_rn(pn[nb], tr);
            v = n ? __dadd_rn(v, w) : w;
            n++;
        }
        if (c) {
            const long long nb = ind - (long long)sz * g.XY;
            const double tr = __dmul_rn(__dmul_rn(__dmul_rn(0.5, __dadd_rn((double)aw[ind * stride], (double)aw[nb * stride])), dz), rho);
            const double w = sz < 0 ? __dadd_rn(pn[nb], tr) : __dsub_rn(pn[nb], tr);
            v = n ? __dadd_rn(v, w) : w;
            n++;
        }
        pn[ind] = n == 1 ? v : __ddiv_rn(v, n == 2 ? 2.0 : 3.0);
    }
}

__global__ void k_to_float(long long V, const double *__restrict__ in, float *out)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        out[v] = (float)in[v];
}

unsigned grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    if (b > 152LL * 64) b = 152LL * 64;
    if (b < 1) b = 1;
    return (unsigned)b;
}

// p and pncnt are the walks' copies (f.lay) of the pressure and of the accumulators.
template <typename ACC>
cudaError_t sweep_full_t(const Geometry &geo, const Field &f, int method, const float *p, ACC *pncnt,
                         cudaStream_t st, const double *fix = nullptr)
{
    if (geo.n_lines == 0) return cudaSuccess;
    // every pointer the kernels dereference must be set: refuse to launch otherwise
    const bool edge = f.lay.wrap != 0;
    if (!geo.d_lines || !geo.d_groups || !geo.d_desc || !p || !pncnt || (edge ? !f.edge : !f.f32)) return cudaErrorInvalidValue;
    const unsigned blocks = group_blocks(geo, kSweepThreads);
    const WalkLines W{geo.d_groups, geo.n_groups, geo.d_lines, geo.d_desc};
    const WalkField F{f.f32, f.edge};
    auto launch = [&](auto e, auto v) {
        auto kernel = edge ? e : v;
        kernel<<<blocks, kSweepThreads, 0, st>>>(geo.grid, f.lay, W, F, p, pncnt, fix);
        OM_COUNT_LAUNCH();
    };
    if constexpr (std::is_same<ACC, float>::value || std::is_same<ACC, double>::value || std::is_same<ACC, unsigned long long>::value) {
        if (method_accum(method) != kAccPlain) return cudaErrorInvalidValue;  // the other methods' counts are sums of weights
        launch(k_sweep_plain<kGradEdge, true, ACC>, k_sweep_plain<kGradVoxel, true, ACC>);
    } else {
        switch (method_accum(method)) {
        case kAccWeighted: launch(k_sweep_weighted<kGradEdge, false, ACC>, k_sweep_weighted<kGradVoxel, false, ACC>); break;
        case kAccWeightedRawCurl: launch(k_sweep_weighted<kGradEdge, true, ACC>, k_sweep_weighted<kGradVoxel, true, ACC>); break;
        case kAccSelect: launch(k_sweep_select<kGradEdge, ACC>, k_sweep_select<kGradVoxel, ACC>); break;
        case kAccPlainNoEntry: launch(k_sweep_plain<kGradEdge, false, ACC>, k_sweep_plain<kGradVoxel, false, ACC>); break;
        default: launch(k_sweep_plain<kGradEdge, true, ACC>, k_sweep_plain<kGradVoxel, true, ACC>); break;
        }
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t sweep_full(const Geometry &geo, const Field &f, int method, const float *p, const Sums<float> &s,
                       cudaStream_t st)
{
    if (s.through) return sweep_full_t(geo, f, method, p, s.mem, st);
    return sweep_full_t(geo, f, method, p, reinterpret_cast<float2 *>(s.mem), st);
}

cudaError_t sweep_full64(const Geometry &geo, const Field &f, int method, const float *p, const Sums<double> &s,
                         cudaStream_t st)
{
    if (s.through) return sweep_full_t(geo, f, method, p, s.mem, st);
    return sweep_full_t(geo, f, method, p, reinterpret_cast<double2 *>(s.mem), st);
}

cudaError_t sweep_full_fix(const Geometry &geo, const Field &f, int method, const float *p, const Sums<long long> &s,
                           const double *scale, cudaStream_t st)
{
    if (!scale) return cudaErrorInvalidValue;
    if (s.through) return sweep_full_t(geo, f, method, p, reinterpret_cast<unsigned long long *>(s.mem), st, scale);
    return sweep_full_t(geo, f, method, p, s.mem, st, scale);
}

namespace {

template <typename ACC>
cudaError_t init_accum_t(const Grid &g, const Layout &lay, const float *p_init, bool seed, ACC *pncnt, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(pncnt, 0, sizeof(ACC) * (size_t)lay.copies * (size_t)g.V, st);
    if (e != cudaSuccess || !seed || !p_init) return e;
    k_seed_accum<ACC><<<grid_for(g.V), 256, 0, st>>>(g, lay, p_init, pncnt);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

// f of every voxel's (pn, count), a pair ACC of T
template <typename ACC, typename T, typename F>
cudaError_t fold_sums(const Grid &g, const Layout &lay, const Sums<T> &s, const F &f, cudaStream_t st)
{
    if (s.through) return fold_copies(g, lay, (const T *)s.mem, Counted<ACC, F>{f, s.through}, st);
    return fold_copies(g, lay, reinterpret_cast<const ACC *>(s.mem), f, st);
}

}  // namespace

cudaError_t init_accum64(const Grid &g, const Layout &lay, const float *p_init, bool seed, const Sums<double> &s, cudaStream_t st)
{
    if (s.through) return init_accum_t(g, lay, p_init, seed, s.mem, st);
    return init_accum_t(g, lay, p_init, seed, reinterpret_cast<double2 *>(s.mem), st);
}

cudaError_t normalize64(const Grid &g, const Layout &lay, const Sums<double> &s, const float *p_keep, float *p_out,
                        float *cnt_out, cudaStream_t st)
{
    return fold_sums<double2>(g, lay, s, Normalize<double2>{p_keep, p_out, cnt_out}, st);
}

cudaError_t normalize(const Grid &g, const Layout &lay, const Sums<float> &s, const float *p_keep, float *p_out,
                      float *cnt_out, cudaStream_t st)
{
    return fold_sums<float2>(g, lay, s, Normalize<float2>{p_keep, p_out, cnt_out}, st);
}

cudaError_t accum_split(const Grid &g, const Layout &lay, const Sums<float> &s, float *pn, float *cnt, cudaStream_t st)
{
    return fold_sums<float2>(g, lay, s, AddTo{pn, cnt}, st);
}

cudaError_t init_accum(const Grid &g, const Layout &lay, const float *p_init, bool seed, const Sums<float> &s, cudaStream_t st)
{
    if (s.through) return init_accum_t(g, lay, p_init, seed, s.mem, st);
    return init_accum_t(g, lay, p_init, seed, reinterpret_cast<float2 *>(s.mem), st);
}

cudaError_t spread_volume(const Grid &g, const Layout &lay, const float *in, float *out, cudaStream_t st)
{
    if (!lay.wrap) return in == out ? cudaSuccess : cudaErrorInvalidValue;
    if (by_tiles(g, lay)) k_spread<<<tile_blocks(g), kTileThreads, 0, st>>>(g, lay, in, out);
    else k_spread_voxels<<<voxel_blocks(g), kTileThreads, 0, st>>>(g, lay, in, out);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

cudaError_t pack_field(const Grid &g, const float *ax, const float *ay, const float *az, const float *curl,
                       Field *f, bool round_bf16, cudaStream_t st, float *curl_rounded,
                       const float *p, float *pw)
{
    if (!f->f32 || (f->lay.wrap && !f->edge)) return cudaErrorInvalidValue;
    const PackIn in{ax, ay, az, curl, round_bf16 ? 1 : 0};
    if (by_tiles(g, f->lay)) k_pack<<<tile_blocks(g), kTileThreads, 0, st>>>(g, in, f->f32, f->lay, f->edge, curl_rounded);
    else k_pack_voxels<<<voxel_blocks(g), kTileThreads, 0, st>>>(g, in, f->f32, f->lay, f->edge, curl_rounded, p, pw);
    OM_COUNT_LAUNCH();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess && p && by_tiles(g, f->lay) ? spread_volume(g, f->lay, p, pw, st) : e;
}

namespace {
__global__ void k_field_curl(long long V, const float4 *__restrict__ f32, float *out)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        out[v] = f32[v].w;
}
}  // namespace

cudaError_t field_curl(long long V, const float4 *f32, float *out, cudaStream_t st)
{
    k_field_curl<<<grid_for(V), 256, 0, st>>>(V, f32, out);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

cudaError_t curl_field(const Grid &g, const float *ax, const float *ay, const float *az, const float *mask,
                       float *out, cudaStream_t st)
{
    k_curl<<<grid_for(g.V), 256, 0, st>>>(g, ax, ay, az, mask, out);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

cudaError_t apply_gauge(long long V, int gauge, long long ref, const float *cnt, float *p, double *scratch,
                        cudaStream_t st)
{
    if (gauge == OMNI3D_GAUGE_NONE) return cudaSuccess;
    if (gauge == OMNI3D_GAUGE_MEAN) {
        k_masked_sum<<<kRedBlocks, kRedThreads, 0, st>>>(V, p, cnt, scratch + 2);
        OM_COUNT_LAUNCH();
        k_finish_sums<<<1, 32, 0, st>>>(scratch + 2, kRedBlocks, 2, scratch);
        OM_COUNT_LAUNCH();
    } else {
        k_read_point<<<1, 1, 0, st>>>(p, ref, scratch);
        OM_COUNT_LAUNCH();
    }
    k_shift<<<grid_for(V), 256, 0, st>>>(V, scratch, p);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

size_t gauge_scratch_doubles() { return 2 + 2 * kRedBlocks; }

cudaError_t centre_integration(const Grid &g, const float *ax, const float *ay, const float *az, int stride,
                               double pref, double *scratch, float *out, cudaStream_t st)
{
    if (!ax || !ay || !az || !scratch || !out) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(double) * (size_t)g.V, st);
    if (e != cudaSuccess) return e;
    // voxel 0 takes pref first, as in the reference; its own wavefront overwrites it
    if ((e = cudaMemcpyAsync(scratch, &pref, sizeof(double), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;  // pref is a host stack value
    const int cx = g.X / 2, cy = g.Y / 2, cz = g.Z / 2;
    const int lmax = std::max(cx, g.X - 1 - cx) + std::max(cy, g.Y - 1 - cy) + std::max(cz, g.Z - 1 - cz);
    for (int L = 1; L <= lmax; L++) {
        const long long n = ((long long)L + 1) * ((long long)L + 1);
        k_centre_level<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(g, L, ax, ay, az, stride, scratch);
        OM_COUNT_LAUNCH();
    }
    k_to_float<<<grid_for(g.V), 256, 0, st>>>(g.V, scratch, out);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

}  // namespace omni3d
