// Adjoint of a solve: the gradient of <g, p_K> with respect to the gradient field
// (ax, ay, az), for every method, with the curl field held fixed.  No stored iterates are
// needed: with the curl fixed, a line's walk, segments, weights and the steps whose
// increments enter its integral depend on the curl alone, so the K-iteration map is affine
// in the field,
//     q_k = D^-1 (b + M q_{k-1} + seeding)        on the anchors, k = 1 .. K-1,
//     p(v) = (B(v) + S(v; q_{K-1}) + seeding) / c(v)  on every voxel with c(v) > 0,
// where a voxel v receives from every contribution c of a segment through it the weight
// w_c times (q(start_c) + I_c): B(v) = sum w_c I_c, S(v; q) = sum w_c q(start_c), c = sum w_c,
// b = B and M the weighted links on the anchors.  Its transpose is
//     mu = g / c;  lambda_{K-1} = S^T mu  (each segment's sum of w mu, sent to its start);
//     for k = K-1 .. 1:  acc += D^-1 lambda_k;  lambda_{k-1} = M^T D^-1 lambda_k (+ lambda_k
//                        where c = 0);
//     dL/dB = mu + acc on the anchors;
//     dL/da: along every segment, the suffix sum R_t of w dL/dB over the contributions at or
//     after step t multiplies the trapezoid coefficient h_t of every step whose increment
//     enters the integral, and is scattered to the two voxels of that step
//     (I_c = sum over those steps t <= c of h_t (a(v_t) + a(v_{t-1})) along the step's axis).
// The selected method (K:2280-2537), the weighted ones (K:1993-2135, 2937-3085) and the
// plain ones (K:1743-1863, 2797-2936) differ only in the line program below.  The curl of
// a voxel is read from .w of the packed FP32 field of the solve (the stored curl for BF16
// storage).  The derivative through the curl (its weights and segment decisions, which
// are piecewise constant in it) is not included.
#include <algorithm>
#include <utility>

#include "fold.cuh"
#include "links.cuh"
#include "omni3d_internal.h"
#include "sums.cuh"
#include "walk.cuh"

namespace omni3d {

namespace {

// The per-line program of a method's accumulation (the forward kernels' state machines and
// weight arithmetic): init() at the entry gives the entry's contribution weight and whether
// a segment starts there; step() for each step gives the contribution weight w (0: none),
// whether the step's increment enters the integral, and whether a new segment starts at the
// step's voxel.
template <int ACC>
struct LineProg {
    bool started = true, paused = false;
    float csum = 0.0f, nseg = 0.0f;
    __device__ __forceinline__ void init(float ce, float thr, float &w, bool &seg)
    {
        w = 0.0f;
        seg = true;
        if (ACC == kAccPlain) w = 1.0f;
        if (ACC == kAccWeightedRawCurl) {
            csum = ce;
            nseg = 1.0f;
            w = __frcp_rn(csum);
        }
        if (ACC == kAccSelect) {
            started = !(ce == 0.0f || ce > thr);
            seg = started;
        }
    }
    __device__ __forceinline__ void step(int a, float cn, float thr, float &w, bool &term, bool &restart)
    {
        w = 0.0f;
        term = false;
        restart = false;
        if (ACC == kAccPlain || ACC == kAccPlainNoEntry) {
            w = 1.0f;
            term = true;
        } else if (ACC == kAccWeighted) {
            term = true;
            csum += __fdiv_rn(cn, 1.0e4f);
            nseg += 1.0f;
            if (csum != 0.0f) w = __fdividef(nseg, csum);
        } else if (ACC == kAccWeightedRawCurl) {
            term = true;
            csum += cn;
            nseg += 1.0f;
            w = __fdividef(nseg, csum);
        } else {  // selected
            if (!started) {
                const bool ok = (a == 0) ? (cn != 0.0f && cn < thr) : (cn != 0.0f);
                if (ok) {
                    started = true;
                    restart = true;
                    nseg = 0.0f;
                    csum = 0.0f;
                }
            } else {
                const bool good = cn < thr && cn != 0.0f;
                if (!paused && good) {
                    term = true;
                    csum += cn * 1.0e-4f;
                    nseg += 1.0f;
                    w = __fdividef(nseg, csum);
                }
                const bool enter_bad = (a == 0) ? ((!paused && cn >= thr) || cn == 0.0f) : (!paused && cn >= thr);
                if (enter_bad) paused = true;
                if (paused && good) {
                    restart = true;
                    paused = false;
                    if (a != 2) {
                        nseg = 0.0f;
                        csum = 0.0f;
                    }
                }
            }
        }
    }
};

// Step decoder over a line's staircase (2-bit steps), from its own entry.
struct StepCursor {
    uint32_t word;
    uint32_t s;
    uint32_t v;
    __device__ __forceinline__ bool next(const LineWalk &L, int &a, uint32_t &prev)
    {
        if (s >= L.m) return false;
        if ((s & 15) == 0) word = L.own(s >> 4);
        a = (int)(word & 3u);
        word >>= 2;
        s++;
        prev = v;
        v += (uint32_t)(a == 0 ? L.d0 : (a == 1 ? L.d1 : L.d2));
        return true;
    }
};

__device__ __forceinline__ float curl_at(const float4 *f32, uint32_t v) { return __ldg(&f32[v].w); }

// mu = g / c where c > 0, else 0
__global__ void k_adj_mu(long long V, const float *g, const float *cnt, float *mu)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        mu[v] = cnt[v] > 0.0f ? __fdiv_rn(g[v], cnt[v]) : 0.0f;
}

// lambda[id(start)] += sum of w mu over each segment (S^T mu)
template <int ACC>
__global__ void __launch_bounds__(256) k_adj_gather(Grid g, Layout lay, WalkLines W,
                                                    const float4 *__restrict__ f32, const float *__restrict__ mu,
                                                    const int32_t *__restrict__ id, float *lam)
{
    LineWalk L;
    if (!L.init<true>(g, lay, W) || !L.on) return;
    LineProg<ACC> P;
    float w;
    bool seg;
    P.init(curl_at(f32, L.v), g.thr, w, seg);
    long long start = seg ? (long long)L.v : -1;
    float t = w != 0.0f ? w * __ldg(mu + L.v) : 0.0f;
    StepCursor c{0u, 0u, L.v};
    int a;
    uint32_t prev;
    while (c.next(L, a, prev)) {
        bool term, restart;
        P.step(a, curl_at(f32, c.v), g.thr, w, term, restart);
        if (restart) {
            if (start >= 0 && t != 0.0f) {
                const int row = __ldg(id + start);
                if (row >= 0) atomicAdd(lam + row, t);
            }
            start = c.v;
            t = 0.0f;
        }
        if (w != 0.0f) t += w * __ldg(mu + c.v);
    }
    if (start >= 0 && t != 0.0f) {
        const int row = __ldg(id + start);
        if (row >= 0) atomicAdd(lam + row, t);
    }
}

// The sum of w dB over the contributions of the segment that follows the cursor's position
// (up to the next segment start or the end of the line), without moving the cursor.
template <int ACC>
__device__ __forceinline__ float segment_total(const Grid &g, const LineWalk &L, StepCursor c, LineProg<ACC> P,
                                               const float4 *f32, const float *dB)
{
    float T = 0.0f;
    int a;
    uint32_t prev;
    while (c.next(L, a, prev)) {
        float w;
        bool term, restart;
        P.step(a, curl_at(f32, c.v), g.thr, w, term, restart);
        if (restart) break;
        if (w != 0.0f) T += w * __ldg(dB + c.v);
    }
    return T;
}

// dL/da along every segment: suffix sums R_t of w dB times the trapezoid coefficients
template <int ACC>
__global__ void __launch_bounds__(256) k_adj_grad(Grid g, Layout lay, WalkLines W,
                                                  const float4 *__restrict__ f32, const float *__restrict__ dB,
                                                  float *gx, float *gy, float *gz)
{
    LineWalk L;
    if (!L.init<true>(g, lay, W) || !L.on) return;
    LineProg<ACC> P;
    float w;
    bool seg;
    P.init(curl_at(f32, L.v), g.thr, w, seg);
    StepCursor c{0u, 0u, L.v};
    float R = seg ? segment_total<ACC>(g, L, c, P, f32, dB) : 0.0f;
    int a;
    uint32_t prev;
    while (c.next(L, a, prev)) {
        bool term, restart;
        P.step(a, curl_at(f32, c.v), g.thr, w, term, restart);
        if (restart) R = segment_total<ACC>(g, L, c, P, f32, dB);  // the new segment's contributions
        if (term) {
            const float val = (a == 0 ? L.h0 : (a == 1 ? L.h1 : L.h2)) * R;
            float *ga = a == 0 ? gx : (a == 1 ? gy : gz);
            atomicAdd(ga + c.v, val);
            atomicAdd(ga + prev, val);
        }
        if (w != 0.0f) R -= w * __ldg(dB + c.v);
    }
}

// The plain methods' line passes over skewed copies (the passes above serve the other methods,
// whose weights follow from the curl, and row-major layouts).  Their lines are one segment of
// unit weights, so S^T mu is a sum along the line, and R a sum from its far end.  96^3 / 642
// directions: S^T mu 1.86 -> 0.78 ms, dL/da 6.8 -> 2.15 ms (a walk over every line for R and one
// with two reductions per step before).
constexpr int kAdjBatch = 4, kAdjThreads = 64, kAdjBlocks = 16;

struct SumAlong {
    float t;
    template <bool MASK>
    __device__ __forceinline__ bool quick(uint32_t, const float4 (&)[kAdjBatch], const int32_t (&)[kAdjBatch]) const { return true; }
    template <bool MASK>
    __device__ __forceinline__ void batch(uint32_t, uint32_t idle, const uint32_t (&)[kAdjBatch], const float4 (&)[kAdjBatch],
                                          const int32_t (&x)[kAdjBatch])
    {
#pragma unroll
        for (int q = 0; q < kAdjBatch; q++) t += taken<MASK>(idle, q) ? __int_as_float(x[q]) : 0.0f;
    }
    template <bool MASK>
    __device__ __forceinline__ void general(uint32_t, uint32_t, const uint32_t (&)[kAdjBatch], const float4 (&)[kAdjBatch],
                                            const int32_t (&)[kAdjBatch]) {}
};

// mu: its copies; id: row-major.  SELF: the entry contributes too.
template <bool SELF>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocks) k_adj_gather_plain(Grid g, Layout lay, WalkLines W,
                                                                              const float *__restrict__ mu,
                                                                              const int32_t *__restrict__ id, float *lam)
{
    LineWalk L;
    if (!L.init(g, lay, W)) return;
    mu += L.copy;
    SumAlong f{SELF ? __ldg(mu + L.v) : 0.0f};
    walk_steps<kAdjBatch, kNoGrad, true, false>(L, nullptr, reinterpret_cast<const int32_t *>(mu), f);
    if (!L.on || f.t == 0.0f) return;
    const int row = __ldg(id + L.e);
    if (row >= 0) atomicAdd(lam + row, f.t);
}

// dL/de of the edges e, from the lines' far ends: R = sum of dB from there to the step, and
// the step adds h R to its edge.  An edge (the two voxels of a step) is one for both octants of a
// class, kept at the voxel that the upward octant enters by it: E holds, per class, the edges
// along x, y and z in the class's copy.  One reduction per step, where dL/da itself takes two.
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocks) k_adj_grad_plain(Grid g, Layout lay, WalkLines W,
                                                                            const float *__restrict__ dB, float *E)
{
    LineWalk L;
    if (!L.init(g, lay, W)) return;
    const bool up = (L.oct & 1) != 0;
    dB += L.copy;
    E += 3 * L.copy;
    const uint32_t off = L.on ? 0u : 0xffffffffu;
    const int words = (int)((L.span + 15) >> 4);
    // the far end: the entry and the steps along each axis (the walk may have ended early, so the
    // line's intended exit does not tell)
    int n1 = 0, n2 = 0, taken_steps = 0;
    for (int w = 0; w < words; w++) {
        const uint32_t c = __ldg(L.dp + 32 * w) | off, odd = c & 0x55555555u, high = (c >> 1) & 0x55555555u;
        const uint32_t live = 0x55555555u & ~(odd & high) & (w == words - 1 && (L.span & 15) ? (1u << (2 * (L.span & 15))) - 1u : ~0u);
        taken_steps += __popc(live);
        n1 += __popc(live & odd);
        n2 += __popc(live & high);
    }
    const uint32_t X = (uint32_t)g.X, row = L.e / X;
    const int s0 = L.d0 - L.d1 > 0 ? 1 : -1, c = L.oct >> 1;
    const int s1 = (c & 1) ? -s0 : s0, s2 = (c & 2) ? -s0 : s0;
    uint32_t v = layout_index(lay, g.X, g.Y, c, (int)(L.e - row * X) + s0 * (taken_steps - n1 - n2),
                              (int)(row % (uint32_t)g.Y) + s1 * n1, (int)(row / (uint32_t)g.Y) + s2 * n2);
    const uint32_t wv = 0u - L.wv;  // the steps back go the other way round
    float R = 0.0f;
    for (int w = words - 1; w >= 0; w--) {
        uint32_t word = __ldg(L.dp + 32 * w) | off;
        if (w == words - 1 && (L.span & 15)) word |= ~0u << (2 * (L.span & 15));  // codes past the span
        for (int b = 16 / kAdjBatch; b--; word <<= 2 * kAdjBatch) {
            const uint32_t c4 = word >> (32 - 2 * kAdjBatch);
            const uint32_t idle = c4 & (c4 >> 1) & 0x55555555u;
            if (__all_sync(0xffffffffu, idle == (0x55555555u & ((1u << (2 * kAdjBatch)) - 1u)))) continue;
            uint32_t at[kAdjBatch + 1];
            float x[kAdjBatch];
            at[kAdjBatch] = v;
#pragma unroll
            for (int q = kAdjBatch - 1; q >= 0; q--) {
                const uint32_t d = by_axis(c4, q, (uint32_t)L.d0, (uint32_t)L.d1, (uint32_t)L.d2);
                v -= taken<true>(idle, q) ? d : 0u;
                v = min(v, v + wv);
                at[q] = v;
            }
#pragma unroll
            for (int q = 0; q < kAdjBatch; q++) x[q] = __ldg(dB + at[q + 1]);
#pragma unroll
            for (int q = kAdjBatch - 1; q >= 0; q--) {
                if (!taken<true>(idle, q)) continue;
                R += x[q];
                const uint32_t axis = by_axis(c4, q, 0u, (uint32_t)lay.stride, 2u * (uint32_t)lay.stride);
                const float h = by_axis(c4, q, L.h0, L.h1, L.h2);
                atomicAdd(E + (size_t)(axis + (up ? at[q + 1] : at[q])), h * R);
            }
        }
    }
}

// dL/da(v): the edges at v along each axis, over the classes.
__global__ void __launch_bounds__(kTileThreads) k_adj_edges(Grid g, Layout lay, const float *__restrict__ E, float *gx, float *gy,
                                                            float *gz)
{
    __shared__ float sum[3][kTile * kTile];
    const TileAt at(g);
    for (int c = 0; c < 4; c++) {
        const float *ex = E + 3 * (size_t)c * (size_t)lay.stride, *ey = ex + lay.stride, *ez = ey + lay.stride;
        const int sy = (c & 1) ? -1 : 1, sz = (c & 2) ? -1 : 1;  // the upward steps
        at.diagonals(g, lay, c, [&](int p, uint32_t q) {
            const int i = at.i0 + (p & 31), j = at.j0 + (p >> 5), k = at.k;
            auto next = [&](const float *e, int di, int dj, int dk) {
                return e[layout_index(lay, g.X, g.Y, c, i + di, j + dj, k + dk)];
            };
            float x = ex[q], y = ey[q], z = ez[q];
            if (i + 1 < g.X) x += next(ex, 1, 0, 0);
            if ((unsigned)(j + sy) < (unsigned)g.Y) y += next(ey, 0, sy, 0);
            if ((unsigned)(k + sz) < (unsigned)g.Z) z += next(ez, 0, 0, sz);
            sum[0][p] = c ? sum[0][p] + x : x;
            sum[1][p] = c ? sum[1][p] + y : y;
            sum[2][p] = c ? sum[2][p] + z : z;
        });
        __syncthreads();
    }
    at.rows(g, [&](int p, long long v, int, int) {
        gx[v] = sum[0][p];
        gy[v] = sum[1][p];
        gz[v] = sum[2][p];
    });
}

// The operator's links, a warp per row: transposed rows' lengths, and the transposed links.
// With two panels (split columns each) of both: row 2 i + p holds row i's links into panel p.
template <int KIND>
__global__ void k_adj_tcount(long long n, uint32_t split, const unsigned long long *rowptr, const uint32_t *rowlen,
                             const void *links, uint32_t *tcnt)
{
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= n) return;
    if ((threadIdx.x & 31) >= lanes_per_row(KIND)) return;
    const uint32_t panels = split ? 2 : 1, mine = split && row >= split ? 1 : 0;
    for (uint32_t p = 0; p < panels; p++)
        row_links<KIND>(links, rowptr[row * panels + p], rowlen[row * panels + p], threadIdx.x & 31,
                        [&](uint32_t c, float, int) { atomicAdd(tcnt + (size_t)(c + p * split) * panels + mine, 1u); });
}

template <int KIND>
__global__ void k_adj_tfill(long long n, uint32_t split, const unsigned long long *rowptr, const uint32_t *rowlen, const void *links,
                            const unsigned long long *tptr, uint32_t *tcur, void *tlinks)
{
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (row >= n) return;
    if ((threadIdx.x & 31) >= lanes_per_row(KIND)) return;
    const uint32_t panels = split ? 2 : 1, mine = split && row >= split ? 1 : 0;
    for (uint32_t p = 0; p < panels; p++)
        row_links<KIND>(links, rowptr[row * panels + p], rowlen[row * panels + p], threadIdx.x & 31, [&](uint32_t c, float w, int) {
            const size_t t = (size_t)(c + p * split) * panels + mine;
            store_link<KIND>(tlinks, tptr[t] + atomicAdd(tcur + t, 1u), (uint32_t)row - mine * split, w);
        });
}

// Capacities of the transposed rows: whole 16-byte vectors of `per` links.
__global__ void k_adj_capacity(long long n, const uint32_t *in, unsigned per, unsigned long long *out)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = (in[i] + per - 1) / per * per;
}

// u = lambda / c where c > 0, else 0; acc = u: the first term of the backward iterations.
__global__ void k_adj_first(long long n, const float *lam, const float2 *bc, float *u, float *acc)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float c = bc[i].y, x = c > 0.0f ? __fdiv_rn(lam[i], c) : 0.0f;
        u[i] = x;
        acc[i] = x;
    }
}

// One backward iteration, lambda <- M^T D^-1 lambda (+ lambda where c = 0), from u = D^-1 lambda:
// a warp per transposed row; then u <- D^-1 lambda and acc += u.  96^3 / 642 directions (34 M
// links): 133 us with a gather of lambda and of c and a division per link, 46 us with one gather, 30 us with u
// in shared memory and several rows per warp at a time.
template <int KIND, bool SMEM>
__global__ void __launch_bounds__(SMEM ? 1024 : 256, SMEM ? 1 : 4) k_adj_iterate(
    long long n, int rows, uint32_t split, const unsigned long long *__restrict__ tptr, const uint32_t *__restrict__ tlen,
    const void *__restrict__ tlinks, const float2 *__restrict__ bc, const float *__restrict__ u, float *__restrict__ unext,
    float *lam, float *acc)
{
    extern __shared__ float4 sh_vector[];
    constexpr int kWarps = (SMEM ? 1024 : 256) / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long row0 = ((long long)blockIdx.x * kWarps + warp) * rows;
    const long long mine = row0 + lane;  // the row this lane finishes
    const bool has = lane < rows && mine < n;
    float sum = 0.0f;
    constexpr int kLanes = lanes_per_row(KIND), kRows = 32 / kLanes;
    const int panels = KIND == kLink16 && split ? 2 : 1;
    for (int p = 0; p < panels; p++) {
        if (SMEM && p) __syncthreads();  // the first panel has been read
        const long long c0 = p ? (long long)split : 0;
        const float *x = gather_vector<SMEM>(u + c0, panels == 1 ? n : min((long long)split, n - c0), reinterpret_cast<float *>(sh_vector));
        const unsigned long long ptr = has ? tptr[mine * panels + p] : 0ull;
        const uint32_t len = has ? tlen[mine * panels + p] : 0u;
        for (int r = 0; r < rows; r += kRows) {
            if (row0 + r >= n) break;  // whole warps
            const int at = r + lane / kLanes;
            const unsigned long long j0 = __shfl_sync(0xffffffffu, ptr, at & 31);
            const uint32_t m = __shfl_sync(0xffffffffu, len, at & 31);
            LaneSum q;
            row_links<KIND>(tlinks, j0, at < rows ? m : 0u, lane % kLanes, [&](uint32_t c, float w, int i) {
                const float y = SMEM ? x[c] : __ldg(x + c);
                q.add(i, KIND == kLinkPair ? w * y : y);
            });
            float s = q.total();
            __syncwarp();
            for (int o = kLanes / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            s = __shfl_sync(0xffffffffu, s, ((lane - r) * kLanes) & 31);  // the row of lane r + i
            if (lane >= r && lane < r + kRows) sum += s;
        }
    }
    if (!has) return;
    const float c = bc[mine].y;
    const float l = sum + (c > 0.0f ? 0.0f : lam[mine]);
    const float t = c > 0.0f ? __fdiv_rn(l, c) : 0.0f;
    lam[mine] = l;
    unext[mine] = t;
    acc[mine] += t;
}

// dB[vox[a]] += acc[a]
__global__ void k_adj_add_anchor(long long n, const uint32_t *vox, const float *acc, float *dB)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dB[vox[i]] += acc[i];
}

// Transpose of the gauge applied to the output: G = I - 1 w^T with w = [count > 0] / n_c
// (mean) or the unit vector at ref (point), so G^T g = g - w * sum(g).
constexpr int kRB = 256;
__global__ void k_sum_g(long long V, const float *g, const float *cnt, double *part)
{
    __shared__ double sh[2][32];
    double s = 0.0, n = 0.0;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x) {
        s += (double)g[v];
        n += cnt[v] > 0.0f ? 1.0 : 0.0;
    }
    for (int o = 16; o; o >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, o);
        n += __shfl_down_sync(0xffffffffu, n, o);
    }
    if ((threadIdx.x & 31) == 0) { sh[0][threadIdx.x >> 5] = s; sh[1][threadIdx.x >> 5] = n; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) { a += sh[0][w]; b += sh[1][w]; }
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
    }
}

__global__ void k_gauge_T(long long V, const float *g, const float *cnt, const double *part, int nblk, int gauge,
                          long long ref, float *out)
{
    // the blocks' sums, added once per block in their order (a thread each took 0.4 ms at 96^3)
    __shared__ double sh[2];
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int b = 0; b < nblk; b++) t += part[2 * b + threadIdx.x];
        sh[threadIdx.x] = t;
    }
    __syncthreads();
    const double S = sh[0], N = sh[1];
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x) {
        double x = (double)g[v];
        if (gauge == OMNI3D_GAUGE_MEAN && cnt[v] > 0.0f && N > 0) x -= S / N;
        if (gauge == OMNI3D_GAUGE_POINT && v == ref) x -= S;
        out[v] = (float)x;
    }
}

unsigned grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    if (b > 152LL * 64) b = 152LL * 64;
    if (b < 1) b = 1;
    return (unsigned)b;
}

}  // namespace

cudaError_t gauge_transpose(long long V, int gauge, long long ref, const float *g, const float *cnt, float *out,
                            double *part, cudaStream_t st)
{
    if (gauge == OMNI3D_GAUGE_NONE)
        return cudaMemcpyAsync(out, g, sizeof(float) * (size_t)V, cudaMemcpyDeviceToDevice, st);
    k_sum_g<<<kRB, 256, 0, st>>>(V, g, cnt, part);
    OM_COUNT_LAUNCH();
    k_gauge_T<<<grid_for(V), 256, 0, st>>>(V, g, cnt, part, kRB, gauge, ref, out);
    OM_COUNT_LAUNCH();
    return cudaGetLastError();
}

size_t gauge_transpose_scratch_doubles() { return 2 * kRB; }

void adjoint_free(AdjointBuffers *B)
{
    cudaFree(B->tptr);
    cudaFree(B->tlen);
    cudaFree(B->tlinks);
    cudaFree(B->mu);
    cudaFree(B->lam);
    cudaFree(B->u);
    cudaFree(B->unext);
    cudaFree(B->acc);
    cudaFree(B->edges);
    *B = AdjointBuffers();
}

#define ADJ_TRY(x)                               \
    do {                                         \
        cudaError_t e_ = (x);                    \
        if (e_ != cudaSuccess) return e_;        \
    } while (0)

// A temporary of the transposed operator's build, freed on every way out.
struct AdjTemp {
    void *p = nullptr;
    template <typename T>
    cudaError_t alloc(T **out, size_t elems)
    {
        const cudaError_t e = cudaMalloc(&p, sizeof(T) * std::max<size_t>(elems, 1));
        *out = e == cudaSuccess ? static_cast<T *>(p) : nullptr;
        return e;
    }
    ~AdjTemp() { cudaFree(p); }
};

template <int ACC>
void launch_adj_lines(const Geometry &geo, bool gather, const float4 *f32, const float *in, const int32_t *id,
                      float *lam, float *gx, float *gy, float *gz, cudaStream_t st)
{
    const unsigned lblocks = group_blocks(geo, 256);
    const Layout lay = row_major_layout(geo.grid);
    const WalkLines W{geo.d_groups, geo.n_groups, geo.d_lines, geo.d_desc};
    if (gather)
        k_adj_gather<ACC><<<lblocks, 256, 0, st>>>(geo.grid, lay, W, f32, in,
                                                   id, lam);
    else
        k_adj_grad<ACC><<<lblocks, 256, 0, st>>>(geo.grid, lay, W, f32, in,
                                                 gx, gy, gz);
    OM_COUNT_LAUNCH();
}

void adj_lines(int acc, const Geometry &geo, bool gather, const float4 *f32, const float *in, const int32_t *id,
               float *lam, float *gx, float *gy, float *gz, cudaStream_t st)
{
    switch (acc) {
    case kAccSelect: launch_adj_lines<kAccSelect>(geo, gather, f32, in, id, lam, gx, gy, gz, st); break;
    case kAccWeighted: launch_adj_lines<kAccWeighted>(geo, gather, f32, in, id, lam, gx, gy, gz, st); break;
    case kAccPlainNoEntry: launch_adj_lines<kAccPlainNoEntry>(geo, gather, f32, in, id, lam, gx, gy, gz, st); break;
    case kAccWeightedRawCurl: launch_adj_lines<kAccWeightedRawCurl>(geo, gather, f32, in, id, lam, gx, gy, gz, st); break;
    default: launch_adj_lines<kAccPlain>(geo, gather, f32, in, id, lam, gx, gy, gz, st); break;
    }
}

// Whether the line passes take skewed copies: the plain methods where the layout has them and
// the edges' copies fit beside what is there (12 floats per voxel, kept with the transposed operator).
bool skewed_passes(int acc, const Geometry &geo, const Layout &lay, const float *copies, AdjointBuffers *B)
{
    if (!lay.wrap || !copies || (acc != kAccPlain && acc != kAccPlainNoEntry)) return false;
    if (B->edges) return true;
    if (cudaMalloc(&B->edges, 3 * sizeof(float) * (size_t)lay.copies * (size_t)geo.grid.V) == cudaSuccess) return true;
    cudaGetLastError();
    B->edges = nullptr;
    return false;
}

cudaError_t adjoint_solve(const Geometry &geo, const Anchor &A, AdjointBuffers *B, int K, int method, const float4 *f32,
                          const Layout &lay, float *copies, const float *g, const float *cnt, float *gx, float *gy, float *gz,
                          cudaStream_t st)
{
    if (!f32 || !A.id || !A.bc || !A.vox || !A.rowptr || !A.rowlen || !A.links)
        return cudaErrorInvalidValue;
    const int acc = method_accum(method);
    const long long V = geo.grid.V, n = A.n;
    ADJ_TRY(cudaMemsetAsync(gx, 0, sizeof(float) * (size_t)V, st));
    ADJ_TRY(cudaMemsetAsync(gy, 0, sizeof(float) * (size_t)V, st));
    ADJ_TRY(cudaMemsetAsync(gz, 0, sizeof(float) * (size_t)V, st));
    if (K <= 0 || geo.n_lines == 0) return cudaSuccess;
    if (!B->mu) ADJ_TRY(cudaMalloc(&B->mu, sizeof(float) * (size_t)V));
    if (!B->lam) {
        ADJ_TRY(cudaMalloc(&B->lam, sizeof(float) * (size_t)std::max(n, 1LL)));
        ADJ_TRY(cudaMalloc(&B->u, sizeof(float) * (size_t)std::max(n, 1LL)));
        ADJ_TRY(cudaMalloc(&B->unext, sizeof(float) * (size_t)std::max(n, 1LL)));
        ADJ_TRY(cudaMalloc(&B->acc, sizeof(float) * (size_t)std::max(n, 1LL)));
    }
    // transposed operator (once per operator)
    const unsigned row_blocks = (unsigned)((n * 32 + 255) / 256);
    if (!B->tptr) {
        const long long trows = n * A.panels();
        AdjTemp t64_mem, tmp_mem, tcur_mem;
        unsigned long long *t64 = nullptr, *tmp = nullptr;
        uint32_t *tcur = nullptr;
        ADJ_TRY(cudaMalloc(&B->tlen, sizeof(uint32_t) * (size_t)std::max(trows, 1LL)));
        ADJ_TRY(tcur_mem.alloc(&tcur, (size_t)trows));
        ADJ_TRY(t64_mem.alloc(&t64, (size_t)trows));
        ADJ_TRY(tmp_mem.alloc(&tmp, scan_tmp_elems(trows)));
        ADJ_TRY(cudaMalloc(&B->tptr, sizeof(unsigned long long) * (size_t)(trows + 1)));
        ADJ_TRY(cudaMemsetAsync(B->tlen, 0, sizeof(uint32_t) * (size_t)std::max(trows, 1LL), st));
        auto count = [&](auto kernel) { kernel<<<row_blocks, 256, 0, st>>>(n, A.split, A.rowptr, A.rowlen, A.links, B->tlen); };
        if (n) {
            A.kind == kLink16 ? count(k_adj_tcount<kLink16>)
                              : (A.kind == kLink32 ? count(k_adj_tcount<kLink32>) : count(k_adj_tcount<kLinkPair>));
            OM_COUNT_LAUNCH();
            k_adj_capacity<<<grid_for(trows), 256, 0, st>>>(trows, B->tlen, (unsigned)links_per_vector(A.kind), t64);
            OM_COUNT_LAUNCH();
        }
        ADJ_TRY(exclusive_scan_u64(t64, B->tptr, trows, tmp, st));
        unsigned long long tn = 0;
        ADJ_TRY(cudaMemcpyAsync(&tn, B->tptr + trows, sizeof(tn), cudaMemcpyDeviceToHost, st));
        ADJ_TRY(cudaStreamSynchronize(st));
        if (B->no_links) return cudaErrorMemoryAllocation;
        ADJ_TRY(cudaMalloc(&B->tlinks, link_size(A.kind) * (size_t)std::max(tn, 1ULL)));
        ADJ_TRY(cudaMemsetAsync(tcur, 0, sizeof(uint32_t) * (size_t)std::max(trows, 1LL), st));
        auto fill = [&](auto kernel) { kernel<<<row_blocks, 256, 0, st>>>(n, A.split, A.rowptr, A.rowlen, A.links, B->tptr, tcur, B->tlinks); };
        if (n) {
            A.kind == kLink16 ? fill(k_adj_tfill<kLink16>)
                              : (A.kind == kLink32 ? fill(k_adj_tfill<kLink32>) : fill(k_adj_tfill<kLinkPair>));
            OM_COUNT_LAUNCH();
        }
        ADJ_TRY(cudaGetLastError());
        ADJ_TRY(cudaStreamSynchronize(st));
    }
    // mu = g / c; lambda_{K-1} = S^T mu
    k_adj_mu<<<grid_for(V), 256, 0, st>>>(V, g, cnt, B->mu);
    OM_COUNT_LAUNCH();
    ADJ_TRY(cudaMemsetAsync(B->lam, 0, sizeof(float) * (size_t)std::max(n, 1LL), st));
    ADJ_TRY(cudaMemsetAsync(B->acc, 0, sizeof(float) * (size_t)std::max(n, 1LL), st));
    const bool skewed = skewed_passes(acc, geo, lay, copies, B);
    const WalkLines W{geo.d_groups, geo.n_groups, geo.d_lines, geo.d_desc};
    const unsigned lblocks = group_blocks(geo, kAdjThreads);
    if (skewed) {
        ADJ_TRY(spread_volume(geo.grid, lay, B->mu, copies, st));
        auto kernel = acc == kAccPlain ? k_adj_gather_plain<true> : k_adj_gather_plain<false>;
        kernel<<<lblocks, kAdjThreads, 0, st>>>(geo.grid, lay, W, copies, A.id, B->lam);
        OM_COUNT_LAUNCH();
    } else {
        adj_lines(acc, geo, true, f32, B->mu, A.id, B->lam, nullptr, nullptr, nullptr, st);
    }
    // anchor iterations, backwards
    if (K > 1 && n) {
        k_adj_first<<<grid_for(n), 256, 0, st>>>(n, B->lam, A.bc, B->u, B->acc);
        OM_COUNT_LAUNCH();
        const IterShape I = iter_shape(n, true, A.kind, A.split, A.uneven);
        auto launch = [&](auto kernel) {
            if (I.bytes > 48 * 1024)
                ADJ_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kIterSmemMax));
            for (int k = K - 1; k > 1; k--) {
                kernel<<<I.blocks, I.threads, I.bytes, st>>>(n, I.rows, A.split, B->tptr, B->tlen, B->tlinks, A.bc, B->u, B->unext, B->lam,
                                                             B->acc);
                OM_COUNT_LAUNCH();
                std::swap(B->u, B->unext);
            }
            return cudaGetLastError();
        };
        ADJ_TRY(A.kind == kLink16   ? (I.smem ? launch(k_adj_iterate<kLink16, true>) : launch(k_adj_iterate<kLink16, false>))
                : A.kind == kLink32 ? launch(k_adj_iterate<kLink32, false>)
                                    : launch(k_adj_iterate<kLinkPair, false>));
    }
    // dL/dB = mu + acc on the anchors, then the line scatter
    if (n) {
        k_adj_add_anchor<<<grid_for(n), 256, 0, st>>>(n, A.vox, B->acc, B->mu);
        OM_COUNT_LAUNCH();
    }
    if (skewed) {
        ADJ_TRY(spread_volume(geo.grid, lay, B->mu, copies, st));
        ADJ_TRY(cudaMemsetAsync(B->edges, 0, 3 * sizeof(float) * (size_t)lay.copies * (size_t)V, st));
        k_adj_grad_plain<<<lblocks, kAdjThreads, 0, st>>>(geo.grid, lay, W, copies, B->edges);
        OM_COUNT_LAUNCH();
        k_adj_edges<<<tile_blocks(geo.grid), kTileThreads, 0, st>>>(geo.grid, lay, B->edges, gx, gy, gz);
        OM_COUNT_LAUNCH();
    } else {
        adj_lines(acc, geo, false, f32, B->mu, nullptr, nullptr, gx, gy, gz, st);
    }
    return cudaGetLastError();
}

}  // namespace omni3d
