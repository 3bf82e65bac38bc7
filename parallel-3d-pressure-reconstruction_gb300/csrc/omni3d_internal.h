// Internal declarations shared by the CUDA translation units of libomni3d_gb300.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "omni3d.h"

namespace omni3d {

// Number of kernels this library has launched (process-wide, all contexts).
extern unsigned long long g_kernel_launches;
#define OM_COUNT_LAUNCH() (__atomic_fetch_add(&omni3d::g_kernel_launches, 1ull, __ATOMIC_RELAXED))

// Per-direction constants, computed once on the host (exact libm evaluation of the
// rotation of K:6175-6191) and read by the tracing kernels.
struct DirEntry {
    float ct, st, cp, sp;  // cos/sin of theta and phi
    float k1, k2, k3;      // the direction as read from the direction file
    int cas;               // which branch of cross2point (K:663-1113) applies: 1..7, 0 none
    int orig;              // index of the direction in the caller's list
    int pad_;
};

// Grid constants passed by value to every kernel.
struct Grid {
    int X, Y, Z;
    long long XY, V;
    float cx, cy, cz;       // (N-1)/2 in float, K:665-667
    float dx, dy, dz, rho;  // spacing and density
    float ls;               // line spacing
    float thr;              // select threshold the kernels compare against (thr_src, or with
                            // BF16 storage its BF16 stand-in, see k_pack)
    int ng;                 // lattice points per row, K:6159-6167
    float thr_src;          // select threshold as given
    int curl_map;           // 1: BF16 storage of a thresholded method (curl rounded so that
                            // every threshold decision is kept)
};

// One traced line (16 bytes): entry voxel, exit voxel (linear indices), direction and
// number of staircase steps.  The sign of every axis step is fixed per line: toward the
// exit.
struct LineRec {
    uint32_t e, x;
    int32_t dir;
    int32_t m;
};

// One group of lines: the lines of one direction through one tile of 32 lattice points, walked
// by one warp, one line per lane.
struct GroupRec {
    uint32_t line0;  // first line; lane l walks line line0 + l
    uint32_t word0;  // step words: word w of lane l at desc[32 * (word0 + w) + l]
    uint32_t span;   // steps from the group's lowest entry level to its highest exit level
    uint32_t info;   // lines (1..32) in the low bits, the direction's signs (bit a: k_a >= 0) above
};
constexpr uint32_t kGroupCount = 0xffu;
constexpr int kGroupSigns = 8;

// The filtered walk (geometry.cuh) takes directions with | |k|^2 - 1 | up to this.
constexpr float kUnitMax = 6.103515625e-5f;  // 2^-14

// Device-resident geometry of one (grid, direction set, line spacing) triple.  Lines are
// grouped by (direction, lattice tile), a warp each; a group's step words are interleaved
// lane by lane, 16 steps of 2 bits per word: the axis of the step or kIdle (walk.cuh).
struct Geometry {
    Grid grid;
    int nv = 0;
    int dir_group = 4;              // neighbouring directions interleaved per lattice tile
    int tile_width = 8;             // lattice tile width in points (4, 8 or 16; 32 points a tile)
    DirEntry *d_dirs = nullptr;
    float4 *d_off = nullptr;        // per line: centred offset (x, y, z) of its lattice point
    LineRec *d_lines = nullptr;
    GroupRec *d_groups = nullptr;
    uint32_t *d_desc = nullptr;
    uint32_t *d_lines_through = nullptr;  // per voxel: lines through it (built on first use)
    unsigned max_through = 0;       // the most lines through one voxel (0: not computed)
    unsigned long long *d_counters = nullptr;  // walk counters (early stops, voxel visits)
    int unit_dirs = 0;              // directions of unit length to within kUnitMax (the filtered walk's)
    int walk_rule = 0;              // OmWalker rule of the staircases (3: per field, minimum curl)
    long long walk_generation = 0;  // incremented by every walk
    long long n_lines = 0, n_groups = 0, n_words = 0;
    long long n_units = 0;          // sum over lines of (steps + 1)
    long long walk_errors = 0;
};

// CTAs of `threads` threads that give every group a warp.
inline unsigned group_blocks(const Geometry &g, int threads)
{
    const long long per = threads / 32;
    return (unsigned)((g.n_groups + per - 1) / per);
}

// How a walk addresses a volume.  wrap = 0: one row-major copy.  Otherwise four skewed copies,
// one per pair of opposite step-sign octants, each `stride` entries after the last: with the
// signs (1, oy, oz) of the class, voxel (i, j, k) lies in plane (i + oy j + oz k) mod Y at
// k X + i (a bijection: j follows from the plane).  The voxels of one level of a walk are then
// one plane, and the 32 lines of a group, which cross a level together, touch a patch of a few
// short contiguous rows of it, where in the row-major volume no two voxels of a level share a
// row.  Simulated over the traced staircases (128^3, 16 directions of the 642), a warp's
// reductions touch 0.48 sectors per voxel visit instead of 0.75 and its 16-byte gathers 0.46
// instead of 0.84.  A step adds one plane (XZ entries), upward or downward; leaving the copy
// (index >= wrap after the step) wraps it around by wrap = V, which one unsigned minimum does.
struct Layout {
    uint32_t wrap = 0;
    int XZ = 0;
    int Y = 0;
    int copies = 1;
    long long stride = 0;
};

#ifdef __CUDACC__
#define OM_HD __host__ __device__ __forceinline__
#else
#define OM_HD inline
#endif

// Step signs of a line (bit a set: upward along axis a), those of its direction along an axis
// it does not move on.
OM_HD int line_signs(int ie, int je, int ke, int ix, int jx, int kx, int dir_signs)
{
    int s = dir_signs & 7;
    if (ix != ie) s = (s & ~1) | (ix > ie ? 1 : 0);
    if (jx != je) s = (s & ~2) | (jx > je ? 2 : 0);
    if (kx != ke) s = (s & ~4) | (kx > ke ? 4 : 0);
    return s;
}

// Class of the signs: bit 0 when y steps against x, bit 1 when z does.
OM_HD int layout_class(int signs)
{
    const int x = signs & 1, y = (signs >> 1) & 1, z = (signs >> 2) & 1;
    return (x ^ y) | ((x ^ z) << 1);
}

// Index of voxel (i, j, k) within the class-c copy of a skewed layout (X, Y: grid sizes).
OM_HD uint32_t layout_index(const Layout &lay, int X, int Y, int c, int i, int j, int k)
{
    int p = (i + ((c & 1) ? -j : j) + ((c & 2) ? -k : k)) % Y;
    if (p < 0) p += Y;
    return (uint32_t)p * (uint32_t)lay.XZ + (uint32_t)k * (uint32_t)X + (uint32_t)i;
}

// The skewed layout of a grid (row-major when its indices would not fit: 2^30 voxels or more).
inline Layout skewed_layout(const Grid &g)
{
    Layout l;
    l.stride = g.V;
    if (g.V >= (1LL << 30)) return l;
    l.wrap = (uint32_t)g.V;
    l.XZ = g.X * g.Z;
    l.Y = g.Y;
    l.copies = 4;
    return l;
}
inline Layout row_major_layout(const Grid &g)
{
    Layout l;
    l.stride = g.V;
    return l;
}

// ---------------------------------------------------------------- launchers (kernels_*.cu)
// All launchers are asynchronous on `st` and return the launch status.

// Lines of every (direction, lattice point) pair, in that order.  Allocates and fills
// g->d_off, g->d_lines, g->d_groups, g->d_desc; walks every line.  Synchronises `st`.
cudaError_t build_geometry(Geometry *g, cudaStream_t st, std::string *err);
void free_geometry(Geometry *g);
// (Re)walk every line with walk rule `rule` (curl: the field for rule 3).  Synchronises st,
// updates n_units / walk_errors and drops d_lines_through.
cudaError_t run_walk(Geometry *g, int rule, const float *curl, cudaStream_t st);
// Count the lines through every voxel into g->d_lines_through (once per geometry).  scratch: the
// layout's copies of a 4-byte volume (overwritten; unused when row-major).
cudaError_t ensure_lines_through(Geometry *g, const Layout &lay, uint32_t *scratch, cudaStream_t st);
// The most lines through one voxel (once per geometry; synchronises st).
cudaError_t max_lines_through(Geometry *g, const Layout &lay, uint32_t *scratch, cudaStream_t st, unsigned *out);

// Exclusive scans (out has n + 1 entries; out[n] = total).  tmp must hold
// scan_tmp_elems(n) elements.
size_t scan_tmp_elems(long long n);
cudaError_t exclusive_scan_u32(const uint32_t *in, uint32_t *out, long long n, uint32_t *tmp,
                               cudaStream_t st);
cudaError_t exclusive_scan_u64(const unsigned long long *in, unsigned long long *out,
                               long long n, unsigned long long *tmp, cudaStream_t st);

// Brick-staged form of the geometry (kernels_brick.cu): every line cut at the boundaries of
// 16^3 voxel bricks into segments, stored brick-major; plus the per-solve segment
// summaries and carry-in states.
struct Bricks {
    bool built = false;
    int nbx = 0, nby = 0, nbz = 0;
    long long n_bricks = 0, n_segs = 0;
    uint4 *rec = nullptr;            // 2 x uint4 per segment, grouped by brick
    uint32_t *brick_off = nullptr;   // n_bricks + 1 segment offsets
    uint32_t *line_seg = nullptr;    // n_lines + 1: line-major id of each line's first segment
    uint4 *items = nullptr;          // work items (brick, first segment, end segment, 0)
    uint32_t n_items = 0;
    int grid = 0;                    // CTAs per brick pass (one per SM)
    uint32_t *work = nullptr;        // [0] work counter, [1] error flag (a TMA wait gave up)
    void *summ = nullptr;            // per-segment summaries of the prepared method
    void *carry = nullptr;           // per-segment carry-in states
    size_t summ_cap = 0, carry_cap = 0;
    int prepared_method = -1;
    const void *map_for = nullptr;   // field the tensor map describes
    alignas(64) unsigned char map[128];  // CUtensorMap of the float4 field
};

// Cut the lines into brick segments (once per geometry); cudaErrorNotSupported when the
// engine cannot be used (no tensor-map support, more than 2^32 segments).
cudaError_t build_bricks(const Geometry &geo, Bricks *B, cudaStream_t st, std::string *err);
void free_bricks(Bricks *B);

// Gradient field on the device; with BF16 storage every value in it is a BF16 one.
struct Field {
    float4 *f32 = nullptr;          // (ax, ay, az, curl), row-major, always present
    Layout lay;                     // layout of the walks' copies
    float4 *edge = nullptr;         // skewed layouts: the walks' edge records (see k_pack)
    float *curl = nullptr;          // curl (methods that read it), also in f32[v].w
};

// Sums of a full sweep, in the walks' copies: (pn, count) of every voxel, or pn alone where the
// count is known beforehand (`through`: the plain method's is the number of lines through the
// voxel, which the geometry has once an operator has been built).
template <typename T>
struct Sums {
    T *mem = nullptr;
    const uint32_t *through = nullptr;  // row-major counts: pn alone is summed
};

// Brick passes B1 + L for the field f (FP32) and the method: per-segment carry-in states.
cudaError_t brick_prepare(const Geometry &geo, Bricks *B, const Field &f, int method, cudaStream_t st,
                          std::string *err);
// Brick pass B2: one full sweep from p into pncnt, the same contributions as sweep_full.
cudaError_t brick_sweep(const Geometry &geo, Bricks *B, int method, const float *p, float2 *pncnt,
                        cudaStream_t st);
// The error flag of the brick passes (1: a TMA wait gave up).  Synchronises st.
cudaError_t brick_error(const Bricks &B, int *flag, cudaStream_t st);

// initialIntegration.cpp on the device: p integrated outward from the centre voxel in FP64
// (scratch: V doubles), written to out as float.  The components are read at
// ax[v * stride] (stride 1: three arrays; 4: the float4 field).  Synchronises st once.
cudaError_t centre_integration(const Grid &g, const float *ax, const float *ay, const float *az, int stride,
                               double pref, double *scratch, float *out, cudaStream_t st);

// Pack three component arrays (+ optional curl) into the field and its edge records.  With
// round_bf16 the values are rounded to BF16 first, and the rounded curl is also written to
// curl_rounded (when given; it may be curl).  With p its copies for a sweep go to pw (skewed layouts).
cudaError_t pack_field(const Grid &g, const float *ax, const float *ay, const float *az,
                       const float *curl, Field *f, bool round_bf16, cudaStream_t st,
                       float *curl_rounded = nullptr, const float *p = nullptr, float *pw = nullptr);
// The curl a solve used (.w of its packed FP32 field) into out.
cudaError_t field_curl(long long V, const float4 *f32, float *out, cudaStream_t st);
// |curl a| x mask into out (and into field .w when f is given).
cudaError_t curl_field(const Grid &g, const float *ax, const float *ay, const float *az,
                       const float *mask, float *out, cudaStream_t st);

// One full sweep: pncnt += (sum of contributions, sum of weights) over all lines; p and pncnt
// are the walks' copies (f.lay).
// Every method but the plain one reads the curl indicator.
inline bool method_uses_curl(int method) { return method != OMNI3D_METHOD_PLAIN; }

// Walk rule of a method (OmWalker::step): 1 and 2 the fixed-boundary walks, 3 the
// minimum-curl walk (re-walked per field), 0 the nearest-candidate walk.
inline int method_walk_rule(int method)
{
    switch (method) {
    case OMNI3D_METHOD_WEIGHTED_FIXED_BC: return 1;
    case OMNI3D_METHOD_SELECT_FIXED_BC: return 2;
    case OMNI3D_METHOD_MINI_CURL:
    case OMNI3D_METHOD_WEIGHTED_MINI_CURL: return 3;
    default: return 0;
    }
}

// The accumulation along a line of a method: the variants share their base method's.
enum Accum { kAccPlain = 0, kAccSelect = 1, kAccWeighted = 2, kAccPlainNoEntry = 3, kAccWeightedRawCurl = 4 };
inline int method_accum(int method)
{
    switch (method) {
    case OMNI3D_METHOD_SELECT:
    case OMNI3D_METHOD_SELECT_FIXED_BC: return kAccSelect;
    case OMNI3D_METHOD_WEIGHTED:
    case OMNI3D_METHOD_WEIGHTED_FIXED_BC: return kAccWeighted;
    case OMNI3D_METHOD_MINI_CURL: return kAccPlainNoEntry;
    case OMNI3D_METHOD_WEIGHTED_MINI_CURL: return kAccWeightedRawCurl;
    default: return kAccPlain;
    }
}

// method: OMNI3D_METHOD_*; p is read at line entries / segment starts.
cudaError_t sweep_full(const Geometry &geo, const Field &f, int method,
                       const float *p, const Sums<float> &pncnt, cudaStream_t st);
// The same sweep accumulated in FP64 (two FP64 L2 reductions per contribution): the
// defect-correction sweep of params.sweep_fp64.
cudaError_t sweep_full64(const Geometry &geo, const Field &f, int method, const float *p,
                         const Sums<double> &pncnt, cudaStream_t st);
cudaError_t init_accum64(const Grid &g, const Layout &lay, const float *p_init, bool seed, const Sums<double> &pncnt,
                         cudaStream_t st);
// The same sweep accumulated in 64-bit fixed point (the bit-reproducible mode), with the
// voxel scales scale[kFixPn], scale[kFixCnt] (fixed.cuh).
cudaError_t sweep_full_fix(const Geometry &geo, const Field &f, int method, const float *p, const Sums<long long> &pncnt,
                           const double *scale, cudaStream_t st);
cudaError_t normalize64(const Grid &g, const Layout &lay, const Sums<double> &pncnt, const float *p_keep, float *p_out,
                        float *cnt_out, cudaStream_t st);

// p_out[v] = cnt > 0 ? pn / cnt : p_keep[v]; cnt_out[v] = cnt (either may be null), with
// (pn, cnt) the sum of the copies' accumulators.
cudaError_t normalize(const Grid &g, const Layout &lay, const Sums<float> &pncnt, const float *p_keep, float *p_out,
                      float *cnt_out, cudaStream_t st);
// pn[v] += acc[v].x, cnt[v] += acc[v].y (summed over the copies)
cudaError_t accum_split(const Grid &g, const Layout &lay, const Sums<float> &acc, float *pn, float *cnt, cudaStream_t st);
// pncnt = (seed ? p_init : 0, 0): the seed in the first copy, zero in the others
cudaError_t init_accum(const Grid &g, const Layout &lay, const float *p_init, bool seed, const Sums<float> &pncnt, cudaStream_t st);
// The walks' copies of a row-major volume (a row-major layout has one, the volume itself).
cudaError_t spread_volume(const Grid &g, const Layout &lay, const float *in, float *out, cudaStream_t st);

// Bit-reproducible mode (fixed.cuh, kernels_fixed.cu): device scales and bounds, and the
// operator rows' fixed-point (b, c) while filling.  Kernels that get a null Fixed pointer (or
// scale pointer) take the default FP32 sums.
struct Fixed {
    double *scale = nullptr;        // kFixSlots scales (device)
    unsigned *bits = nullptr;       // kBitsSlots float bits (device)
    long long *bc64 = nullptr;      // 2 per operator row (device)
    size_t cap_bc64 = 0;
    double lmax = 0.0;              // most lines through one voxel (geometry)
    int acc = 0;                    // the method's accumulation kind (weight bound)
    double hmax = 0.0;              // largest trapezoid coefficient rho * spacing / 2
    double path = 0.0;              // X + Y + Z: bound of a staircase's length
};
// Field bounds (max |a|, least nonzero curl) of the packed field into fx->bits.
cudaError_t fix_field_bounds(long long V, const float4 *f32, const Fixed &fx, cudaStream_t st);
// Scales for filling the operator (b, c), for the row sums of an iteration from the
// operator values pa (n of them), and for a full sweep reading the volume vol (V voxels).
cudaError_t fix_fill_scales(const Fixed &fx, cudaStream_t st);
cudaError_t fix_row_scale(long long n, const float *pa, const Fixed &fx, cudaStream_t st, const int *stop = nullptr);
cudaError_t fix_sweep_scales(long long V, const float *vol, const Fixed &fx, cudaStream_t st);
// bc = the fixed-point (b, c) rows as floats (only b when keep_c).
cudaError_t fix_rows_to_float(long long n, const Fixed &fx, float2 *bc, bool keep_c, cudaStream_t st);
// Fixed-point voxel sums: init (pn = seed ? p_init : 0, count = 0), one full sweep,
// normalisation (p = pn / count where count > 0, else p_keep) -- in FP64 from the exact sums.
cudaError_t init_accum_fix(const Grid &g, const Layout &lay, const float *p_init, bool seed, const Fixed &fx, const Sums<long long> &acc, cudaStream_t st);
cudaError_t normalize_fix(const Grid &g, const Layout &lay, const Sums<long long> &acc, const Fixed &fx, const float *p_keep, float *p_out,
                          float *cnt_out, cudaStream_t st);

// Anchor operator (kernels_anchor.cu).
struct Anchor {
    long long n = 0, nnz = 0;
    unsigned long long slots = 0;   // link slots of all rows
    long long placed = 0;           // walk generation + 1 whose lines' entries the anchors and row capacities are (0: none)
    uint8_t *flag = nullptr;        // V bytes: voxel is an anchor
    int32_t *wid = nullptr;         // the walks' copies of id (skewed layouts)
    int32_t *id = nullptr;          // V: anchor id or -1
    uint32_t *vox = nullptr;        // n: voxel of anchor
    unsigned long long *rowptr = nullptr;  // n x panels + 1: row capacities (lines through the voxel, in whole vectors)
    uint32_t *rowlen = nullptr;     // n x panels: entries in each row
    void *links = nullptr;          // per link the start anchor and, in weighted operators, the weight
    int kind = 0;                   // LinkKind of the links (links.cuh)
    uint32_t split = 0;             // columns of a panel (links.cuh); 0: one panel.  Two: rows 2 i, 2 i + 1 are row i's
    bool uneven = false;            // rows of very unequal lengths (minimum-curl walks; see iter_shape)
    int panels() const { return split ? 2 : 1; }
    float2 *bc = nullptr;           // n: (b, c) = (sum of w * I, sum of w)
    float *pa = nullptr, *pb = nullptr;  // iterates
    double *red = nullptr;          // reduction scratch
    // build scratch (kept between builds)
    uint32_t *u = nullptr, *pos = nullptr, *tmp = nullptr;
    unsigned long long *cnt64 = nullptr, *tmp64 = nullptr;
    uint32_t *neg = nullptr;        // 1 word: some curl value has its sign bit set
    unsigned long long *next = nullptr;  // n x panels: next free link slot of each row while filling
    // capacities in bytes, one per buffer above, so that rebuilding for a new field of the
    // same geometry allocates nothing
    size_t cap[20] = {};
};
// Builds the operator from the float4 entries of f (with BF16 storage they hold the stored
// values); returns cudaErrorNotSupported (nothing filled) when it would hold more than
// max_nnz entries (max_nnz < 0: no limit; 0: what 80 % of the free memory holds).
// fx (bit-reproducible mode): the rows' (b, c) are summed in fixed point with the scales of
// fix_fill_scales, which the caller sets before.
// scratch: the layout's copies of a 4-byte volume, overwritten.
cudaError_t anchor_build(Geometry &geo, const Field &f, int method, long long ref_voxel,
                         long long max_nnz, Anchor *A, cudaStream_t st, std::string *err,
                         Fixed *fx, uint32_t *scratch);
void anchor_free(Anchor *A);
// Entries that an operator may hold in `fr` bytes of free memory: 80 % of it (column + weight).
inline long long anchor_link_limit(size_t fr) { return (long long)(0.8 * (double)fr / 8.0); }
// Plain method: recompute only b (the field-dependent part) of an operator built by
// anchor_build for the same geometry; rows, columns and c depend on the geometry alone.
cudaError_t anchor_refresh_rhs(const Geometry &geo, const Field &f, Anchor *A, cudaStream_t st,
                               const Fixed *fx = nullptr);
// The convergence test of a step of a graph-captured chunk: rel_out[step] = sqrt(change / norm),
// *stop = step + 1 when it is below tol; a step returns at once while *stop != 0.
struct ChunkTest {
    double tol;
    int step;
    int *stop;
    double *rel_out;
};
// One iteration p_next = (b + seed * p_init_a + M p_cur) / c.  With red2 also the gauged change
// and norm sums red2[0..1] of the relative change over all anchors, and the chunk's test;
// `first`: the solve's first iteration; alone: see iter_shape.
cudaError_t anchor_step(const Anchor &A, const float *p_init, bool seed, bool first, int gauge,
                        long long ref_anchor, const float *p_cur, float *p_next, double *red2,
                        cudaStream_t st, const ChunkTest *test = nullptr, const Fixed *fx = nullptr,
                        bool alone = true);
// Gauged relative-change sums over the n values selected by mask (all when mask is null):
// out2 = {sum (d - d_ref)^2, sum (p - p_ref)^2} with d = pn - pc; the shift is the value at
// `ref` (point gauge), the mean (mean gauge) or zero.  Deterministic FP64 reduction;
// scratch holds change_scratch_doubles().
size_t change_scratch_doubles();
cudaError_t change_sums(long long n, const float *pc, const float *pn, int gauge, long long ref,
                        double *scratch, double *out2, cudaStream_t st, const uint8_t *mask);
// Flag the anchor voxels (line entries, or the segment starts of the selected method or a
// small superset of them, plus ref_voxel when >= 0) into a V-byte array.  count1 is one
// device word of scratch.
cudaError_t anchor_mark(const Geometry &geo, const Field &f, int method, long long ref_voxel,
                        uint8_t *flag, unsigned long long *count1, cudaStream_t st);
// Scatter anchor values into the walks' copies of a volume.
cudaError_t anchor_scatter(const Grid &g, const Layout &lay, const Anchor &A, const float *pa, float *vol,
                           cudaStream_t st);
// Gather anchor values from a volume.
cudaError_t anchor_gather(const Anchor &A, const float *vol, float *pa, cudaStream_t st);

// Adjoint of the plain-method solve (kernels_adjoint.cu).
struct AdjointBuffers {
    unsigned long long *tptr = nullptr;  // transposed operator (built once per operator): row starts,
    uint32_t *tlen = nullptr;            // lengths
    void *tlinks = nullptr;              // and links, of the operator's kind
    float *mu = nullptr, *lam = nullptr, *u = nullptr, *unext = nullptr, *acc = nullptr;
    float *edges = nullptr;  // the plain methods' dL/de, 3 axes of every copy of the layout
    bool no_links = false;   // tests: the transposed links find no memory
};
void adjoint_free(AdjointBuffers *B);
// gx, gy, gz = d<g, p_K>/d(ax, ay, az) for `method` after K iterations with the curl held
// fixed, given the operator A of that solve, its per-voxel count cnt and its packed FP32
// field f32 (whose .w holds the curl the solve used); copies: a volume in every copy of lay.  After an
// error B may hold a part of the transposed operator: adjoint_free it.
cudaError_t adjoint_solve(const Geometry &geo, const Anchor &A, AdjointBuffers *B, int K, int method,
                          const float4 *f32, const Layout &lay, float *copies, const float *g, const float *cnt,
                          float *gx, float *gy, float *gz, cudaStream_t st);
// out = G^T g for the output gauge G (part: gauge_transpose_scratch_doubles()).
cudaError_t gauge_transpose(long long V, int gauge, long long ref, const float *g,
                            const float *cnt, float *out, double *part, cudaStream_t st);
size_t gauge_transpose_scratch_doubles();

// Gauge: subtract p[ref] (mode POINT) or the mean over count > 0 (MEAN), FP64 reduction.
cudaError_t apply_gauge(long long V, int gauge, long long ref, const float *cnt, float *p,
                        double *scratch, cudaStream_t st);
size_t gauge_scratch_doubles();

}  // namespace omni3d
