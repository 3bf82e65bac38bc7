// Device line geometry, bit-exact with the reference's FP32 host evaluation.
//
// Which voxels a line visits is decided by FP32 comparisons in the reference (cross2point,
// K:663-1113, and the nearest-candidate walk, K:1762-1861).  Every float operation below
// is an explicitly rounded intrinsic, so nvcc cannot contract a multiply and an add into
// an FMA and change a rounding; the order of operations is the reference's left-to-right
// C evaluation.
#pragma once

#include "omni3d_internal.h"

namespace omni3d {

#define OM_MUL __fmul_rn
#define OM_ADD __fadd_rn
#define OM_SUB __fsub_rn
#define OM_DIV __fdiv_rn

// floor(f + 0.5) with the addition exact, as the reference evaluates it in double (K:703).
__device__ __forceinline__ int om_round_half(float f)
{
    float fl = floorf(f);
    return (int)fl + (OM_SUB(f, fl) >= 0.5f ? 1 : 0);
}

// Centred offset of lattice point pt of a direction (K:6171-6194).  The reference forms
// (row - (ng-1)/2) * spacing in double and rounds to float; the difference is an exact
// half-integer in float, so one rounded float product gives the same value.
__device__ __forceinline__ void om_line_offset(long long pt, int ng, float ls, const DirEntry &D,
                                               float &x, float &y, float &z)
{
    int row = (int)(pt / ng);
    int col = (int)(pt - (long long)row * ng);
    float h = 0.5f * (float)(ng - 1);
    float xp = OM_MUL(OM_SUB((float)row, h), ls);
    float yp = OM_MUL(OM_SUB((float)col, h), ls);
    float t = OM_MUL(xp, D.ct);
    x = OM_SUB(OM_MUL(t, D.cp), OM_MUL(yp, D.sp));
    y = OM_ADD(OM_MUL(t, D.sp), OM_MUL(yp, D.cp));
    z = OM_MUL(-xp, D.st);
}

// cross2point (K:663-1113).  `cases` has bit c-1 set when the direction satisfies the
// test of case c (evaluated once per direction on the host); a case whose offset test
// fails falls through to the next, as in the reference.  in/out keep the sentinel
// (X, Y, Z) when no intersection is recorded.
__device__ __forceinline__ void om_cross2point(const Grid &g, float x, float y, float z,
                                               float k1, float k2, float k3, int cases,
                                               int in[3], int out[3])
{
    const float cx = g.cx, cy = g.cy, cz = g.cz;
    const int X = g.X, Y = g.Y, Z = g.Z;
    in[0] = X; in[1] = Y; in[2] = Z;
    out[0] = X; out[1] = Y; out[2] = Z;
    float r;
    int t;
    if ((cases & 1) && x > -cx && x < cx) {  // case 1: k1 == 0
        float z1, z2, y3, y4;
        r = OM_DIV(OM_SUB(-cy, y), k2); z1 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(cy, y), k2); z2 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(-cz, z), k3); y3 = OM_ADD(y, OM_MUL(k2, r));
        r = OM_DIV(OM_SUB(cz, z), k3); y4 = OM_ADD(y, OM_MUL(k2, r));
        bool flag = false;
        int ic = om_round_half(OM_ADD(x, cx));
        if (z1 <= cz && z1 >= -cz) { in[0] = ic; in[1] = 0; in[2] = om_round_half(OM_ADD(z1, cz)); flag = true; }
        if (z2 <= cz && z2 >= -cz) {
            int *o = flag ? out : in;
            o[0] = ic; o[1] = Y - 1; o[2] = om_round_half(OM_ADD(z2, cz)); flag = true;
        }
        if (y3 <= cy && y3 >= -cy) {
            int *o = flag ? out : in;
            o[0] = ic; o[1] = om_round_half(OM_ADD(y3, cy)); o[2] = 0; flag = true;
        }
        if (y4 <= cy && y4 >= -cy) {
            int *o = flag ? out : in;
            o[0] = ic; o[1] = om_round_half(OM_ADD(y4, cy)); o[2] = Z - 1;
        }
        if (flag) {
            if (OM_ADD(OM_MUL((float)(out[1] - in[1]), k2), OM_MUL((float)(out[2] - in[2]), k3)) < 0) {
                t = in[1]; in[1] = out[1]; out[1] = t;
                t = in[2]; in[2] = out[2]; out[2] = t;
            }
        }
        return;
    }
    if ((cases & 2) && y > -cy && y < cy) {  // case 2: k2 == 0
        float z1, z2, x3, x4;
        r = OM_DIV(OM_SUB(-cx, x), k1); z1 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(cx, x), k1); z2 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(-cz, z), k3); x3 = OM_ADD(x, OM_MUL(k1, r));
        r = OM_DIV(OM_SUB(cz, z), k3); x4 = OM_ADD(x, OM_MUL(k1, r));
        bool flag = false;
        int jc = om_round_half(OM_ADD(y, cy));
        if (z1 <= cz && z1 >= -cz) { in[0] = 0; in[1] = jc; in[2] = om_round_half(OM_ADD(z1, cz)); flag = true; }
        if (z2 <= cz && z2 >= -cz) {
            int *o = flag ? out : in;
            o[0] = X - 1; o[1] = jc; o[2] = om_round_half(OM_ADD(z2, cz)); flag = true;
        }
        if (x3 <= cx && x3 >= -cx) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x3, cx)); o[1] = jc; o[2] = 0; flag = true;
        }
        if (x4 <= cx && x4 >= -cx) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x4, cx)); o[1] = jc; o[2] = Z - 1; flag = true;
        }
        if (flag) {
            if (OM_ADD(OM_MUL((float)(out[0] - in[0]), k1), OM_MUL((float)(out[2] - in[2]), k3)) < 0) {
                t = in[0]; in[0] = out[0]; out[0] = t;
                t = in[2]; in[2] = out[2]; out[2] = t;
            }
        }
        return;
    }
    if ((cases & 4) && z > -cz && z < cz) {  // case 3: k3 == 0 (z where y is meant, K:854-855)
        float y1, y2, x3, x4;
        r = OM_DIV(OM_SUB(-cx, x), k1); y1 = OM_ADD(y, OM_MUL(k2, r));
        r = OM_DIV(OM_SUB(cx, x), k1); y2 = OM_ADD(y, OM_MUL(k2, r));
        r = OM_DIV(OM_SUB(-cy, z), k2); x3 = OM_ADD(x, OM_MUL(k1, r));
        r = OM_DIV(OM_SUB(cy, z), k2); x4 = OM_ADD(x, OM_MUL(k1, r));
        bool flag = false;
        int kc = om_round_half(OM_ADD(z, cz));
        if (y1 <= cy && y1 >= -cy) { in[0] = 0; in[1] = om_round_half(OM_ADD(y1, cy)); in[2] = kc; flag = true; }
        if (y2 <= cy && y2 >= -cy) {
            int *o = flag ? out : in;
            o[0] = X - 1; o[1] = om_round_half(OM_ADD(y2, cy)); o[2] = kc; flag = true;
        }
        if (x3 <= cx && x3 >= -cx) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x3, cx)); o[1] = 0; o[2] = kc; flag = true;
        }
        if (x4 <= cx && x4 >= -cx) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x4, cx)); o[1] = Y - 1; o[2] = kc; flag = true;
        }
        if (flag) {
            if (OM_ADD(OM_MUL((float)(out[0] - in[0]), k1), OM_MUL((float)(out[1] - in[1]), k2)) < 0) {
                t = in[0]; in[0] = out[0]; out[0] = t;
                t = in[1]; in[1] = out[1]; out[1] = t;
            }
        }
        return;
    }
    if ((cases & 8) && x < cx && x > -cx && y < cy && y > -cy) {  // case 4: along z
        in[0] = out[0] = om_round_half(OM_ADD(x, cx));
        in[1] = out[1] = om_round_half(OM_ADD(y, cy));
        if (k3 > 0) { in[2] = 0; out[2] = Z - 1; } else { in[2] = Z - 1; out[2] = 0; }
        return;
    }
    if ((cases & 16) && x > -cx && x < cx && z > -cz && z < cz) {  // case 5: along y
        in[0] = out[0] = om_round_half(OM_ADD(x, cx));
        in[2] = out[2] = om_round_half(OM_ADD(z, cz));
        if (k2 > 0) { out[1] = Y - 1; in[1] = 0; } else { in[1] = Y - 1; out[1] = 0; }
        return;
    }
    if (cases & 32) {  // case 6: along x; reports success even on a miss (K:989)
        if (y > -cy && y < cy && z > -cz && z < cz) {
            in[1] = out[1] = om_round_half(OM_ADD(y, cy));
            in[2] = out[2] = om_round_half(OM_ADD(z, cz));
            if (k1 > 0) { out[0] = X - 1; in[0] = 0; } else { in[0] = X - 1; out[0] = 0; }
        }
        return;
    }
    if (cases & 64) {  // case 7: general direction, six face intersections
        float y1, z1, y2, z2, x3, z3, x4, z4, x5, y5, x6, y6;
        r = OM_DIV(OM_SUB(-cx, x), k1); y1 = OM_ADD(y, OM_MUL(k2, r)); z1 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(cx, x), k1); y2 = OM_ADD(y, OM_MUL(k2, r)); z2 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(-cy, y), k2); x3 = OM_ADD(x, OM_MUL(k1, r)); z3 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(cy, y), k2); x4 = OM_ADD(x, OM_MUL(k1, r)); z4 = OM_ADD(z, OM_MUL(k3, r));
        r = OM_DIV(OM_SUB(-cz, z), k3); x5 = OM_ADD(x, OM_MUL(k1, r)); y5 = OM_ADD(y, OM_MUL(k2, r));
        r = OM_DIV(OM_SUB(cz, z), k3); x6 = OM_ADD(x, OM_MUL(k1, r)); y6 = OM_ADD(y, OM_MUL(k2, r));
        bool flag = false;
        if (y1 <= cy && y1 >= -cy && z1 <= cz && z1 >= -cz) {
            in[0] = 0; in[1] = om_round_half(OM_ADD(y1, cy)); in[2] = om_round_half(OM_ADD(z1, cz)); flag = true;
        }
        if (y2 <= cy && y2 >= -cy && z2 <= cz && z2 >= -cz) {
            int *o = flag ? out : in;
            o[0] = X - 1; o[1] = om_round_half(OM_ADD(y2, cy)); o[2] = om_round_half(OM_ADD(z2, cz)); flag = true;
        }
        if (x3 <= cx && x3 >= -cx && z3 <= cz && z3 >= -cz) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x3, cx)); o[1] = 0; o[2] = om_round_half(OM_ADD(z3, cz)); flag = true;
        }
        if (x4 <= cx && x4 >= -cx && z4 <= cz && z4 >= -cz) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x4, cx)); o[1] = Y - 1; o[2] = om_round_half(OM_ADD(z4, cz)); flag = true;
        }
        if (x5 <= cx && x5 >= -cx && y5 <= cy && y5 >= -cy) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x5, cx)); o[1] = om_round_half(OM_ADD(y5, cy)); o[2] = 0; flag = true;
        }
        if (x6 <= cx && x6 >= -cx && y6 <= cy && y6 >= -cy) {
            int *o = flag ? out : in;
            o[0] = om_round_half(OM_ADD(x6, cx)); o[1] = om_round_half(OM_ADD(y6, cy)); o[2] = Z - 1; flag = true;
        }
        float dot = OM_ADD(OM_ADD(OM_MUL((float)(out[0] - in[0]), k1), OM_MUL((float)(out[1] - in[1]), k2)),
                           OM_MUL((float)(out[2] - in[2]), k3));
        if (dot < 0) {
            t = in[0]; in[0] = out[0]; out[0] = t;
            t = in[1]; in[1] = out[1]; out[1] = t;
            t = in[2]; in[2] = out[2]; out[2] = t;
        }
        return;
    }
}

// A line of a general direction (case 7 alone) that certainly misses the volume: some pair of
// axes has its projection outside the rectangle's by more than a thousand times what the roundings
// of om_cross2point amount to (its accepted face points are off by 10 u M at most, M the longest
// side, times the largest component of k: of the rotation's k2 and k3 none is above 1, but k1 may be
// anything).  Half of the lattice points of a cube miss, almost all of a long volume's; the full
// evaluation takes 12 divisions.
__device__ __forceinline__ bool om_certain_miss(const Grid &g, float x, float y, float z, float k1, float k2, float k3, int cases)
{
    if (cases != 64) return false;
    const float a1 = fabsf(k1), a2 = fabsf(k2), a3 = fabsf(k3);
    const float slack = 1.0e-3f * (float)max(max(g.X, g.Y), g.Z) * fmaxf(a1, 1.0f);
    return (fabsf(x * k2 - y * k1) > g.cx * a2 + g.cy * a1 + slack) | (fabsf(x * k3 - z * k1) > g.cx * a3 + g.cz * a1 + slack) |
           (fabsf(y * k3 - z * k2) > g.cy * a3 + g.cz * a2 + slack);
}

// Acceptance test of the caller (K:6202-6206): both voxels inside and distinct.
__device__ __forceinline__ bool om_line_valid(const Grid &g, const int in[3], const int out[3])
{
    bool inside = in[0] >= 0 && in[0] < g.X && in[1] >= 0 && in[1] < g.Y && in[2] >= 0 && in[2] < g.Z &&
                  out[0] >= 0 && out[0] < g.X && out[1] >= 0 && out[1] < g.Y && out[2] >= 0 && out[2] < g.Z;
    return inside && !(in[0] == out[0] && in[1] == out[1] && in[2] == out[2]);
}

// sqrt_rn(a) <= sqrt_rn(b) and sqrt_rn(a) < sqrt_rn(b) without computing the square roots
// unless a and b are within 2^-21 of each other (two correctly rounded square roots can
// only be equal when a / b < (1 + 2^-23)^2).  NaN compares false, as in the reference.
__device__ __forceinline__ bool om_sqrt_le(float a, float b)
{
    if (a <= b) return true;
    if (!(OM_SUB(a, b) <= OM_MUL(b, 4.76837158203125e-7f))) return false;
    return __fsqrt_rn(a) == __fsqrt_rn(b);
}
__device__ __forceinline__ bool om_sqrt_lt(float a, float b)
{
    if (!(a < b)) return false;
    if (!(OM_SUB(b, a) <= OM_MUL(a, 4.76837158203125e-7f))) return true;
    return __fsqrt_rn(a) != __fsqrt_rn(b);
}

// Squared distance of candidate voxel (ci, cj, ck) from the line at parameter r
// (K:1800-1810).
__device__ __forceinline__ float om_dist2(float x, float y, float z, float k1, float k2, float k3,
                                          float r, float ci, float cj, float ck)
{
    float a = OM_SUB(OM_ADD(x, OM_MUL(k1, r)), ci);
    float b = OM_SUB(OM_ADD(y, OM_MUL(k2, r)), cj);
    float c = OM_SUB(OM_ADD(z, OM_MUL(k3, r)), ck);
    return OM_ADD(OM_ADD(OM_MUL(a, a), OM_MUL(b, b)), OM_MUL(c, c));
}

// Walker state of one line (K:1745-1761).
struct OmWalker {
    float x, y, z, k1, k2, k3, xk1, yk2, zk3;
    int il, jl, kl, io, jo, ko;

    __device__ __forceinline__ void init(const Grid &g, float ox, float oy, float oz, float d1,
                                         float d2, float d3, int ie, int je, int ke, int ix,
                                         int jx, int kx)
    {
        x = OM_ADD(ox, g.cx); y = OM_ADD(oy, g.cy); z = OM_ADD(oz, g.cz);
        il = ie; jl = je; kl = ke; io = ix; jo = jx; ko = kx;
        float dot = OM_ADD(OM_ADD(OM_MUL(d1, (float)(ix - ie)), OM_MUL(d2, (float)(jx - je))),
                           OM_MUL(d3, (float)(kx - ke)));
        if (dot < 0) { d1 = -d1; d2 = -d2; d3 = -d3; }
        k1 = d1; k2 = d2; k3 = d3;
        xk1 = OM_MUL(x, k1); yk2 = OM_MUL(k2, y); zk3 = OM_MUL(k3, z);
    }

    // One step of the walk.  Returns the axis moved along (0, 1, 2) or -1 when no candidate
    // qualifies (the reference's loop ends there).  RULE:
    //   0  nearest candidate to the line, ties x, y, z (K:1762-1840);
    //   1  as 0, but no y step into j = 0 (bodyIntegralInnerWeightedFixedBC, K:2227);
    //   2  nearest candidate, ties y, x, z; no y step into j = 0 and no x or z step on
    //      j = 0 (bodyIntegralInnerSelectFixedBC, K:2628, 2675, 2722);
    //   3  the candidate with the smallest curl, read at the candidate's linear index when
    //      that index lies inside the volume and 1e10 otherwise, ties x, y, z
    //      (bodyIntegralInner(Weighted)MiniCurl, K:2869-2883).  The far candidate of an axis
    //      already at its exit coordinate (60000 cells away) may land inside the volume at an
    //      unrelated voxel, as in the reference; its coordinate test still rejects it.
    template <int RULE>
    __device__ __forceinline__ int step(const float *curl, int X, long long XY, long long V)
    {
        int i1 = il < io ? il + 1 : (il == io ? il - 60000 : il - 1);
        int j2 = jl < jo ? jl + 1 : (jl == jo ? jl - 60000 : jl - 1);
        int k3n = kl < ko ? kl + 1 : (kl == ko ? kl - 60000 : kl - 1);
        if (RULE == 3) {
            const long long q1 = (long long)i1 + (long long)jl * X + (long long)kl * XY;
            const long long q2 = (long long)il + (long long)j2 * X + (long long)kl * XY;
            const long long q3 = (long long)il + (long long)jl * X + (long long)k3n * XY;
            const float c1 = (q1 >= 0 && q1 < V) ? __ldg(curl + q1) : 1e10f;
            const float c2 = (q2 >= 0 && q2 < V) ? __ldg(curl + q2) : 1e10f;
            const float c3 = (q3 >= 0 && q3 < V) ? __ldg(curl + q3) : 1e10f;
            if (il != io && c1 <= c2 && c1 <= c3) { il = i1; return 0; }
            if (jl != jo && c2 < c1 && c2 <= c3) { jl = j2; return 1; }
            if (kl != ko && c3 < c1 && c3 < c2) { kl = k3n; return 2; }
            return -1;
        }
        float fil = (float)il, fjl = (float)jl, fkl = (float)kl;
        float fi1 = (float)i1, fj2 = (float)j2, fk3 = (float)k3n;
        float k2jl = OM_MUL(k2, fjl), k3kl = OM_MUL(k3, fkl);
        float A = OM_SUB(OM_MUL(k1, fil), xk1);
        float r1 = OM_SUB(OM_ADD(OM_SUB(OM_ADD(OM_SUB(OM_MUL(k1, fi1), xk1), k2jl), yk2), k3kl), zk3);
        float r2 = OM_SUB(OM_ADD(OM_SUB(OM_ADD(A, OM_MUL(k2, fj2)), yk2), k3kl), zk3);
        float r3 = OM_SUB(OM_ADD(OM_SUB(OM_ADD(A, k2jl), yk2), OM_MUL(k3, fk3)), zk3);
        float q1 = om_dist2(x, y, z, k1, k2, k3, r1, fi1, fjl, fkl);
        float q2 = om_dist2(x, y, z, k1, k2, k3, r2, fil, fj2, fkl);
        float q3 = om_dist2(x, y, z, k1, k2, k3, r3, fil, fjl, fk3);
        // the candidate toward the exit is always inside; the far (-60000) one never is
        if (RULE == 2) {
            if (il != io && jl != 0 && om_sqrt_lt(q1, q2) && om_sqrt_le(q1, q3)) { il = i1; return 0; }
            if (jl != jo && j2 != 0 && om_sqrt_le(q2, q1) && om_sqrt_le(q2, q3)) { jl = j2; return 1; }
            if (kl != ko && jl != 0 && om_sqrt_lt(q3, q1) && om_sqrt_lt(q3, q2)) { kl = k3n; return 2; }
            return -1;
        }
        if (il != io && om_sqrt_le(q1, q2) && om_sqrt_le(q1, q3)) { il = i1; return 0; }
        if (jl != jo && (RULE != 1 || j2 != 0) && om_sqrt_lt(q2, q1) && om_sqrt_le(q2, q3)) { jl = j2; return 1; }
        if (kl != ko && om_sqrt_lt(q3, q1) && om_sqrt_lt(q3, q2)) { kl = k3n; return 2; }
        return -1;
    }
};

// OmWalker for the rules that read no field (0, 1, 2) on grids of fewer than kFastWalkMax cells a
// side: the same operations in the same order, with the coordinates kept as floats (exact there)
// and the decisions taken without branches, which the lanes of a warp would take differently at
// almost every step.  Plain comparisons of the squared distances decide, unless two of them are
// within 2^-20 of each other: then the reference's comparisons of their roots.
// 256^3 / 642 directions: 79 -> 60 ms (OmWalker: 183 instructions per step at 160^3, issue 92 % busy).
constexpr int kFastWalkMax = 1 << 23;
struct OmFastWalker {
    float x, y, z, k1, k2, k3, xk1, yk2, zk3;
    float fi, fj, fk;  // current voxel
    float oi, oj, ok;  // exit voxel
    float si, sj, sk;  // step toward it

    __device__ __forceinline__ void init(const Grid &g, float ox, float oy, float oz, float d1, float d2, float d3, int ie,
                                         int je, int ke, int ix, int jx, int kx)
    {
        OmWalker w;
        w.init(g, ox, oy, oz, d1, d2, d3, ie, je, ke, ix, jx, kx);
        x = w.x; y = w.y; z = w.z; k1 = w.k1; k2 = w.k2; k3 = w.k3;
        xk1 = w.xk1; yk2 = w.yk2; zk3 = w.zk3;
        fi = (float)ie; fj = (float)je; fk = (float)ke;
        oi = (float)ix; oj = (float)jx; ok = (float)kx;
        si = ie < ix ? 1.0f : -1.0f; sj = je < jx ? 1.0f : -1.0f; sk = ke < kx ? 1.0f : -1.0f;
    }

    // One step: the axis moved along, or -1 when no candidate qualifies.
    template <int RULE>
    __device__ __forceinline__ int step()
    {
        static_assert(RULE != 3, "the minimum-curl walk reads a field");
        const bool mi = fi != oi, mj = fj != oj, mk = fk != ok;
        const float f1 = OM_ADD(fi, mi ? si : -60000.0f), f2 = OM_ADD(fj, mj ? sj : -60000.0f),
                    f3 = OM_ADD(fk, mk ? sk : -60000.0f);
        const float k2jl = OM_MUL(k2, fj), k3kl = OM_MUL(k3, fk);
        const float A = OM_SUB(OM_MUL(k1, fi), xk1);
        const float r1 = OM_SUB(OM_ADD(OM_SUB(OM_ADD(OM_SUB(OM_MUL(k1, f1), xk1), k2jl), yk2), k3kl), zk3);
        const float r2 = OM_SUB(OM_ADD(OM_SUB(OM_ADD(A, OM_MUL(k2, f2)), yk2), k3kl), zk3);
        const float r3 = OM_SUB(OM_ADD(OM_SUB(OM_ADD(A, k2jl), yk2), OM_MUL(k3, f3)), zk3);
        const float q1 = om_dist2(x, y, z, k1, k2, k3, r1, f1, fj, fk);
        const float q2 = om_dist2(x, y, z, k1, k2, k3, r2, fi, f2, fk);
        const float q3 = om_dist2(x, y, z, k1, k2, k3, r3, fi, fj, f3);
        constexpr float c = 9.5367431640625e-7f;  // 2^-20
        const bool near = (fabsf(OM_SUB(q1, q2)) <= OM_MUL(c, fminf(q1, q2))) | (fabsf(OM_SUB(q1, q3)) <= OM_MUL(c, fminf(q1, q3))) |
                          (fabsf(OM_SUB(q2, q3)) <= OM_MUL(c, fminf(q2, q3)));
        bool b0, b1, b2;
        if (near) {
            b0 = (RULE == 2 ? om_sqrt_lt(q1, q2) : om_sqrt_le(q1, q2)) & om_sqrt_le(q1, q3);
            b1 = (RULE == 2 ? om_sqrt_le(q2, q1) : om_sqrt_lt(q2, q1)) & om_sqrt_le(q2, q3);
            b2 = om_sqrt_lt(q3, q1) & om_sqrt_lt(q3, q2);
        } else {
            b0 = (RULE == 2 ? q1 < q2 : q1 <= q2) & (q1 <= q3);
            b1 = (RULE == 2 ? q2 <= q1 : q2 < q1) & (q2 <= q3);
            b2 = (q3 < q1) & (q3 < q2);
        }
        b0 = b0 & mi & ((RULE != 2) | (fj != 0.0f));
        b1 = b1 & mj & ((RULE == 0) | (f2 != 0.0f)) & !b0;
        b2 = b2 & mk & ((RULE != 2) | (fj != 0.0f)) & !b0 & !b1;
        fi = b0 ? f1 : fi;
        fj = b1 ? f2 : fj;
        fk = b2 ? f3 : fk;
        return b0 ? 0 : (b1 ? 1 : (b2 ? 2 : -1));
    }
};

// OmFastWalker for rule 0 behind a filter.  In exact arithmetic the squared distances from the
// line of the three candidates differ by those of D_a = 2 s_a d_a - g k_a^2, where s_a = +-1 is
// the step along axis a, d = w - g (k.w) k the deviation of the current voxel (w from the line's
// point) and g = 2 - |k|^2 (r = k.u in |u - k r|^2).  A step along b adds
// 2 [a = b] - 2 c_a c_b to D_a, c_a = s_a k_a sqrt(g), so that a step costs three multiply-adds
// where the distances themselves take 60 operations.  The smallest D decides if it is the smallest by more
// than what both roundings can amount to; else, and where a |D| is above 3, OmFastWalker decides.
//
// That margin, with u = 2^-24 and M the longest side, for |D| <= 3 (deviations of at most 2 an
// axis, candidates at most 4 from the line):
//   distances as the reference rounds them: their error along the line is of second order; across
//     it, k r (1.7 M) and x + k r (M) are rounded per axis, 3.5 u M in all, times 2 x 4: 28 u M;
//   D at the entry: w 1.7, k.w 7 and g 3 u M, so d 13 u M, D 26 u M;
//   the steps, at most 3 M of them: 14 u each (4 of the product, 5 of each of two sums): 42 u M.
// 96 u M for a D, 192 u M for two: 208 u (M + 8) is taken (the 8 for lines whose nearest point to
// the centre lies outside a small grid; 0.0033 at M = 256, where a warp of 32 lines calls the exact
// form at one step of eight).  Beyond kFilterMax cells it would at most steps.
//
// An axis at its exit coordinate has its candidate 60000 cells away, across the line by
// 60000 sqrt(1 - k_a^2), far beyond the others unless the direction is within two degrees of the
// axis: such directions take the exact form throughout.  So do those whose e = |k|^2 - 1 is above
// kUnitMax: the "distances" then hold (e r)^2 with r up to 1.7 M, whose rounding is of first order
// in r's.  Up to kUnitMax (directions in FP32, or written with five decimals) that adds
// 2 e x 1.7 M x 12 u M, 5 u M at kFilterMax, and a candidate is at most e x 1.7 M = 0.2 further away,
// which adds 2 u M.
// 256^3 / 642 directions: 60 -> 31 ms (23.6 G steps over 67 grids and sets of directions: no step
// other than the exact form's).
constexpr int kFilterMax = 2048;
struct OmFilteredWalker {
    float x, y, z, k1, k2, k3;
    float oi, oj, ok;     // exit voxel
    float si, sj, sk;     // step toward it
    float ni, nj, nk;     // steps left
    float ci, cj, ck;
    float Di, Dj, Dk;
    float margin;         // infinite: never sure

    __device__ __forceinline__ void init(const Grid &g, float ox, float oy, float oz, float d1, float d2, float d3, int ie,
                                         int je, int ke, int ix, int jx, int kx)
    {
        OmWalker w;
        w.init(g, ox, oy, oz, d1, d2, d3, ie, je, ke, ix, jx, kx);
        x = w.x; y = w.y; z = w.z; k1 = w.k1; k2 = w.k2; k3 = w.k3;
        oi = (float)ix; oj = (float)jx; ok = (float)kx;
        si = ie < ix ? 1.0f : -1.0f; sj = je < jx ? 1.0f : -1.0f; sk = ke < kx ? 1.0f : -1.0f;
        ni = fabsf(oi - (float)ie); nj = fabsf(oj - (float)je); nk = fabsf(ok - (float)ke);
        const float a = (float)ie - x, b = (float)je - y, c = (float)ke - z;
        const float e = fmaf(k3, k3, fmaf(k2, k2, fmaf(k1, k1, -1.0f)));  // |k|^2 - 1
        const float r = fmaf(k1, a, fmaf(k2, b, k3 * c)), t = fmaf(-e, r, r), f = 1.0f - e;  // g (k.w), g
        const float root = sqrtf(f);
        ci = si * k1 * root; cj = sj * k2 * root; ck = sk * k3 * root;
        Di = fmaf(2.0f * si, fmaf(-k1, t, a), -f * k1 * k1);
        Dj = fmaf(2.0f * sj, fmaf(-k2, t, b), -f * k2 * k2);
        Dk = fmaf(2.0f * sk, fmaf(-k3, t, c), -f * k3 * k3);
        const float km = fmaxf(fmaxf(fabsf(k1), fabsf(k2)), fabsf(k3));
        margin = km * km <= 0.999f && fabsf(e) <= kUnitMax ? 208.0f * 5.9604644775390625e-8f * (float)(max(max(g.X, g.Y), g.Z) + 8) : INFINITY;
    }

    // OmFastWalker's step from the current voxel.
    __device__ __forceinline__ int exact() const
    {
        OmFastWalker w;
        w.x = x; w.y = y; w.z = z; w.k1 = k1; w.k2 = k2; w.k3 = k3;
        w.xk1 = OM_MUL(x, k1); w.yk2 = OM_MUL(k2, y); w.zk3 = OM_MUL(k3, z);
        w.fi = fmaf(-si, ni, oi); w.fj = fmaf(-sj, nj, oj); w.fk = fmaf(-sk, nk, ok);
        w.oi = oi; w.oj = oj; w.ok = ok;
        w.si = si; w.sj = sj; w.sk = sk;
        return w.template step<0>();
    }

    template <int RULE>
    __device__ __forceinline__ int step()
    {
        static_assert(RULE == 0, "the other rules look at coordinates or a field");
        constexpr float kFar = 1.0e30f;
        // D, or kFar along an axis at its exit coordinate
        const float Ei = fmaxf(fmaf(-2.0f * kFar, ni, kFar), Di), Ej = fmaxf(fmaf(-2.0f * kFar, nj, kFar), Dj),
                    Ek = fmaxf(fmaf(-2.0f * kFar, nk, kFar), Dk);
        bool b0 = Ei + margin < fminf(Ej, Ek), b1 = Ej + margin < fminf(Ei, Ek), b2 = Ek + margin < fminf(Ei, Ej);
        const bool sure = (b0 | b1 | b2) & (fmaxf(fmaxf(fabsf(Di), fabsf(Dj)), fabsf(Dk)) <= 3.0f);
        if (!sure) {
            const int a = exact();
            if (a < 0) return a;
            b0 = a == 0;
            b1 = a == 1;
            b2 = a == 2;
        }
        const float c = -2.0f * (b0 ? ci : (b1 ? cj : ck));
        if (b0) { Di += 2.0f; ni -= 1.0f; }
        if (b1) { Dj += 2.0f; nj -= 1.0f; }
        if (b2) { Dk += 2.0f; nk -= 1.0f; }
        Di = fmaf(ci, c, Di);
        Dj = fmaf(cj, c, Dj);
        Dk = fmaf(ck, c, Dk);
        return b0 ? 0 : (b1 ? 1 : 2);
    }
};

}  // namespace omni3d
