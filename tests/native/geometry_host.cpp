// The device line geometry (geometry.cuh) compiled for the host: every operation in it is a
// single rounded FP32 operation or a fused multiply-add, so the host's results are the device's.
#include <cmath>
#include <cstring>

#include <cuda_runtime.h>

static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __fsqrt_rn(float a) { return std::sqrt(a); }
static inline float __ldg(const float *p) { return *p; }
static inline int max(int a, int b) { return a > b ? a : b; }
using std::fabs;

#include "geometry.cuh"

using namespace omni3d;

static Grid grid_of(int X, int Y, int Z)
{
    Grid g;
    std::memset(&g, 0, sizeof(g));
    g.X = X;
    g.Y = Y;
    g.Z = Z;
    g.XY = (long long)X * Y;
    g.V = g.XY * Z;
    g.cx = (float)((X - 1) / 2.0);
    g.cy = (float)((Y - 1) / 2.0);
    g.cz = (float)((Z - 1) / 2.0);
    return g;
}

extern "C" {

// Lines (n of direction k: entry and exit voxels, offsets) whose staircase by the filtered walk
// is not that of the reference's operations.
long long filtered_walk_differences(int X, int Y, int Z, const float *k, long long n, const int *inout, const float *xyz)
{
    const Grid g = grid_of(X, Y, Z);
    long long differ = 0;
    for (long long l = 0; l < n; l++) {
        const int *e = inout + 6 * l, *x = e + 3;
        const float *o = xyz + 3 * l;
        OmWalker exact;
        OmFilteredWalker fast;
        exact.init(g, o[0], o[1], o[2], k[0], k[1], k[2], e[0], e[1], e[2], x[0], x[1], x[2]);
        fast.init(g, o[0], o[1], o[2], k[0], k[1], k[2], e[0], e[1], e[2], x[0], x[1], x[2]);
        const int m = std::abs(x[0] - e[0]) + std::abs(x[1] - e[1]) + std::abs(x[2] - e[2]);
        for (int s = 0; s < m; s++) {
            const int a = exact.step<0>(nullptr, g.X, g.XY, g.V), b = fast.step<0>();
            if (a != b) {
                differ++;
                break;
            }
            if (a < 0) break;
        }
    }
    return differ;
}

// Of the n offsets, those that om_certain_miss leaves out although the line of direction k (case 7)
// through them crosses the grid.
long long wrong_misses(int X, int Y, int Z, const float *k, long long n, const float *xyz)
{
    const Grid g = grid_of(X, Y, Z);
    long long wrong = 0;
    for (long long l = 0; l < n; l++) {
        const float *o = xyz + 3 * l;
        int in[3], out[3];
        om_cross2point(g, o[0], o[1], o[2], k[0], k[1], k[2], 64, in, out);
        wrong += om_line_valid(g, in, out) && om_certain_miss(g, o[0], o[1], o[2], k[0], k[1], k[2], 64);
    }
    return wrong;
}

}  // extern "C"
