// The rows' sums (sums.cuh) compiled for the host: rows of n unit links over `lanes` lanes, each load of
// `per` links to the next lane, the lane sums in a butterfly.
#include <cmath>

#include <cuda_runtime.h>

static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }

#include "sums.cuh"

using namespace omni3d;

// A row of the operator with unit weights.
extern "C" double unit_row_sum(const float *x, long long n, int lanes, int per)
{
    float h[32] = {}, l[32] = {};
    for (long long i = 0; i < n; i++) two_sum_add(h[i / per % lanes], l[i / per % lanes], x[i]);
    for (int o = lanes / 2; o; o >>= 1)
        for (int a = 0; a < o; a++) add_pair(h[a], l[a], h[a + o], l[a + o]);
    return (double)h[0] + (double)l[0];
}

// A row of the transposed operator.
extern "C" float adjoint_row_sum(const float *x, long long n, int lanes, int per)
{
    LaneSum q[32];
    for (long long i = 0; i < n; i++) q[i / per % lanes].add((int)(i % per), x[i]);
    float s[32];
    for (int a = 0; a < lanes; a++) s[a] = q[a].total();
    for (int o = lanes / 2; o; o >>= 1)
        for (int a = 0; a < o; a++) s[a] += s[a + o];
    return s[0];
}
