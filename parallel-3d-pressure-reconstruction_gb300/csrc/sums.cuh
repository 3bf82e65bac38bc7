// FP32 sums along lines and over a row's links.  The compensated ones name every rounding.
#pragma once

#include <cuda_runtime.h>

namespace omni3d {

// Kahan's sum s - c, c the error of the last addition.  It is exact to second order while the sum is
// larger than its terms; where a sum of mixed signs passes near zero a term's last bit is lost.
__device__ __forceinline__ void kahan_add(float &s, float &c, float x)
{
    const float y = __fsub_rn(x, c), t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}
// The same of w y, the product not rounded by itself.
__device__ __forceinline__ void kahan_add_product(float &s, float &c, float w, float y)
{
    const float p = __fmaf_rn(w, y, -c), t = __fadd_rn(s, p);
    c = __fsub_rn(__fsub_rn(t, s), p);
    s = t;
}
// s + e += y, e the sum of the additions' errors (Knuth's TwoSum): as a sum in twice the precision,
// whatever the terms' signs.  The anchor iteration's unit-weight rows take it: with 8 lanes a row Kahan's
// sums were off by 1.4 times as much as with 32 lanes on rows of 60 links of mixed signs (1.2e-8 against 9e-9
// of the sum of magnitudes, 1e-15 so; 128^3: 3.45 -> 3.52 ms of iterations).
__device__ __forceinline__ void two_sum_add(float &s, float &e, float y)
{
    const float t = __fadd_rn(s, y), b = __fsub_rn(t, s);
    e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(y, b)));
    s = t;
}

// (hi, lo) += (h2, l2).
__device__ __forceinline__ void add_pair(float &hi, float &lo, float h2, float l2)
{
    lo = __fadd_rn(lo, l2);
    two_sum_add(hi, lo, h2);
}

// A lane's plain sum, in four parts by the links' places i in their loads: with 8 lanes a row (16-bit
// links) as many terms in each as with 32 lanes, where one sum of all of a lane's links was less
// exact (rows of 640 and 1300 links: 5.6e-8 and 7.6e-8 of the sum off, 3.6e-8 and 3.9e-8 in parts).
struct LaneSum {
    float q[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    __device__ __forceinline__ void add(int i, float y) { q[i & 3] += y; }
    __device__ __forceinline__ float total() const { return (q[0] + q[1]) + (q[2] + q[3]); }
};

}  // namespace omni3d
