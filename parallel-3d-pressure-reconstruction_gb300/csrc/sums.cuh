// FP32 sums of a row's links.
#pragma once

#include <cuda_runtime.h>

namespace omni3d {

// A lane's plain sum, in four parts by the links' places i in their loads: with 8 lanes a row (16-bit
// links) as many terms in each as with 32 lanes, where one sum of all of a lane's links was less
// exact (rows of 640 and 1300 links: 5.6e-8 and 7.6e-8 of the sum off, 3.6e-8 and 3.9e-8 in parts).
struct LaneSum {
    float q[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    __device__ __forceinline__ void add(int i, float y) { q[i & 3] += y; }
    __device__ __forceinline__ float total() const { return (q[0] + q[1]) + (q[2] + q[3]); }
};

}  // namespace omni3d
