// The launch shape of the anchor iterations (links.cuh) compiled for the host.
#include <cuda_runtime.h>

template <typename T>
static inline T __ldg(const T *p) { return *p; }
static inline float __uint_as_float(unsigned u) { float f; __builtin_memcpy(&f, &u, 4); return f; }
static inline unsigned __float_as_uint(float f) { unsigned u; __builtin_memcpy(&u, &f, 4); return u; }
static inline void __syncthreads() {}
static dim3 threadIdx, blockDim;

#include "links.cuh"

using namespace omni3d;

// {vector in shared memory, blocks, rows a warp, least rows a warp}
extern "C" void unit_iter_shape(long long n, int *out)
{
    const int kind = link_kind(n, true);
    const IterShape s = iter_shape(n, true, kind, link_split(n, true), false);
    out[0] = s.smem;
    out[1] = (int)s.blocks;
    out[2] = s.rows;
    out[3] = 32 / lanes_per_row(kind);
}
