// 64-bit fixed-point sums of the bit-reproducible mode (params.deterministic).
//
// The default sums are FP32 atomics (voxel accumulators, operator rows' (b, c)) and operator
// rows whose entries land in the order the atomics hand out their slots, so their last bits
// depend on the order in which the GPU schedules the lines.  In the bit-reproducible mode
// every such sum is taken in 64-bit two's-complement fixed point instead: each term x is
// rounded once to round(x * s) with a power-of-two scale s, and integer addition is exact
// and order-independent, so every run gives the same bits.  The scale of each sum is set on
// the device from a bound B of its magnitude (s = 2^(62 - e) with B < 2^e, so no sum can
// overflow), and the bounds follow from the field: every contribution to a voxel is
// w (p(start) + I) with |I| <= 2 max|h| max|a| (X + Y + Z) along a staircase, a voxel
// receives at most one contribution per line through it, and w is at most 1 (plain
// methods), 1e4 / (least nonzero curl) (selected), (X + Y + Z) 1e4 / (least nonzero curl)
// (weighted) or (X + Y + Z + 1) / (least nonzero curl) (weighted, raw curl sums); a factor
// of two covers the FP32 rounding of w.  With B at most about 2^62 / s, a term is resolved to
// B * 2^-62, far below the FP32 rounding of the default sums.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace omni3d {

// Scales in Fixed::scale: voxel pn, voxel count, row b, row c, operator row sums.
enum FixSlot { kFixPn = 0, kFixCnt = 1, kFixB = 2, kFixC = 3, kFixRow = 4, kFixSlots = 5 };
// Float bits in Fixed::bits: max |a|, least nonzero |curl|, max |p| of the operator values,
// max |p| of the volume a full sweep reads.
enum FixBits { kBitsA = 0, kBitsC = 1, kBitsRow = 2, kBitsVol = 3, kBitsSlots = 4 };

// Fixed-point sums of a voxel.  In memory the sums of all copies' pn come first, then those of
// the counts: a warp's additions to one of them are then 4 to a 32-byte sector, which is what the
// L2 takes at a time, and not 2.
struct Fix2 {
    long long pn, cnt;
};
struct FixSums {
    const long long *pn, *cnt;
};

__device__ __forceinline__ void fold_add(Fix2 &a, const Fix2 &b)  // exact in any order
{
    a.pn += b.pn;
    a.cnt += b.cnt;
}
__device__ __forceinline__ Fix2 fold_load(const FixSums &in, size_t i) { return Fix2{in.pn[i], in.cnt[i]}; }

// A scale 2^k as two FP32 factors.  x * lo * hi is the x * 2^k of FP64 wherever its rounding to
// an integer is not 0: the first factor takes k as far as FP32's normal range goes, so only a
// product that is far below 1 loses bits.  FP64 arithmetic and conversions run at 2 lanes per
// cycle and SM here: they were 14 of the 16.8 ms of a selected 112^3 sweep.
struct FixScale {
    float lo, hi;
};
__device__ __forceinline__ FixScale fix_scale(double s)
{
    const uint32_t up = (uint32_t)__double2hiint(s);
    if (up == 0u) return FixScale{0.0f, 1.0f};  // no scale holds the sum
    auto pow2 = [](int e) { return __uint_as_float((uint32_t)(e + 127) << 23); };
    const int k = (int)(up >> 20) - 1023, a = min(max(k, -126), 127);
    return FixScale{pow2(a), pow2(min(max(k - a, -126), 127))};
}

__device__ __forceinline__ unsigned long long fix_term(float x, const FixScale &s)
{
    return (unsigned long long)__float2ll_rn(x * s.lo * s.hi);
}

__device__ __forceinline__ void fix_add(long long *a, float x, const FixScale &s)
{
    // stated as a reduction: of an address that the compiler cannot tell to be global it makes an
    // atomic with a result (112^3 selected sweep: 8.9 -> 6.3 ms)
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(a)), "l"(fix_term(x, s)) : "memory");
}

}  // namespace omni3d
