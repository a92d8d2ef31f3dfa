// sel_bound.cuh -- comparisons that k_select settles from FP32 bounds.
//
// An integral's selection compares margins with the FP32 path's uncertainty of sums over
// its regions.  A FP64 sum of those uncertainties takes three instructions per region of a
// pipe that issues one per 64 cycles, so the sums are formed in FP32 from the operands'
// leading bits, and in FP64 only where that does not settle the comparison.
#pragma once
#include "idiv64.cuh"

namespace g3l {

constexpr int SEL_BS = 256;  // threads of a selection, over which the FP32 sums are split

// x 2^s as FP32, truncated (x >= 0); odd is set where x does not fit
__host__ __device__ __forceinline__ float f32_scaled(double x, int s, bool &odd)
{
    const uint64_t u = bits_of(x);
    const int e = (int)((u >> 52) & 0x7ffu) - 1023 + s;
    if (u == 0) return 0.f;
    if (e < -126 || e > 60 || (u >> 52) == 0) odd = true;  // out of range, or a subnormal x
    const uint32_t m = (uint32_t)(u >> 29) & 0x7fffffu;
    return e < -126 ? 0.f : f32_of_bits((uint32_t)((e < 60 ? e : 60) + 127) << 23 | m);
}

// The FP64 comparison dist <= bound from FP32 values of both, the bound a sum over R
// regions: 0 no, 1 yes, 2 not told apart (and with operands FP32 does not hold, odd).
// A thread adds n = R / SEL_BS terms, each cut to 24 bits; with the block's sum and the
// factors around it the bound is off by at most (n + 22) 2^-24 of itself to first order,
// and the margin by 2^-23.  A gap of (n + 32) 2^-23 therefore decides as FP64 does while
// that is below 1/4 (n < 2^21; beyond, nothing is settled here).  Up to 2 million regions
// it is below the 0.1% that is asked for anyway.
__host__ __device__ __forceinline__ int f32_within(float dist, float bound, int R, bool odd)
{
    const float err = ((float)(R / SEL_BS) + 33.f) * 1.1920929e-7f;  // 2^-23
    const float tol = err > 1e-3f ? err : 1e-3f, gap = dist < bound ? bound - dist : dist - bound;
    return odd || err > 0.25f || !(bound > 1e-30f) || !(bound < 1e30f) || !(gap > tol * bound)
               ? 2 : (int)(dist <= bound);
}

}  // namespace g3l
