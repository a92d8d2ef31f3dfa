// idiv64.cuh -- IEEE FP64 division on the integer pipes.
//
// GB300's FP64 pipe takes one warp instruction per 64 cycles and SM quarter, and a division
// is eight or more of them (over 500 cycles of the pipe), while the integer and FP32 pipes
// of the FP64-bound kernels idle.  ddiv(a, b) forms the correctly rounded quotient (round to
// nearest even, so the bits of a / b) from integer arithmetic on the significands: a 32-bit
// fixed-point reciprocal of the divisor (FP32 reciprocal, one Newton step), two quotient
// digits of ~30 and ~27 bits with exact remainders mod 2^64, one correction of the last
// digit, and the rounding decided by the exact remainder: about 75 integer instructions.
// Operands or results outside the normal range take the hardware division.
#pragma once
#include <cstdint>
#ifndef __CUDA_ARCH__
#include <cstring>
#endif

namespace g3l {

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t mulhi_u32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
__device__ __forceinline__ int32_t mulhi_s32(int32_t a, int32_t b) { return __mulhi(a, b); }
__device__ __forceinline__ uint64_t bits_of(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double of_bits(uint64_t u) { return __longlong_as_double((long long)u); }
// 1 / x for x in [1, 2), relative error below 2^-22
__device__ __forceinline__ float recip_f32(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float f32_of_bits(uint32_t u) { return __uint_as_float(u); }
__device__ __forceinline__ uint32_t bits_of_f32(float f) { return __float_as_uint(f); }
#else
inline uint32_t mulhi_u32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline int32_t mulhi_s32(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
inline uint64_t bits_of(double x)
{
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
}
inline double of_bits(uint64_t u)
{
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}
inline float recip_f32(float x) { return 1.0f / x; }
inline float f32_of_bits(uint32_t u)
{
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
inline uint32_t bits_of_f32(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
#endif

// 2^63 / b1 for the divisor's leading 32 bits b1 (top bit set), rounded down, within a few
// units (a Newton step's result does not exceed the reciprocal, so 2^32 is not reached)
__host__ __device__ __forceinline__ uint32_t recip_u32(uint32_t b1)
{
    // y = 1 / (b1 2^-31) in [0.5, 1), and y 2^32 (exponent field 126)
    const float y = recip_f32(f32_of_bits(0x3f800000u | ((b1 >> 8) & 0x7fffffu)));
    uint32_t yb = bits_of_f32(y);
    yb = yb < 0x3f000000u ? 0x3f000000u : (yb > 0x3f7fffffu ? 0x3f7fffffu : yb);
    const uint32_t r0 = ((yb & 0x7fffffu) | 0x800000u) << 8;
    // Newton: r1 = r0 + r0 (2^63 - b1 r0) / 2^63
    const int64_t e = (int64_t)(0x8000000000000000ull - (uint64_t)b1 * r0);
    const int32_t e1 = (int32_t)(e >> 12);
    // r0 may exceed 2^31: e1 r0 as e1 (r0 - 2^32) + e1 2^32 in signed arithmetic
    const int32_t h = mulhi_s32(e1, (int32_t)r0) + e1;
    return r0 + (uint32_t)(h >> 19);
}

__host__ __device__ __forceinline__ double ddiv(double a, double b)
{
    const uint64_t ua = bits_of(a), ub = bits_of(b);
    const uint32_t ah = (uint32_t)(ua >> 32), bh = (uint32_t)(ub >> 32);
    const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
    // significands (53 bits)
    const uint64_t ma = ((uint64_t)((ah & 0xfffffu) | 0x100000u) << 32) | (uint32_t)ua;
    const uint64_t mb = ((uint64_t)((bh & 0xfffffu) | 0x100000u) << 32) | (uint32_t)ub;
    const uint32_t a1 = (uint32_t)(ma >> 21), b1 = (uint32_t)(mb >> 21);
    const uint32_t r = recip_u32(b1);
    // first digit: (ma / mb) 2^31, at most a few units too small
    const uint32_t q1 = mulhi_u32(a1, r) - 6u;
    const uint64_t rem1 = (ma << 31) - (uint64_t)q1 * mb;  // in [0, 16 mb)
    // second digit: (rem1 / mb) 2^27, within a few units
    const uint32_t q2 = mulhi_u32((uint32_t)(rem1 >> 25), r);
    uint64_t q = ((uint64_t)q1 << 27) + q2;
    int64_t rem = (int64_t)((rem1 << 27) - (uint64_t)q2 * mb);  // |rem| < 16 mb
    // units the digit is off by
    {
        const int32_t c = mulhi_s32((int32_t)(rem >> 27), (int32_t)(r >> 1)) >> 24;
        q += (int64_t)c;
        rem -= (int64_t)c * (int64_t)mb;
    }
    if (rem < 0) {
        rem += (int64_t)mb;
        --q;
    }
    if (rem >= (int64_t)mb) {
        rem -= (int64_t)mb;
        ++q;
    }
    // q = floor(2^58 ma / mb) in (2^57, 2^59); round to 53 bits
    const uint32_t big = (uint32_t)(q >> 58);  // 1: 59 bits (ma >= mb), 0: 58 bits
    const uint32_t n = 5u + big;
    q |= rem != 0 ? 1u : 0u;  // sticky (the lowest of at least 5 extra bits)
    const uint64_t half = (uint64_t)(1u << (n - 1u)) - 1u + ((q >> n) & 1u);
    const uint64_t m = (q + half) >> n;  // 53 bits, or 2^53 after a carry
    const int32_t e = (int32_t)ea - (int32_t)eb + 1022 + (int32_t)big;
    // out of the normal range (or zero, infinite, NaN operands): the hardware's division
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || (uint32_t)(e - 1) >= 2045u) return a / b;
    // the significand's leading bit adds one to the exponent field
    return of_bits((ua ^ ub) & 0x8000000000000000ull | (((uint64_t)(uint32_t)(e - 1) << 52) + m));
}

}  // namespace g3l
