// ddiv (idiv64.cuh) against the division operator, bit for bit: on the host, or on the
// device with argument "gpu".  Random significands and exponents, leading and trailing runs
// of ones and zeros, exact quotients, quotients next to a rounding midpoint, and operands
// or results outside the normal range.  Prints the number of differing quotients.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "idiv64.cuh"

using namespace g3l;

__host__ __device__ inline uint64_t mix(uint64_t x)
{   // splitmix64 (Steele, Lea & Flood 2014)
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// the two operands of test t
__host__ __device__ inline void operands(uint64_t t, double &a, double &b)
{
    const uint64_t u = mix(2 * t), v = mix(2 * t + 1), frac = 0xfffffffffffffull;
    const uint64_t sp[10] = {0, 0x8000000000000000ull, 0x7ff0000000000000ull, 0x7ff8000000000000ull, 1,
                             0x000fffffffffffffull, 0x0010000000000000ull, 0x7fefffffffffffffull,
                             0x3ff0000000000000ull, 0xbff0000000000001ull};
    const uint64_t one = 0x3ff0000000000000ull;
    const double x = of_bits((u & 0x8000000000000000ull) | ((983 + (u >> 52) % 80) << 52) | (u & frac));
    const double y = of_bits((v & 0x8000000000000000ull) | ((983 + (v >> 52) % 80) << 52) | (v & frac));
    const double z = of_bits(one | ((1ull << (u % 53)) - 1)), w = of_bits(one | (frac & ~((1ull << (v % 53)) - 1)));
    switch (t % 12) {
    case 0: case 1: case 2: a = x; b = y; break;
    case 3: a = z; b = w; break;
    case 4: a = w; b = z; break;
    case 5: a = x; b = (t & 16) ? z : w; break;
    case 6: a = of_bits(one + u % 64); b = of_bits(2 * 0x2000000000000000ull - v % 64); break;
    case 7: a = of_bits(2 * 0x2000000000000000ull - u % 64); b = of_bits(2 * 0x2000000000000000ull - v % 64); break;
    case 8: a = x * y; b = y; break;                                   // next to a representable quotient
    case 9: a = of_bits(bits_of(x * y) + (t & 64 ? 1 : -1)); b = y; break;
    case 10: a = of_bits(u); b = of_bits(v); break;                    // any bits
    default: a = (t & 32) ? of_bits(sp[u % 10]) : x; b = of_bits(sp[v % 10]); break;
    }
}

__host__ __device__ inline bool differs(uint64_t t)
{
    double a, b;
    operands(t, a, b);
    const double q = ddiv(a, b), r = a / b;
    return bits_of(q) != bits_of(r) && !(q != q && r != r);
}

__global__ void k_check(uint64_t n, unsigned long long *bad)
{
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x)
        if (differs(t)) atomicAdd(bad, 1ull);
}

int main(int argc, char **argv)
{
    const bool gpu = argc > 1 && !std::strcmp(argv[1], "gpu");
    const uint64_t n = gpu ? 400000000ull : 6000000ull;
    unsigned long long bad = 0;
    if (gpu) {
        unsigned long long *d;
        if (cudaMalloc(&d, 8) || cudaMemset(d, 0, 8)) return 2;
        k_check<<<1216, 256>>>(n, d);
        if (cudaMemcpy(&bad, d, 8, cudaMemcpyDeviceToHost)) return 2;
    } else {
        for (uint64_t t = 0; t < n; ++t) bad += differs(t);
    }
    std::printf("%llu of %llu differ\n", bad, (unsigned long long)n);
    return bad ? 1 : 0;
}
