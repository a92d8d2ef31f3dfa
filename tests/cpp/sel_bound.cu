// Comparisons settled from FP32 bounds (sel_bound.cuh) against FP64 ones, on the host: the
// sums are formed as k_select forms them (SEL_BS threads, strided, one fused multiply-add per
// region, then the threads' sums), for region counts up to 2^26 and for terms whose rounding
// errors all go one way.  Prints the number of wrong decisions and exits 1 if there is any.
#include <cmath>
#include <cstdio>
#include <vector>

#include "sel_bound.cuh"

using namespace g3l;

static long long wrong = 0, settled = 0, asked = 0;

// error e(j) and relative bound u(j) of region j under pattern pat
static double err_of(int pat, long long j)
{
    switch (pat) {
    case 0: return j < SEL_BS ? 1.0 : 0.999 * std::ldexp(1.0, -25);  // each is lost beside its thread's first
    case 1: return j < SEL_BS ? 1.0 : 1.4 * std::ldexp(1.0, -25);    // each is rounded up
    case 2: return 1.0 + std::ldexp((double)((j * 2654435761ll) & 0xffffff), -24);
    default: return std::ldexp(1.0, -(int)((j * 40503) & 31));
    }
}

static void one(int pat, long long R)
{
    // the FP64 form's sum, and the FP32 one from leading bits, relative to 2^0
    std::vector<float> part(SEL_BS, 0.f);
    std::vector<double> part64(SEL_BS, 0.0);
    bool odd = false;
    const float u = 0.75f;
    for (long long j = 0; j < R; ++j) {
        const double e = err_of(pat, j);
        part[j % SEL_BS] = std::fmaf(f32_scaled(e, 0, odd), u, part[j % SEL_BS]);
        part64[j % SEL_BS] += e * (double)u;
    }
    float b32 = 0.f;
    double b64 = 0;
    for (int t = 0; t < SEL_BS; ++t) {
        b32 += part[t];
        b64 += part64[t];
    }
    // margins on both sides of the bound
    for (int k = -170; k <= 170; ++k) {
        const double dist = b64 * (1 + (k < 0 ? -1 : 1) * std::pow(2.0, -std::abs(k) / 16.0) * 0.5);
        bool od = odd;
        const float d32 = f32_scaled(dist, 0, od);
        const int w = f32_within(d32, b32, (int)R, od);
        ++asked;
        if (w == 2) continue;
        ++settled;
        wrong += w != (dist <= b64);
    }
}

// f32_scaled: what it does not flag is x 2^s, cut to 24 bits
static void scaled()
{
    const double x[] = {4.9406564584124654e-324, 1e-320, 1e-310, 2.2250738585072009e-308,
                        2.2250738585072014e-308, 1e-300, 1e-100, 1.0, 1.5, 1e18, 1e300};
    for (double v : x)
        for (int s = -1100; s <= 1100; ++s) {
            bool odd = false;
            const double got = f32_scaled(v, s, odd), want = std::ldexp(v, s);
            if (!odd && !(got <= want && got >= want * (1 - std::ldexp(1.0, -23)))) ++wrong;
        }
}

int main()
{
    scaled();
    const long long R[] = {1, 31, 257, 4099, 100003, 1ll << 20, 1ll << 22, (1ll << 23) + 5, 1ll << 24, 1ll << 26};
    for (long long r : R)
        for (int pat = 0; pat < 4; ++pat) one(pat, r);
    std::printf("%lld wrong of %lld settled of %lld\n", wrong, settled, asked);
    return wrong || settled < asked / 4 ? 1 : 0;
}
