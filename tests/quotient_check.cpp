// quotient (velox_b200/csrc/quotient.cuh) against IEEE division on the host:
// random operands over both ranges, the ranges' ends, mantissas of all ones and
// zeros, and the operands that must be refused. Prints the number of operands
// that failed.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

static uint32_t bitsOf(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
static float ofBits(uint32_t u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
#define VXD inline
#define __fmaf_rn(a, b, c) std::fmaf((a), (b), (c))
#define __float_as_uint(f) bitsOf(f)
#include "quotient.cuh"

using namespace vxb;

int main() {
    std::mt19937 rng(1);
    long bad = 0;
    auto check = [&](float x, float k) {
        if (!quotientBase(k) || !quotientRange(x)) {
            ++bad;
            return;
        }
        const float got = quotient(x, k, 1.0f / k), want = x / k;
        if (x == 0.0f ? got != 0.0f : bitsOf(got) != bitsOf(want)) ++bad;
    };
    auto mantissa = [&]() -> uint32_t {
        const uint32_t r = rng();
        if ((r >> 28) == 0) return 0x7fffffu - (r & 3u);
        if ((r >> 28) == 1) return r & 3u;
        return r & 0x7fffffu;
    };
    auto number = [&](int lo, int hi) {  // exponents lo .. hi
        const uint32_t e = 127 + lo + (int)(rng() % (uint32_t)(hi - lo + 1));
        return ofBits((rng() & 0x80000000u) | e << 23 | mantissa());
    };
    for (long i = 0; i < 20000000; ++i) {
        const float k = std::fabs(number(-29, 29));
        if (!quotientBase(k)) continue;  // (the ends are below)
        check(number(-80, 59), k);
        const float x = number(-40, 25) * k;  // the quotient lies next to a float
        check(x, k);
    }
    const float low = ofBits(47u << 23), high = ofBits(187u << 23);  // 2^-80, 2^60
    std::vector<float> bases{9.5e-10f, 1.0e9f, ofBits(bitsOf(1.0f) | 0x7fffffu), 1.0f};
    for (float k : bases)
        for (float x : {0.0f, -0.0f, low, -low, high, -high, 1.0f, -1.0f, 1e-20f, 3e15f}) check(x, k);
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    for (float x : {ofBits(bitsOf(low) - 1), ofBits(bitsOf(high) + 1), ofBits(1u), 1e-30f, 1e30f, inf, -inf, nan})
        if (quotientRange(x) || quotientRange(-x)) ++bad;
    for (float k : {0.0f, -1.0f, 9.4e-10f, 1.1e9f, inf, nan})
        if (quotientBase(k)) ++bad;
    std::printf("%ld\n", bad);
    return bad != 0;
}
