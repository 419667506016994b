// Checks quotient() (pbrt-v2_gb300/csrc/pbg_quotient.h) against the IEEE
// division on seeded random and adversarial pairs: equal from 2^-100 up, within
// max(2^-23 of the quotient, 2^-149) below.  Prints "cases unequal outside";
// exit status 1 where one is.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../pbrt-v2_gb300/csrc/pbg_quotient.h"

static uint64_t state = 0x9e3779b97f4a7c15ull;
static uint64_t next_u64() {  // splitmix64
    uint64_t z = (state += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
static float from_bits(uint32_t b) {
    float f;
    std::memcpy(&f, &b, 4);
    return f;
}
// a mantissa: any, or near an end or the middle
static uint32_t mantissa() {
    const uint64_t r = next_u64();
    const uint32_t m = (uint32_t)(r >> 8) & 0x7fffffu;
    switch (r & 3) {
        case 0: return m & 15u;
        case 1: return 0x7fffffu - (m & 15u);
        case 2: return (0x400000u + (m & 31u) - 16u) & 0x7fffffu;
        default: return m;
    }
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long unequal = 0, outside = 0;
    for (long k = 0; k < n; ++k) {
        float s = from_bits(((127u + (uint32_t)(next_u64() % 8)) << 23) | mantissa());  // [1, 256)
        if (k % 1000 == 0) s = 256.f;
        float e = k % 3 == 0 ? from_bits((uint32_t)(next_u64() % (28u << 23)))          // [0, 2^-99)
                             : from_bits(((27u + (uint32_t)(next_u64() % 100)) << 23) | mantissa());  // [2^-100, 1)
        if (k % 997 == 0) e = 1.f;
        if (k % 5 == 0 && e >= 0x1p-60f) e = std::fmin(1.f, std::nextafter((float)(std::floor(e * 0x1p30f) * 0x1p-30) * s, 2.f));  // near exact quotients
        const float got = pbg::quotient(e, s, 1.f / s), want = e / s;
        if (e >= 0x1p-100f) {
            if (std::memcmp(&got, &want, 4) != 0) ++unequal;
        } else if (!(std::fabs((double)got - (double)want) <= std::fmax(0x1p-23 * (double)want, 0x1p-149))) {
            ++outside;
        }
    }
    printf("%ld %ld %ld\n", n, unequal, outside);
    return unequal || outside;
}
