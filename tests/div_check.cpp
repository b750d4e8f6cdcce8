// mcg_div_exact against IEEE division (built and run by
// tests/test_div_exact.py with -ffp-contract=off): random operands, and
// significands at both ends of their range, with quotients near powers of two.
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "unpack.h"

static uint64_t state = 88172645463325252ull;
static uint64_t next_random() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}
static float make(uint32_t significand, int exponent) {
    const uint32_t u = ((uint32_t)(exponent + 127) << 23) | (significand & 0x7fffffu);
    float f;
    memcpy(&f, &u, 4);
    return f;
}

int main() {
    long bad = 0, used = 0;
    for (long i = 0; i < 40000000; ++i) {
        const uint64_t r = next_random();
        uint32_t a = (uint32_t)r, b = (uint32_t)(r >> 32);
        const int how = (int)(i % 12);
        if (how == 0) b |= 0x7ffff0u;
        if (how == 1) b &= 0xfu;
        if (how == 2) a |= 0x7ffff0u;
        if (how == 3) a &= 0xfu;
        if (how == 4) a = b + (uint32_t)(r >> 60);
        if (how == 5) b = 0x7ffffeu - (uint32_t)(r >> 62);
        const float d = make(b, (int)(i % 101) - 50), n = make(a, (int)(i % 101) - 52 + (int)(i % 24));
        const float y = mcg_div_reciprocal(d);
        if (y == 0.0f) continue;
        ++used;
        volatile float quotient = n / d;
        const float want = quotient, got = mcg_div_exact(n, d, y);
        uint32_t p, q;
        memcpy(&p, &want, 4);
        memcpy(&q, &got, 4);
        if (p != q && bad++ < 5) printf("%a / %a: got %a\n", n, d, got);
    }
    const float ones = make(0x7fffffu, -7);
    if (mcg_div_reciprocal(ones) != 0.0f || mcg_div_reciprocal(1e-30f) != 0.0f || mcg_div_reciprocal(0.01f) == 0.0f) ++bad;
    printf("%ld used, %ld mismatches\n", used, bad);
    return bad != 0 || used < 30000000;
}
