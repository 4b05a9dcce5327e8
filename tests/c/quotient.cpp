// The replica engine's quotients (rmpcdmd_b200/csrc/quotient.cuh) against the
// division, bit for bit.  Prints the number of pairs tried; exits 1 at the first
// that differs.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline
#include "quotient.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t next()
{
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state * 2685821657736338717ull;
}
static double make(uint64_t sign, int exponent, uint64_t mantissa)
{
    const uint64_t w = (sign << 63) | ((uint64_t)(exponent + 1023) << 52) | (mantissa & ((1ull << 52) - 1));
    double x;
    memcpy(&x, &w, 8);
    return x;
}
static uint64_t mantissa()
{
    const uint64_t r = next(), all = (1ull << 52) - 1;
    switch (r % 6) {
    case 0: return all;                              // ones
    case 1: return all ^ (1ull << (next() % 52));    // ones but for one bit
    case 2: return 1ull << (next() % 52);            // one bit
    case 3: return all << (next() % 52);             // ones, then zeros
    default: return next() & all;
    }
}
static long long tried = 0;
static bool same(double a, const rmpcd::Quotient &q)
{
    const double x = q.of(a), y = a / q.b;
    tried++;
    if (memcmp(&x, &y, 8) == 0 || (x != x && y != y)) return true;
    printf("%a / %a: %a, not %a\n", a, q.b, x, y);
    return false;
}

int main()
{
    std::vector<double> special = {0.0, 1.0, 2.0, 3.0, 1e-100, 1e100, 1e-180, 1e180, 33.510321638291124, 1e-320, 5e-324};
    special.push_back(std::numeric_limits<double>::infinity());
    special.push_back(std::numeric_limits<double>::quiet_NaN());
    special.push_back(std::numeric_limits<double>::max());
    special.push_back(std::numeric_limits<double>::min());
    // both sides of the guards (10^100 and 10^180 lie at 2^332 and 2^598)
    for (int e : {-333, -332, 331, 332, 333, -599, -598, -597, 597, 598, 599})
        for (int k = 0; k < 4; k++) special.push_back(make(0, e, mantissa()));
    rmpcd::Quotient q;
    for (double b : special)
        for (int s = 0; s < 2; s++) {
            q.set(s ? -b : b);
            for (double a : special)
                if (!same(a, q) || !same(-a, q)) return 1;
            for (int k = 0; k < 200; k++)
                if (!same(make(next() & 1, (int)(next() % 2046) - 1022, mantissa()), q)) return 1;
        }
    for (int i = 0; i < 200000; i++) {
        // thermal values in nine cases of ten, the guarded range in one
        const int r = i % 10 ? 40 : 700;
        q.set(make(next() & 1, (int)(next() % r) - r / 2, mantissa()));
        for (int k = 0; k < 20; k++)
            if (!same(make(next() & 1, (int)(next() % r) - r / 2, mantissa()), q)) return 1;
    }
    printf("%lld\n", tried);
    return 0;
}
