// Checks quotient_from (physics.cuh) against the division, bit for bit, for
// operands in its range: random ones, and significands next to each other,
// to powers of two and to quotients half way between two doubles.  Host code
// only (test infrastructure); exits non-zero at the first difference.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "physics.cuh"

using namespace sddc;

static std::mt19937_64 rng(2024);
static double make(uint64_t sig, int e, bool neg)
{
    const uint64_t b = ((uint64_t)neg << 63) | ((uint64_t)(e + 1023) << 52) | (sig & ((1ull << 52) - 1));
    double x;
    std::memcpy(&x, &b, 8);
    return x;
}
static bool bad(double a, double b)
{
    const double want = a / b, got = quotient_from(a, b, 1.0 / b);
    if (std::memcmp(&want, &got, 8) == 0) return false;
    std::printf("%a / %a: %a, not %a\n", a, b, got, want);
    return true;
}

int main()
{
    const uint64_t edge[] = {0, 1, 2, 3, (1ull << 52) - 1, (1ull << 52) - 2, (1ull << 52) - 3, 1ull << 51, (1ull << 51) + 1,
                             (1ull << 51) - 1, 0x5555555555555ull, 0xaaaaaaaaaaaaaull, 0x999999999999aull};
    for (uint64_t sa : edge)
        for (uint64_t sb : edge)
            for (int e : {-500, -60, -1, 0, 1, 60, 499})
                for (int f : {-500, -7, 0, 9, 499})
                    if (bad(make(sa, e, false), make(sb, f, true)) || bad(make(sa, e, true), make(sb, f, false))) return 1;
    for (double z : {0.0, -0.0})
        for (uint64_t sb : edge)
            if (bad(z, make(sb, 3, false)) || bad(z, make(sb, -3, true))) return 1;
    std::uniform_int_distribution<int> ex(-500, 499);
    for (long i = 0; i < 4000000; i++) {
        const double b = make(rng(), ex(rng), rng() & 1);
        if (bad(make(rng(), ex(rng), rng() & 1), b)) return 1;
        // a next to b times a double, or times a midpoint of two doubles
        const int eb = std::ilogb(b);
        const double c = make(rng(), 0, false), h = std::ldexp(c, 0) + std::ldexp(1.0, -53);
        double a = b * (i & 1 ? c : h);
        if (std::abs(eb) > 490) continue;
        for (int k = -2; k <= 2; k++) {
            double t = a;
            for (int m = 0; m < std::abs(k); m++) t = std::nextafter(t, k < 0 ? -1e308 : 1e308);
            if (bad(t, b)) return 1;
        }
    }
    // the range test at its ends
    auto hi = [](double x) {
        uint64_t b;
        std::memcpy(&b, &x, 8);
        return (unsigned)(b >> 32);
    };
    const double lo = std::ldexp(1.0, -500), up = std::ldexp(1.0, 500);
    if (!mid_range(hi(lo)) || mid_range(hi(std::nextafter(lo, 0.0))) || mid_range(hi(up)) ||
        !mid_range(hi(std::nextafter(up, 0.0))) || !mid_range(hi(-1.0)) || mid_range(hi(0.0)) || mid_range(hi(INFINITY)) ||
        mid_range(hi(NAN)))
        return 1;
    return 0;
}
