// Host build of csrc/fpdiv.cuh for the CPU test: quotients of random and edge operands against
// the `/` operator, for any value within FPDIV_SEED_ULPS float ulps that the device's
// approximate reciprocal may return.
#include <stdio.h>
#include <stdlib.h>
#include <random>
#include "../cmaq_gb300/csrc/fpdiv.cuh"

static double from(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long bad = 0, covered = 0;
    // every reciprocal seed, with the lowest and the highest significand that share it
    for (uint32_t f = 0; f < 1u << 23; ++f)
        for (int low = 0; low < 2; ++low) {
            const uint64_t mb = (1ull << 52) | (uint64_t)f << 29 | (low ? (1ull << 29) - 1 : 0);
            const uint32_t y = fpdiv::recip31((uint32_t)(mb >> 32), (uint32_t)mb);
            // 2^83 / mb - 4 < y <= 2^83 / mb
            if ((unsigned __int128)y * mb > (unsigned __int128)1 << 83) ++bad;
            if ((unsigned __int128)(y + 4ull) * mb <= (unsigned __int128)1 << 83) ++bad;
        }
    if (bad) printf("%ld reciprocals out of their bounds\n", bad);
    std::mt19937_64 g(7);
    for (long i = 0; i < n; ++i) {
        uint64_t x = g(), y = g();
        const int mode = (int)(i % 8);
        if (mode < 6) {   // the normal range; modes 6 and 7: any bits
            x = (x & 0x800fffffffffffffull) | (uint64_t)(1 + g() % 2046) << 52;
            y = (y & 0x800fffffffffffffull) | (uint64_t)(1 + g() % 2046) << 52;
        }
        if (mode == 1) y |= 0xfffffff000000ull;
        if (mode == 2) y &= ~0xffffffffffull;
        if (mode == 3) x = (x & 0xfff0000000000000ull) | ((y + g() % 5 - 2) & 0xfffffffffffffull);
        if (mode == 4) { x &= ~0xffffffffffull; y |= 0xffffffull; }
        if (mode == 5 && i % 64 == 5) x &= 0x8000000000000000ull;   // +-0 / b
        const double a = from(x), b = from(y);
        bool ok;
        const double q = fpdiv::quotient(a, b, &ok);
        volatile double w = a / b;
        const double want = w;
        covered += ok;
        if (ok && memcmp(&q, &want, 8)) {
            if (bad++ < 5) printf("%a / %a = %a, not %a\n", a, b, q, want);
        }
    }
    printf("%ld quotients, %ld covered, %ld wrong\n", n, covered, bad);
    return bad != 0 || covered < n / 4;
}
