// csrc/emf_diff.cuh against the same expression in doubles, bit for bit
// (zeros of either sign equal); returns the number of differing results.
#include <random>

#include "emf_diff.cuh"

extern "C" long emf_diff_check(int kind, long n, long seed)
{
    std::mt19937_64 g((uint64_t)seed);
    long bad = 0;
    for (long k = 0; k < n; k++) {
        float e[4];
        for (int m = 0; m < 4; m++) {
            uint32_t ex, mant = (uint32_t)(g() & 0x7fffff);
            if (kind == 0) ex = 120 + g() % 8;              // smooth
            else if (kind == 1) ex = 100 + g() % 26;        // around the window's edge
            else if (kind == 2) ex = g() % 256;             // everything, infinities and NaN too
            else ex = 130, mant = (1u << 22) | (g() & 63);  // cancelling
            uint32_t u = (uint32_t)((g() & 1) << 31) | (ex << 23) | mant;
            if (g() % 9 == 0) u &= 0x80000000u;
            if (k % 11 == 0 && m) memcpy(&u, &e[0], 4);
            memcpy(&e[m], &u, 4);
        }
        const double d1 = (double)e[2] - (double)e[1], d2 = (double)e[3] - (double)e[0];
        const double p = 27.0 * d1, ref = p - d2, got = mlau::emf_diff4(e);
        bad += memcmp(&ref, &got, 8) != 0 && ref != got && !(ref != ref && got != got);
    }
    return bad;
}
