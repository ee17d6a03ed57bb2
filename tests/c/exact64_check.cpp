// Integer-path double operations (csrc/exact64.cuh) against the host's own,
// bit for bit; returns the number of differing results.
#include <random>

static int seed_move();  // units in the last place added to each FP32 seed
#define MLAU_X64_SEED_ULPS seed_move()
#include "exact64.cuh"

static int g_move = 0;
static std::mt19937_64 g_rng;
static int seed_move() { return g_move ? (int)(g_rng() % (2 * g_move + 1)) - g_move : 0; }

// kind 0: exponents near 1; 1: significands with long runs of zeros or ones;
// 2: every exponent, subnormals, infinities and NaN included
static double draw(int kind)
{
    uint64_t m = g_rng() & 0xfffffffffffffull, e;
    if (kind == 0) e = 1003 + g_rng() % 41;
    else if (kind == 1) {
        e = 1022 + g_rng() % 3;
        const int k = (int)(g_rng() % 53);
        m = (g_rng() & 1) ? (m >> k) << k : m | ((1ull << k) - 1);
        if (g_rng() & 1) m ^= 1ull << (g_rng() % 52);
        m &= 0xfffffffffffffull;
    } else e = g_rng() % 2048;
    const uint64_t u = ((g_rng() & 1) << 63) | (e << 52) | m;
    double x;
    memcpy(&x, &u, 8);
    return x;
}

static bool same(double a, double b) { return memcmp(&a, &b, 8) == 0 || (a != a && b != b); }

extern "C" long exact64_check(int kind, int ulps, long n, long seed)
{
    using namespace mlau;
    g_rng.seed((uint64_t)seed);
    g_move = ulps;
    long bad = 0;
    const double edge[] = {0.0, -0.0, 1.0, -1.0, 2.0, 3.0, 0x1.fffffffffffffp0, INFINITY, NAN,
                           0x1p-255, 0x1.fffffffffffffp256, 0x1p257, 0x1p-1074, 0x1p1023};
    const long ne = (long)(sizeof(edge) / sizeof(edge[0]));
    for (long i = 0; i < n; i++) {
        const double a = i < ne * ne ? edge[i / ne] : draw(kind);
        const double b = i < ne * ne ? edge[i % ne] : draw(kind);
        bad += !same(x64::rcp(a), 1.0 / a);
        bad += !same(x64::half_over(a), 0.5 / a);
        bad += !same(x64::div(a, b), a / b);
        bad += !same(x64::div24(a), a / 24.0);
        bad += !same(x64::sqrt(a), std::sqrt(a));
        if (!x64::off_wide(a)) {
            uint32_t out = 0;
            const double q = x64::sqr(a, out);
            if (!out) bad += !same(q, a * a);
            bad += !same(x64::mulk<3>(a), 3.0 * a) + !same(x64::mulk<15>(a), 15.0 * a) +
                   !same(x64::mulk<7>(a), 7.0 * a) + !same(x64::mulk<9>(a), 9.0 * a) +
                   !same(x64::mulk<11>(a), 11.0 * a) + !same(x64::mulk<117>(a), 117.0 * a) + !same(x64::scale<-3>(a), 0.125 * a);
            if (!x64::off_wide(b)) {
                out = 0;
                const double p = x64::mul(a, b, out);
                if (!out) bad += !same(p, a * b);
                uint32_t nz = 0;
                const double r = x64::mul_nz(a, b, nz), s2 = x64::sqr_nz(a, nz);
                if (!nz) bad += !same(r, a * b) + !same(s2, a * a);
                if (a == 0.0 || b == 0.0) bad += nz == 0;
                if (out) bad += a * b == 0.0 || (std::fabs(a * b) > 0x1p-500 && std::fabs(a * b) < 0x1p500);
            }
        }
    }
    return bad;
}
