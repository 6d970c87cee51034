// Magnitude and shift of a fixed-point contribution (fixed_parts) against the
// 128-bit integers of fixed_of, for FP32 and FP64 patterns over the grid's
// scales, and the 26-bit limbs of a warp's signed sum against the 128-bit
// sum. Prints the counts; exits 1 on any difference.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "sph_fixed.cuh"

using namespace sphgb;

static long g_bad = 0, g_checked = 0;

template <typename C, typename U> static unsigned __int128 value(C c, int S, U &M, int &k)
{
    if (!fixed_parts(c, S, M, k)) return 0;
    unsigned __int128 v = (unsigned __int128)M << k;
    return c < 0 ? ~v + 1 : v;
}

template <typename C, typename U> static void check(C c, int S)
{
    U M;
    int k;
    Fixed128 b{0, 0};
    if (!fixed_of((double)c, S, b)) b = Fixed128{0, 0};
    const unsigned __int128 v = value(c, S, M, k);
    ++g_checked;
    if ((unsigned long long)v != b.lo || (unsigned long long)(v >> 64) != b.hi) ++g_bad;
}

template <typename C, typename U> static void sweep(std::mt19937_64 &g, long n, int lo, int hi)
{
    for (long t = 0; t < n; ++t) {
        const double m = 1.0 + (double)(g() >> 12) * 0x1p-52;
        const C c = (C)std::ldexp(g() & 1 ? m : -m, lo + (int)(g() % (uint64_t)(hi - lo)));
        if (c == 0 || !std::isfinite((double)c)) continue;
        const int top = std::ilogb((double)c) + 1;
        const int S = -top + (int)(g() % 180) - 60; // |c| 2^S from 2^-60 to 2^120
        check<C, U>(c, S);
    }
}

// 32 contributions as limbs relative to the smallest shift, as the kernel adds them
template <typename C, typename U> static void warp(std::mt19937_64 &g, int spread)
{
    unsigned __int128 want = 0, got = 0;
    U M[32];
    int k[32], kmin = 1 << 20, kmax = 0;
    bool neg[32], any = false;
    for (int l = 0; l < 32; ++l) {
        const double m = 1.0 + (double)(g() >> 12) * 0x1p-52;
        const C c = (C)std::ldexp(g() & 1 ? m : -m, -(int)(g() % (uint64_t)spread));
        neg[l] = c < 0;
        want += value(c, 110, M[l], k[l]);
        if (!M[l]) continue;
        any = true;
        kmin = k[l] < kmin ? k[l] : kmin;
        kmax = k[l] > kmax ? k[l] : kmax;
    }
    if (!any) return;
    const int bits = kmax - kmin + (sizeof(C) == 4 ? 25 : 54);
    for (int j = 0; 26 * j < bits; ++j) {
        long long s = 0;
        for (int l = 0; l < 32; ++l) {
            const int t = 26 * j - (k[l] - kmin);
            uint64_t b = t >= 64 ? 0 : t >= 0 ? (uint64_t)M[l] >> t : -t < 32 ? (uint64_t)M[l] << -t : 0;
            b &= (1u << 26) - 1u;
            s += neg[l] ? -(long long)b : (long long)b;
        }
        if (s >= (1ll << 31) || s < -(1ll << 31)) ++g_bad; // the 32-bit warp sum holds it
        got += (unsigned __int128)(__int128)s << (26 * j);
    }
    ++g_checked;
    if ((got << kmin) != want) ++g_bad;
}

int main()
{
    std::mt19937_64 g(7);
    sweep<float, uint32_t>(g, 1000000, -149, 100);
    sweep<double, uint64_t>(g, 1000000, -1074, 900);
    for (int S = -60; S < 4; ++S) // halfway cases of the rounding
        for (uint64_t m = 1; m < 400; ++m) {
            check<double, uint64_t>(std::ldexp((double)m, 20), S);
            check<double, uint64_t>(-std::ldexp((double)(2 * m + 1), 20), S);
            check<float, uint32_t>((float)std::ldexp((double)(2 * m + 1), 20), S);
        }
    for (int t = 0; t < 20000; ++t) {
        warp<float, uint32_t>(g, 1 + t % 100);
        warp<double, uint64_t>(g, 1 + t % 100);
    }
    std::printf("checked %ld, mismatches %ld\n", g_checked, g_bad);
    return g_bad ? 1 : 0;
}
