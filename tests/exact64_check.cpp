// The integer square root and division (sph_exact64.cuh) against the machine's
// IEEE operations, with float estimates off by up to 2^-21.5 in either
// direction, on random patterns, near exact roots and quotients, and on
// operands that are not normal. Prints the counts; exits 1 on any difference.
#include <cfenv>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#define SPH_EX_ESTIMATES
static double g_off = 0.0;
namespace sphgb {
inline float ex_rsqrt(float m) { return (float)((1.0 + g_off) / std::sqrt((double)m)); }
inline float ex_rcp(float m) { return (float)((1.0 + g_off) / (double)m); }
}
#include "sph_exact64.cuh"

using namespace sphgb;

static long g_bad = 0, g_checked = 0;

static bool same(double a, double b) { return ex_bits(a) == ex_bits(b) || (a != a && b != b); }
static void root(double x)
{
    ++g_checked;
    if (!same(sqrt_rn(x), std::sqrt(x)) && g_bad++ < 5) std::printf("sqrt %a off %g\n", x, g_off);
}
static void quot(double a, double b)
{
    ++g_checked;
    if (!same(div_rn(a, b), a / b) && g_bad++ < 5) std::printf("%a / %a off %g\n", a, b, g_off);
}

int main()
{
    std::mt19937_64 g(3);
    const double offs[] = {0.0, 3.3e-7, -3.3e-7, 1.7e-7, -1.7e-7};
    for (double off : offs) {
        g_off = off;
        for (long t = 0; t < 600000; ++t) {
            const uint64_t u = g(), v = g();
            root(ex_double(u));
            quot(ex_double(u), ex_double(v));
            const double a = ex_double((u & kExMant) | (1023ull << 52)); // [1, 2)
            const double b = ex_double((v & kExMant) | (1023ull << 52));
            root(a);
            root(2.0 * a);
            quot(a, b);
            // exact roots, exact quotients and their neighbours
            const double s = ex_double(ex_bits(a) & ~((1ull << (20 + v % 33)) - 1));
            for (int d = -1; d <= 1; ++d) {
                root(ex_double(ex_bits(s * s) + (uint64_t)(int64_t)d));
                quot(ex_double(ex_bits(s * b) + (uint64_t)(int64_t)d), b);
                quot(a, ex_double(ex_bits(a) + (uint64_t)(int64_t)d));
            }
        }
        for (int d = 0; d < 2000; ++d) { // the ends of the significand's range
            const double lo = ex_double((1023ull << 52) + (uint64_t)d);
            const double hi = ex_double((1024ull << 52) - 1 - (uint64_t)d);
            root(lo), root(hi), root(2 * lo), root(2 * hi);
            quot(lo, hi), quot(hi, lo), quot(1.0, hi), quot(1.0, lo), quot(hi, hi), quot(lo, lo);
        }
        const double odd[] = {0.0, -0.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324, 1e-310,
                              2.2250738585072014e-308, 1.7976931348623157e308, 1e-300, 1e300};
        for (double a : odd) {
            root(a);
            for (double b : odd) quot(a, b), quot(-a, b);
        }
    }
    std::printf("checked %ld, mismatches %ld\n", g_checked, g_bad);
    return g_bad ? 1 : 0;
}
