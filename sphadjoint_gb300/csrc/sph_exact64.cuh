// IEEE square root and division of doubles, rounded to nearest even, with
// integer instructions. GB300 runs double precision at 1/64 of its integer
// rate (measured 1.8 FP64 results per clock and SM, a square root or a
// division counting 7.5 of them), and the FP64 kernels are bound by that pipe.
// Both functions take a float estimate of the reciprocal (square root), refine
// it in 64-bit fixed point by Newton steps whose remainders are exact (they are
// taken modulo 2^64, where the small true remainder survives), and settle the
// last bit on the sign of the exact remainder, so the result is the correctly
// rounded one and equals the FP64 instruction's. Operands or results that are
// not normal numbers go to the FP64 operation. Measured, 152 SMs, all lanes
// busy: square root 70 -> 308 G/s, division 70 -> 228 G/s, and the FP64 pipe
// stays free meanwhile; the FP64 solve of 66k particles 7.2 -> 5.5 ms, of 2072
// particles 13.9 -> 12.0 ms (128 steps). An integer product of the same kind
// runs at the FP64 pipe's own rate (497 G/s) and was not worth it.
//
// Compiled for the device by the kernels and for the host by their test, which
// replaces the float estimates by perturbed ones.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define SPH_EX_HD __host__ __device__ __forceinline__
#else
#define SPH_EX_HD inline
#endif

namespace sphgb {

SPH_EX_HD uint64_t ex_bits(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, sizeof b);
    return b;
#endif
}
SPH_EX_HD double ex_double(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, sizeof x);
    return x;
#endif
}
SPH_EX_HD float ex_float(uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, sizeof x);
    return x;
#endif
}
SPH_EX_HD uint32_t ex_fbits(float x)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, sizeof b);
    return b;
#endif
}

// 1/sqrt(m) for m in [1, 4) and 1/m for m in [1, 2), within 2^-21.5 relative
// (the PTX approximations are within 2^-22.4 and 2^-23)
#if !defined(SPH_EX_ESTIMATES)
SPH_EX_HD float ex_rsqrt(float m)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(m));
    return y;
#else
    return 1.0f / std::sqrt(m);
#endif
}
SPH_EX_HD float ex_rcp(float m)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(m));
    return y;
#else
    return 1.0f / m;
#endif
}
#endif

constexpr uint64_t kExMant = 0x000fffffffffffffull, kExOne = 0x0010000000000000ull;

// y in (0.5, 1] as a multiple of 2^-30
SPH_EX_HD int32_t ex_fixed30(float y)
{
    const uint32_t b = ex_fbits(y);
    return (int32_t)(((b & 0x007fffffu) | 0x00800000u) << ((b >> 23) - 120u));
}

SPH_EX_HD double sqrt_rn(double x)
{
    const uint64_t b = ex_bits(x);
    const uint32_t h = (uint32_t)(b >> 32);
    if (h - 0x00100000u >= 0x7fe00000u) return sqrt(x); // 0, subnormal, negative, inf, NaN
    // x = m 2^e with e even and m in [1, 4): mant = m 2^52
    const uint32_t odd = ((h >> 20) + 1u) & 1u;
    const uint64_t mant = ((b & kExMant) | kExOne) << odd;
    const float mf = ex_float(((uint32_t)(b >> 29) & 0x007fffffu) | ((127u + odd) << 23));
    const float y = ex_rsqrt(mf);
    float sf = mf * y;
    sf = sf < 1.0f ? 1.0f : (sf > 1.99999988f ? 1.99999988f : sf);
    const int32_t Y = ex_fixed30(y > 1.0f ? 1.0f : y);
    // s0 = sqrt(m) 2^31 within 2^10; its exact remainder (units 2^-62) gives the
    // next 22 bits: the root in units of 2^-44 within a few units
    const uint32_t s0 = ((ex_fbits(sf) & 0x007fffffu) | 0x00800000u) << 8;
    const int64_t r1 = (int64_t)((mant << 10) - (uint64_t)s0 * s0); // |r1| < 2^44
    const int64_t d1 = ((int64_t)(int32_t)(r1 >> 13) * (int64_t)Y) >> 36;
    const uint64_t s1 = ((uint64_t)s0 << 13) + (uint64_t)d1;
    // its remainder (units 2^-88, below 2^49) modulo 2^64 gives the root in
    // units of 2^-53 within one
    const int64_t r2 = (int64_t)((mant << 36) - s1 * s1);
    const int64_t d2 = ((int64_t)(int32_t)(r2 >> 19) * (int64_t)Y) >> 47;
    uint64_t q = (s1 << 9) + (uint64_t)d2;
    const int64_t rem = (int64_t)((mant << 54) - q * q); // below 2^57
    q = rem < 0 ? q - 1u : q;
    q = rem > (int64_t)(2u * q) ? q + 1u : q; // q = floor(sqrt(m) 2^53)
    // a root is never halfway between two doubles: round on its last bit
    const uint64_t e = ((uint64_t)(h >> 20) + 1023u) >> 1;
    return ex_double(((q + 1u) >> 1) + ((e - 1u) << 52));
}

SPH_EX_HD double div_rn(double a, double b)
{
    const uint64_t ua = ex_bits(a), ub = ex_bits(b);
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7ffu, eb = (uint32_t)(ub >> 52) & 0x7ffu;
    int e = (int)ea - (int)eb + 1023;
    if (ea - 1u >= 0x7feu || eb - 1u >= 0x7feu || (uint32_t)(e - 2) >= 0x7fbu) return a / b;
    uint64_t A = (ua & kExMant) | kExOne;
    const uint64_t B = (ub & kExMant) | kExOne;
    const int lt = A < B ? 1 : 0; // the quotient A / B in [1, 2)
    A <<= lt;
    e -= lt;
    const float y = ex_rcp(ex_float(((uint32_t)(ub >> 29) & 0x007fffffu) | 0x3f800000u));
    const int32_t Y = ex_fixed30(y > 1.0f ? 1.0f : y);
    // digits of 21, 21 and 12 bits; each remainder is exact modulo 2^64
    const uint32_t q0 = (uint32_t)(((uint64_t)(uint32_t)(A >> 22) * (uint32_t)Y) >> 39);
    int64_t r = (int64_t)((A << 21) - (uint64_t)q0 * B); // a few B
    const int64_t q1 = ((int64_t)(int32_t)(r >> 24) * (int64_t)Y) >> 37;
    r = (int64_t)(((uint64_t)r << 21) - (uint64_t)q1 * B);
    const int64_t q2 = ((int64_t)(int32_t)(r >> 24) * (int64_t)Y) >> 46;
    r = (int64_t)(((uint64_t)r << 12) - (uint64_t)q2 * B);
    int64_t q = ((int64_t)q0 << 33) + (q1 << 12) + q2; // floor(A / B 2^54) within one
    q = r < 0 ? q - 1 : q;
    r = r < 0 ? r + (int64_t)B : r;
    const bool more = r >= (int64_t)B;
    q = more ? q + 1 : q;
    r = more ? r - (int64_t)B : r;
    // two bits below the last place, then the remainder
    const uint32_t low = (uint32_t)q & 7u;
    const uint64_t up = (low & 2u) && ((low & 5u) || r != 0) ? 1u : 0u;
    return ex_double(((ua ^ ub) & 0x8000000000000000ull) |
                     (((uint64_t)q >> 2) + up + ((uint64_t)(e - 1) << 52)));
}

SPH_EX_HD float div_rn(float a, float b) { return a / b; }

} // namespace sphgb
