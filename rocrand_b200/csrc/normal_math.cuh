// normal_math.cuh -- single-precision Box-Muller on two units at a time.
//
// A unit is a uniform u in (0, 1] and an angle a in [0, 2 pi], both floats; its results are
// sqrt(-2 log u) sin a and sqrt(-2 log u) cos a.  The floating-point steps run on the two units'
// values packed in one 64-bit register pair (add / mul / fma .rn.f32x2).  The kernels are short of
// instructions issued and not of the FMA pipe: with CUDA's logf, square root and sincosf, one unit
// at a time, they ran at 84 % of the issue slots with that pipe 47 % busy.  (A packed fma holds
// the pipe for 2.3 cycles with constant operands and 3.1 with three registers, a scalar one for 1.)
// A product and a sum are each rounded only where nothing joins them: a packed mul whose result
// goes into a packed add has come out rounded once, as an fma.  Where two roundings are needed the
// products are scalar (angle_pair in dist.cuh); here every sum of a product is an fma to begin with.
//  * u = 2^k z with z in [2/3, 4/3): m = 2 log u = g + g^2 Q(g) + k 2 ln 2 with g = 2z - 2
//    exact and Q a degree-8 minimax polynomial (2^-28 relative; relative to the whole
//    logarithm where k != 0);
//  * the radius with a minus sign (which saves the residual's negation) by one residual step
//    on the hardware reciprocal square root y = (-m)^-1/2 (P. Markstein, IBM J. Res. Dev. 34,
//    1990: s0 = m y, s = s0 + (s0^2 + m) y / 2), 0 for m = 0;
//  * a = n pi/2 + r, n by the rounding of a 2/pi, pi/2 in three parts of which the first
//    product is exact; sin r and cos r by minimax polynomials on |r| <= pi/4 (2^-28, 2^-33);
//  * n swaps the two, and its signs and the radius' minus go into the radius.
// The coefficients are derived by rocrand_b200/data/make_fp32_polynomials.py.  Measured
// on the device against 64 bits from the same uniforms, the products are 4.52e-8 off (2-norm),
// those of the library form 4.72e-8; logarithm 0.87 ulp at most, sine and cosine 1.5
// (tests/test_device_math_gpu.py and, for the host's build, tests/test_normal_math.py hold it there).
// Normal fp32, 2^26 values a call on one B200, library form -> now (the engines' own changes
// included): Philox 124 -> 94 us, XORWOW 123 -> 77, MRG32k3a 233 -> 149, MT19937 191 -> 136,
// ThreeFry4x32 167 -> 137, ThreeFry2x64 206 -> 169, MTGP32 202 -> 151, LFSR113 156 -> 104; half
// 108 -> 80, 120 -> 75, 177 -> 111, 170 -> 109, 130 -> 101, 214 -> 175, 185 -> 114, 138 -> 89.
#pragma once

#include "ieee.cuh"

#include <cmath>
#include <cstdint>
#include <cstring>

namespace rb200
{
namespace nm
{

// Two floats; on the device one 64-bit register pair.
struct F2
{
#if defined(__CUDA_ARCH__)
    unsigned long long v;
#else
    float x, y;
#endif
};

RB_HD F2 pack(float x, float y)
{
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
#else
    r.x = x;
    r.y = y;
#endif
    return r;
}

RB_HD void unpack(F2 a, float& x, float& y)
{
#if defined(__CUDA_ARCH__)
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
#else
    x = a.x;
    y = a.y;
#endif
}

RB_HD F2 rep(float c)
{
    return pack(c, c);
}

RB_HD F2 fma(F2 a, F2 b, F2 c)
{
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
#else
    r.x = std::fma(a.x, b.x, c.x);
    r.y = std::fma(a.y, b.y, c.y);
#endif
    return r;
}

RB_HD F2 mul(F2 a, F2 b)
{
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
#else
    r.x = a.x * b.x;
    r.y = a.y * b.y;
#endif
    return r;
}

RB_HD F2 add(F2 a, F2 b)
{
    F2 r;
#if defined(__CUDA_ARCH__)
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
#else
    r.x = a.x + b.x;
    r.y = a.y + b.y;
#endif
    return r;
}

RB_HD uint32_t bits(float x)
{
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
}

RB_HD float of_bits(uint32_t u)
{
    float x;
    memcpy(&x, &u, 4);
    return x;
}

// 1 / sqrt(-m) to 2^-22, at most 1e18 (m = 0, of either sign: minus_sqrt then gives 0).
RB_HD float rsqrt_seed(float m)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fabsf(m)));
    return fminf(y, 1e18f);
#else
    return std::fmin(1.0f / std::sqrt(std::fabs(m)), 1e18f);
#endif
}

// z in [2/3, 4/3) of a positive normal u = 2^k z, and k 2^23 as a float.
RB_HD void split(float u, float& z, float& k23)
{
    const uint32_t ix = bits(u);
    const uint32_t e  = (ix - 0x3f2aaaabu) & 0xff800000u;
    z                 = of_bits(ix - e);
    k23               = static_cast<float>(static_cast<int32_t>(e)); // exact
}

// 2 log u of two positive normal floats.
RB_HD F2 log_squared(F2 u)
{
    float u0, u1, z0, z1, k0, k1;
    unpack(u, u0, u1);
    split(u0, z0, k0);
    split(u1, z1, k1);
    const F2 g = fma(pack(z0, z1), rep(2.0f), rep(-2.0f)); // exact
    const F2 w = mul(g, g);
    F2       p = fma(rep(-0.00027413980569690466f), g, rep(0.0005520535632967949f));
    p          = fma(p, g, rep(-0.0009267727145925164f));
    p          = fma(p, g, rep(0.0021832501515746117f));
    p          = fma(p, g, rep(-0.005222465377300978f));
    p          = fma(p, g, rep(0.012507922947406769f));
    p          = fma(p, g, rep(-0.031248221173882484f));
    p          = fma(p, g, rep(0.08333292603492737f));
    p          = fma(p, g, rep(-0.2500000596046448f));
    p          = fma(w, p, g);
    return fma(pack(k0, k1), rep(1.6525917e-07f), p); // 2 ln 2 * 2^-23
}

// -sqrt(-m) of two non-positive floats (0 or <= -2^-100).
RB_HD F2 minus_sqrt(F2 m)
{
    float m0, m1;
    unpack(m, m0, m1);
    const F2 y  = pack(rsqrt_seed(m0), rsqrt_seed(m1));
    const F2 s0 = mul(m, y);
    const F2 r  = fma(s0, s0, m);
    return fma(r, mul(y, rep(0.5f)), s0);
}

// The quadrant's share of one unit: (x, y) = (sin r, cos r) swapped for odd n; the signs of
// sin a and cos a put on the radius, which is given as s < 0.
RB_HD void quadrant(uint32_t n, float& x, float& y, float s, float& s_sin, float& s_cos)
{
    const float    a = x, b = y;
    const bool     odd = (n & 1u) != 0u;
    x                  = odd ? b : a;
    y                  = odd ? a : b;
    const uint32_t t   = bits(s) ^ (~(n << 30) & 0x80000000u);
    s_sin              = of_bits(t);
    s_cos              = of_bits(t ^ (n << 31));
}

// Two units: the sine products in `ps`, the cosine products in `pc`.
RB_HD void box_muller(F2 u, F2 a, F2& ps, F2& pc)
{
    const F2 s = minus_sqrt(log_squared(u));
    const F2 t = fma(a, rep(0.63661977f), rep(12582912.0f)); // 1.5 2^23: n in the low bits
    const F2 q = add(t, rep(-12582912.0f));
    F2       r = fma(q, rep(-1.5707963705062866f), a); // exact
    r          = fma(q, rep(4.371139e-08f), r);
    r          = fma(q, rep(1.7151245e-15f), r);
    const F2 z = mul(r, r);
    F2       p = fma(rep(-0.00019515282474458218f), z, rep(0.00833216030150652f));
    p          = fma(p, z, rep(-0.16666655242443085f));
    const F2 sn = fma(p, mul(r, z), r);
    F2       d  = fma(rep(2.44331567955669e-05f), z, rep(-0.0013887316454201937f));
    d           = fma(d, z, rep(0.04166664555668831f));
    d           = fma(d, z, rep(-0.5f));
    const F2 cs = fma(d, z, rep(1.0f));
    float    t0, t1, s0, s1, x0, x1, y0, y1, a0, a1, b0, b1;
    unpack(t, t0, t1);
    unpack(s, s0, s1);
    unpack(sn, x0, x1);
    unpack(cs, y0, y1);
    quadrant(bits(t0), x0, y0, s0, a0, b0);
    quadrant(bits(t1), x1, y1, s1, a1, b1);
    ps = mul(pack(x0, x1), pack(a0, a1));
    pc = mul(pack(y0, y1), pack(b0, b1));
}

} // namespace nm
} // namespace rb200
