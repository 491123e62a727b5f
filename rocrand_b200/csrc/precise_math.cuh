// precise_math.cuh -- natural logarithm and sine/cosine in double precision whose results
// are correctly rounded except in rare near-halfway cases (internal precision ~2^-66).
//
// The reference's host generators evaluate Box-Muller and the inverse-erf normal with the
// C library's log/sin/cos, which are themselves within ~0.52 ulp of the exact value.  The
// normal and log-normal outputs of this library are compared with them at <= 2 ulp (fp64);
// the device's own 1-2 ulp functions can leave a 3-ulp gap after the products, so the fp64
// transforms use these instead.  Method (standard table-driven reduction, written here):
//  * log x: x = 2^k z with z in [OFF, 2 OFF), OFF just above sqrt(1/2), split by integer
//    operations on the bit pattern; the top 8 bits of z's offset pick one of 256
//    subintervals with a tabulated invc = 1/c of at most 9 significant bits, so that
//    r = z invc - 1 is exact in one fma (|r| < 2^-8; the subinterval around 1 has c = 1);
//    log x = (k ln2_hi + log c_hi) + r - r^2/2 + r^3 P(r) + small terms, the first sums
//    compensated and one final rounding;
//  * sin/cos x (0 <= x <= 2 pi): x = m C + b with C = 2 pi / 464 as a double, m the nearest;
//    b is exact in one fma (x and m C are multiples of 2^-60 where m > 0, and |b| < 2^-7), so
//    neither the reduction nor b needs a second word; sin/cos(m C) from a double-double table
//    over the whole circle (15 KB, so no quadrant to select either); sin b and cos b - 1 by
//    short series.
// Both are IEEE operations only (add, mul, fma), so their host and device builds give identical
// results; the tables are computed in binary128 at build time
// (rocrand_b200/data/make_precise_tables.c).  (sqrt_inner below starts from an instruction of the
// device's own and is another function on the host.)
// Issue bounds the transforms (an fp64 instruction takes two to three cycles of its scheduler:
// 2.07 with constant operands, 3.03 with three registers, every other about one): a Philox
// Box-Muller pair took 269 instructions, 108 of them fp64, with a two-step reduction (k pi/2 in
// three parts, then j/64), log's special cases and the rounded square root; now 184 and 76.  Normal
// fp64, 2^25 values a call on one B200, before -> now (the engines' own changes included): Philox
// 191 -> 141 us, XORWOW 197 -> 125, LFSR113 224 -> 149, MRG32k3a 235 -> 150, MT19937 266 -> 195,
// MTGP32 274 -> 236, ThreeFry4x64 249 -> 194.  Misses of correct rounding in 3 10^6: sine 32 -> 27,
// cosine 23 -> 23, log 0.
#pragma once

#include "precise_tables.inc"

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define RB_PM_HD __host__ __device__ __forceinline__
#else
#define RB_PM_HD inline
#endif

namespace rb200
{
namespace pm
{

// rows of four doubles: (invc, head, tail, 0) and (sin hi, sin lo, cos hi, cos lo)
#if defined(__CUDACC__)
struct __align__(16) Row
{
    double v0, v1, v2, v3;
};
static __device__ const Row kLogTabDev[RB_LOG_ROWS]     = RB_LOG_INIT;
static __device__ const Row kScTabDev[RB_SC_TABLE_ROWS] = RB_SC_TABLE_INIT;
#endif
static const double kLogTabHost[RB_LOG_ROWS][4]     = RB_LOG_INIT;
static const double kScTabHost[RB_SC_TABLE_ROWS][4] = RB_SC_TABLE_INIT;

// Row i of a table, read as 16-byte halves through the non-coherent cache on the device.
#if defined(__CUDA_ARCH__)
#define RB_PM_ROW(name, i, r)                                                        \
    const double2 r##_a = __ldg(reinterpret_cast<const double2*>(name##Dev + (i)));  \
    const double2 r##_b = __ldg(reinterpret_cast<const double2*>(name##Dev + (i)) + 1); \
    const double  r[4]  = {r##_a.x, r##_a.y, r##_b.x, r##_b.y}
#else
#define RB_PM_ROW(name, i, r) const double* const r = name##Host[i]
#endif

RB_PM_HD double fma_(double a, double b, double c)
{
#if defined(__CUDA_ARCH__)
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

RB_PM_HD uint64_t bits_of(double x)
{
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
}

RB_PM_HD double from_bits(uint64_t u)
{
    double x;
    memcpy(&x, &u, 8);
    return x;
}

// s + e == a + b exactly when a == 0 or |a| >= |b| (Dekker's fast two-sum)
RB_PM_HD void fast_two_sum(double a, double b, double& s, double& e)
{
    s = a + b;
    e = b - (s - a);
}

// Natural logarithm of a positive normal x, given by its bits, less `down` times ln 2.  (Any
// bits give a table row in range: log() selects its special cases afterwards.)
RB_PM_HD double log_core(uint64_t ix, int down)
{
    const uint64_t tmp = ix - RB_LOG_OFF;
    const unsigned i   = static_cast<unsigned>(tmp >> 44) & 255u;
    const int      k   = static_cast<int>(static_cast<int64_t>(tmp) >> 52) - down;
    const double   z   = from_bits(ix - (tmp & 0xfff0000000000000ull)); // x / 2^k in [OFF, 2 OFF)
    RB_PM_ROW(kLogTab, i, row);
    const double kd = static_cast<double>(k);
    const double r  = fma_(z, row[0], -1.0);          // exact: |r| < 2^-8, invc has <= 9 bits
    const double t1 = fma_(kd, RB_LN2_HI, row[1]);    // exact: both multiples of 2^-42, |t1| < 2^10
    double       s1, e1, s2, e2;
    fast_two_sum(t1, r, s1, e1); // |t1| >= |r| or t1 = 0 (checked over the rows at build time)
    // -r^2 / 2 = q + ql exactly
    const double r2 = r * r;
    const double q  = -0.5 * r2;
    const double ql = -0.5 * fma_(r, r, -r2);
    // |s1| >= |q|: s1 = r when t1 = 0 (the subinterval around 1), else |s1| ~ |log x| >= 2^-10
    fast_two_sum(s1, q, s2, e2);
    // r^3 (1/3 - r/4 + r^2/5 - r^3/6 + r^4/7 - r^5/8): the first term left out, r^9/9, is
    // below 2^-67 of the result
    double p = -1.0 / 8.0;
    p        = fma_(p, r, 1.0 / 7.0);
    p        = fma_(p, r, -1.0 / 6.0);
    p        = fma_(p, r, 1.0 / 5.0);
    p        = fma_(p, r, -1.0 / 4.0);
    p        = fma_(p, r, 1.0 / 3.0);
    const double tail = p * (r2 * r);
    const double low  = ((e1 + e2) + (ql + row[2])) + fma_(kd, RB_LN2_LO, tail);
    return s2 + low;
}

// Natural logarithm, near-correctly rounded.
RB_PM_HD double log(double x)
{
    const bool   sub = x < 0x1p-1022; // subnormal (or zero / negative: replaced below)
    const double y   = log_core(bits_of(sub ? x * 0x1p54 : x), sub ? 54 : 0);
    return x > 0.0 ? (x == INFINITY ? x : y) : (x == 0.0 ? -INFINITY : NAN);
}

// The same for a uniform, 2^-1022 <= x <= 1: no special case.
RB_PM_HD double log_uniform(double x)
{
    return log_core(bits_of(x), 0);
}

// sin and cos of x for 0 <= x <= 2 pi (the Box-Muller angles; 2 pi as a double), near-correctly
// rounded.
RB_PM_HD void sincos(double x, double& s_out, double& c_out)
{
    // m = x / C rounded, as the low bits of t = 1.5 2^52 + m and as a double
    const double t  = fma_(x, RB_SC_INV_STEP, 0x1.8p52);
    const double md = t - 0x1.8p52;
    const int    m  = static_cast<int>(static_cast<uint32_t>(bits_of(t)));
    RB_PM_ROW(kScTab, m, row);
    const double sh = row[0], sl = row[1], ch = row[2], cl = row[3];
    const double b  = fma_(md, -RB_SC_STEP, x); // exact, |b| < 2^-7
    const double b2 = b * b;
    // sin b - b = b^3 (-1/6 + b^2/120 - b^4/5040);  cos b - 1 = b^2 (-1/2 + b^2/24 - b^4/720);
    // the first terms left out (b^9/9!, b^8/8!) are below 2^-73 of b and of 1
    double sp = -1.0 / 5040.0;
    sp        = fma_(sp, b2, 1.0 / 120.0);
    sp        = fma_(sp, b2, -1.0 / 6.0);
    const double sinb_rest = (sp * b2) * b;
    double       cp        = -1.0 / 720.0;
    cp                     = fma_(cp, b2, 1.0 / 24.0);
    cp                     = fma_(cp, b2, -0.5);
    const double cm1 = cp * b2;
    // sin(a + b) = sin a + (cos a * b + sin a * (cos b - 1) + cos a * (sin b - b))
    const double psh = ch * b;
    const double psl = fma_(ch, b, -psh);
    double       ssh, ssl;
    // |sin a| >= sin C > |cos a * b|, or sin a = 0: the rows at the multiples of pi, where it
    // is below 2^-57, have it in their low word alone
    fast_two_sum(sh, psh, ssh, ssl);
    const double s_low = ((ssl + psl) + sl) + fma_(cl, b, fma_(sh, cm1, ch * sinb_rest));
    s_out              = ssh + s_low;
    // cos(a + b) = cos a - (sin a * b) + cos a * (cos b - 1) - sin a * (sin b - b)
    const double pch = sh * b;
    const double pcl = fma_(sh, b, -pch);
    double       csh, csl;
    fast_two_sum(ch, -pch, csh, csl); // likewise
    const double c_low = ((csl - pcl) + cl) + fma_(-sl, b, fma_(ch, cm1, -(sh * sinb_rest)));
    c_out              = csh + c_low;
}

// Square root of t = 0 or 2^-200 <= t <= 2^200, within 2^-103 relative before its one rounding,
// so correctly rounded but where the root is as near as that to a midpoint of two doubles.
// From an approximation y = (1 + d) / sqrt(t) (the reciprocal square root instruction's, |d| <
// 2^-19), Goldschmidt's coupled pair (R. E. Goldschmidt, "Applications of division by
// convergence", MIT 1964) g = t y ~ sqrt(t), h = y / 2 ~ 1 / (2 sqrt(t)):
//   g h = (1 - 2 e) / 2 gives e = 1/2 - g h in one fma, |e| < 2^-18.9;
//   sqrt(t) = g (1 - 2 e)^(-1/2) = g (1 + e + 3/2 e^2 + 5/2 e^3 + ..): with q = e (1 + 3/2 e),
//   g1 = g + g q and h1 = h + h q are 5/2 |e|^3 < 2^-55 and their roundings off, |n| < 2^-52 in
//   all for g1 = sqrt(t) (1 + n).
// Then the residual correction by one fma each (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): r = t - g1^2 = -t (2 n +
// n^2), and g1 + r h1 = sqrt(t) (1 - n^2 / 2 and less than 2^-52 |n|), rounded once.
// 2^25 Philox normals fp64 on one B200 with the rounded root's intrinsic -> this: 146 -> 141 us;
// MT19937 217 -> 193.  On the device the function is not IEEE operations alone (the host has
// std::sqrt); tests/test_device_math_gpu.py compares the device's with the rounded root.
RB_PM_HD double sqrt_inner(double t)
{
#if defined(__CUDA_ARCH__)
    // t = 0 starts from a tiny number instead, and t y = 0 then stays 0
    const double seed = __hiloint2double(max(__double2hiint(t), 0x02000000), __double2loint(t));
    double       y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(seed));
    const double g  = t * y;
    const double h  = 0.5 * y;
    const double e  = fma_(-g, h, 0.5);
    const double q  = e * fma_(1.5, e, 1.0);
    const double g1 = fma_(g, q, g);
    const double h1 = fma_(h, q, h);
    const double r  = fma_(-g1, g1, t);
    return fma_(r, h1, g1);
#else
    return std::sqrt(t);
#endif
}

} // namespace pm
} // namespace rb200
