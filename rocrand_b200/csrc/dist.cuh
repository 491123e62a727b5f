// dist.cuh -- distribution functors fused into the generator kernels (sm_100a).
//
// Each functor reproduces one host functor of the reference (library/src/rng/distribution/
// *.hpp) together with the scalar conversion it calls in the *host* branch of
// library/include/rocrand/rocrand_{uniform,normal,discrete}.h, because parity is defined
// against the reference's host generators.  Every rounding step is written with an
// explicit _rn intrinsic: a product is fused into an FMA only where it is exact (scaling
// by a power of two), so the device rounds exactly where the x86-64 host does.
// The fp32 and half Box-Muller transforms run on two units at a time (normal_math.cuh) on the
// device, within an ulp or two of the host C library, inside the stated fp32 tolerance; the
// log-normals' exponential is CUDA's.  The fp64 Box-Muller transforms and
// the inverse-erf normal take log/sin/cos from precise_math.cuh (correctly rounded but for
// rare near-halfway cases), so that the fp64 outputs stay within 2 ulp of the host's and
// the ill-conditioned inverse-erf formula starts from the same logarithm wherever the host
// library's is itself correctly rounded.
#pragma once

#include <type_traits>
#include "common.hpp"
#include "ieee.cuh"
#include "normal_math.cuh"
#include "precise_math.cuh"

#include <cuda_fp16.h>

#include <cstdint>

namespace rb200
{

// Constants of rocrand_common.h:24-36, spelled as the reference spells them so that they
// round to the same binary values.
#define RB_2POW16_INV (1.5258789e-05f)
#define RB_2POW16_INV_2PI (9.58738e-05f)
#define RB_2POW32_INV (2.3283064e-10f)
#define RB_2POW32_INV_DOUBLE (2.3283064365386963e-10)
#define RB_2POW32_INV_2PI (1.46291807e-09f)
#define RB_2POW53_INV_DOUBLE (1.1102230246251565e-16)
#define RB_PI_DOUBLE (3.1415926535897932)
#define RB_SQRT2 (1.4142135f)

// ---- scalar conversions ----

// rocrand_uniform.h:61-64: 2^-32 + v * 2^-32 (exact product, one rounding).
RB_HD float u32_to_f32(uint32_t v)
{
    return ieee::ffma(ieee::u2f(v), RB_2POW32_INV, RB_2POW32_INV);
}

// rocrand_uniform.h:97-107: 53 bits from (v1, v2 >> 11), 2^-53 + v * 2^-53.
RB_HD double u32x2_to_f64(uint32_t v1, uint32_t v2)
{
    const uint64_t v = (uint64_t)v1 | ((uint64_t)(v2 >> 11) << 32);
    return ieee::dfma(ieee::ull2d(v), RB_2POW53_INV_DOUBLE, RB_2POW53_INV_DOUBLE);
}

// rocrand_uniform.h:92-95: 2^-32 + v * 2^-32 in double (exact).
RB_HD double u32_to_f64(uint32_t v)
{
    return ieee::dfma(ieee::u2d(v), RB_2POW32_INV_DOUBLE, RB_2POW32_INV_DOUBLE);
}

// rocrand_uniform.h:150-153: half of 2^-16 + v * 2^-16 (float math exact, RNE to half).
RB_HD __half u16_to_f16(uint32_t v16)
{
    return __float2half_rn(ieee::ffma((float)(v16 & 0xffffu), RB_2POW16_INV, RB_2POW16_INV));
}

// The Box-Muller products of a unit on the host: (sin a, cos a) sqrt(-2 log u) with the C
// library's functions, every step rounded (rocrand_normal.h:51-66, host branch).
inline float2 box_muller_host(float u, float a)
{
    const float s = ieee::fsqrt(ieee::fmul(-2.0f, std::log(u)));
    return make_float2(ieee::fmul(std::sin(a), s), ieee::fmul(std::cos(a), s));
}

// ---- fp32 and half Box-Muller functors: two units at a time ----
// Such a functor names the uniforms and angles of two units (`uniforms`, `angles`: the inputs'
// own rounding steps) and its parameters; normal_pair makes both units' outputs.  On the device
// one unit alone is the same computation with the unit taken twice, so a value does not depend on
// whether it was made alone or beside another; on the host each unit is made with the C library.

// rocrand_uniform.h:61-64 and rocrand_normal.h:51-66 of two 32-bit words.
RB_HD nm::F2 uniform_pair(uint32_t x0, uint32_t x1)
{
    return nm::fma(nm::pack(ieee::u2f(x0), ieee::u2f(x1)), nm::rep(RB_2POW32_INV), nm::rep(RB_2POW32_INV));
}
// (The products are scalar: packed ones are fused with the packed sum, which rounds once where
// the reference rounds twice.)
RB_HD nm::F2 angle_pair(uint32_t y0, uint32_t y1)
{
    return nm::add(nm::pack(ieee::fmul(ieee::u2f(y0), RB_2POW32_INV_2PI), ieee::fmul(ieee::u2f(y1), RB_2POW32_INV_2PI)),
                   nm::rep(RB_2POW32_INV_2PI));
}

template<class F, class W>
inline float2 box_muller_host(const F& f, const W* in)
{
    float u, a, unused;
    nm::unpack(f.uniforms(in, in), u, unused);
    nm::unpack(f.angles(in, in), a, unused);
    return box_muller_host(u, a);
}

template<class F>
RB_HD void exponentials(const F& f, float (&out)[2])
{
    if(f.exponential())
    {
        out[0] = ieee::expf_(out[0]);
        out[1] = ieee::expf_(out[1]);
    }
}

// The half outputs of one unit from its products (rocrand_normal.h:102-122, float branch used by
// the host build: halves of the products first).
template<class F>
RB_HD void finish_f16(const F& f, float s, float c, __half* out)
{
    const float z = ieee::fadd(f.mean, ieee::fmul(f.stddev, __half2float(__float2half_rn(s))));
    const float w = ieee::fadd(f.mean, ieee::fmul(f.stddev, __half2float(__float2half_rn(c))));
    out[0]        = __float2half_rn(f.exponential() ? ieee::expf_(z) : z);
    out[1]        = __float2half_rn(f.exponential() ? ieee::expf_(w) : w);
}

template<class F, class W>
RB_HD void normal_pair(const F& f, const W* in0, const W* in1, float* out0, float* out1)
{
    float a[2], b[2];
#if defined(__CUDA_ARCH__)
    nm::F2 ps, pc;
    nm::box_muller(f.uniforms(in0, in1), f.angles(in0, in1), ps, pc);
    const nm::F2 m = nm::rep(f.mean), d = nm::rep(f.stddev);
    nm::unpack(nm::fma(ps, d, m), a[0], b[0]);
    nm::unpack(nm::fma(pc, d, m), a[1], b[1]);
#else
    const float2 v = box_muller_host(f, in0), w = box_muller_host(f, in1);
    a[0] = ieee::fadd(f.mean, ieee::fmul(v.x, f.stddev));
    a[1] = ieee::fadd(f.mean, ieee::fmul(v.y, f.stddev));
    b[0] = ieee::fadd(f.mean, ieee::fmul(w.x, f.stddev));
    b[1] = ieee::fadd(f.mean, ieee::fmul(w.y, f.stddev));
#endif
    exponentials(f, a);
    exponentials(f, b);
    out0[0] = a[0];
    out0[1] = a[1];
    out1[0] = b[0];
    out1[1] = b[1];
}

template<class F, class W>
RB_HD void normal_pair(const F& f, const W* in0, const W* in1, __half* out0, __half* out1)
{
#if defined(__CUDA_ARCH__)
    nm::F2 ps, pc;
    float  s0, s1, c0, c1;
    nm::box_muller(f.uniforms(in0, in1), f.angles(in0, in1), ps, pc);
    nm::unpack(ps, s0, s1);
    nm::unpack(pc, c0, c1);
    finish_f16(f, s0, c0, out0);
    finish_f16(f, s1, c1, out1);
#else
    const float2 v = box_muller_host(f, in0), w = box_muller_host(f, in1);
    finish_f16(f, v.x, v.y, out0);
    finish_f16(f, w.x, w.y, out1);
#endif
}

// One unit alone.
template<class F, class W, class T>
RB_HD void normal_unit(const F& f, const W* in, T* out)
{
#if defined(__CUDA_ARCH__)
    T unused[2];
    normal_pair(f, in, in, out, unused);
#else
    const float2 v = box_muller_host(f, in);
    if constexpr(std::is_same_v<T, float>)
    {
        float a[2] = {ieee::fadd(f.mean, ieee::fmul(v.x, f.stddev)), ieee::fadd(f.mean, ieee::fmul(v.y, f.stddev))};
        exponentials(f, a);
        out[0] = a[0];
        out[1] = a[1];
    }
    else
    {
        finish_f16(f, v.x, v.y, out);
    }
#endif
}

RB_HD nm::F2 uniform_pair_f16(uint32_t x0, uint32_t x1)
{
    return nm::fma(nm::pack(static_cast<float>(x0), static_cast<float>(x1)), nm::rep(RB_2POW16_INV),
                   nm::rep(RB_2POW16_INV));
}
RB_HD nm::F2 angle_pair_f16(uint32_t y0, uint32_t y1)
{
    return nm::add(nm::pack(ieee::fmul(static_cast<float>(y0), RB_2POW16_INV_2PI),
                            ieee::fmul(static_cast<float>(y1), RB_2POW16_INV_2PI)),
                   nm::rep(RB_2POW16_INV_2PI));
}

// Two units of any functor: side by side where it has a form for that, one after the other
// elsewhere.
template<class F, class = void>
struct has_pair : std::false_type
{
};
template<class F>
struct has_pair<F, std::enable_if_t<F::kPair>> : std::true_type
{
};
template<class F, class W>
RB_HD void apply_pair(const F& f, const W* in0, const W* in1, typename F::T* out0, typename F::T* out1)
{
    if constexpr(has_pair<F>::value)
    {
        f.pair(in0, in1, out0, out1);
    }
    else
    {
        f(in0, out0);
        f(in1, out1);
    }
}

// mean + stddev v: one rounding on the device, the reference's two on the host.
RB_HD double scaled_f64(double v, double stddev, double mean)
{
#if defined(__CUDA_ARCH__)
    return __fma_rn(v, stddev, mean);
#else
    return mean + v * stddev;
#endif
}

// rocrand_normal.h:68-89 (host branch: sin/cos of w * pi rounded in double).
RB_HD double2 box_muller_f64(uint32_t x, uint32_t y, uint32_t z, uint32_t w)
{
    const uint64_t v1 = (uint64_t)x ^ ((uint64_t)y << 21);
    const double   u  = ieee::dfma(ieee::ull2d(v1), RB_2POW53_INV_DOUBLE, RB_2POW53_INV_DOUBLE);
    const uint64_t v2 = (uint64_t)z ^ ((uint64_t)w << 21);
    const double   ww = ieee::dfma(ieee::ull2d(v2), RB_2POW53_INV_DOUBLE * 2.0, RB_2POW53_INV_DOUBLE * 2.0);
    const double   s  = pm::sqrt_inner(ieee::dmul(-2.0, pm::log_uniform(u)));
    const double   a  = ieee::dmul(ww, RB_PI_DOUBLE);
    double         sv, cv;
    pm::sincos(a, sv, cv);
    return make_double2(ieee::dmul(sv, s), ieee::dmul(cv, s));
}

// rocrand_normal.h:196-220 roc_d_erfinv (host branch).
RB_HD double erfinv_d(double x)
{
    const double sgn = (x < 0.0) ? -1.0 : 1.0;
    x                = ieee::dmul(ieee::dsub(1.0, x), ieee::dadd(1.0, x));
    const double lnx = pm::log(x);
    if(isnan(lnx))
        return 1.0;
    if(isinf(lnx))
        return 0.0;
    const double tt1 = ieee::dadd(2.0 / (RB_PI_DOUBLE * 0.147), ieee::dmul(0.5, lnx));
    const double tt2 = ieee::dmul(1.0 / (0.147), lnx);
    return sgn * ieee::dsqrt(ieee::dadd(-tt1, ieee::dsqrt(ieee::dsub(ieee::dmul(tt1, tt1), tt2))));
}

// rocrand_normal.h:265-270: sqrt(2) is a float literal promoted to double.
RB_HD double normal_from_u32_f64(uint32_t x)
{
    const double p = u32_to_f64(x);
    return ieee::dmul((double)RB_SQRT2, erfinv_d(ieee::dsub(ieee::dmul(2.0, p), 1.0)));
}

// rocrand_discrete.h:33-60 discrete_alias for a 32-bit input.
RB_HD uint32_t alias_lookup(uint32_t r, uint32_t size, uint32_t offset,
                                                 const double* prob, const uint32_t* alias)
{
    const double   x   = ieee::dmul(ieee::u2d(r), RB_2POW32_INV_DOUBLE);
    const double   nx  = ieee::dmul(ieee::u2d(size), x);
    const double   fnx = floor(nx);
    const double   y   = ieee::dsub(nx, fnx);
    const uint32_t i   = ieee::d2u_rz(fnx);
    return offset + (y < prob[i] ? i : alias[i]);
}

// The same pick from packed integer entries (poisson.hpp alias_entry: threshold in the low
// 33 bits, alias above): i = (size r) >> 32, entry i when the low word of size r is below
// the threshold.  One 8-byte read, no conversion or fp64 operation.
RB_HD uint32_t alias_lookup_packed(uint32_t r, uint32_t size, uint32_t offset,
                                                        const unsigned long long* tab)
{
    const unsigned long long p  = static_cast<unsigned long long>(size) * r;
    const uint32_t           i  = static_cast<uint32_t>(p >> 32);
    const unsigned long long e  = tab[i];
    const unsigned long long lo = p & 0xffffffffull;
    return offset + (lo < (e & 0x1ffffffffull) ? i : static_cast<uint32_t>(e >> 33));
}

// poisson.hpp:80-108 poisson_distribution_huge: round(sqrt(lambda) * N + lambda).
RB_HD uint32_t poisson_huge(uint32_t r, double sqrt_lambda, double lambda)
{
    const double nd = normal_from_u32_f64(r);
    return (uint32_t)(long long)round(ieee::dadd(ieee::dmul(sqrt_lambda, nd), lambda));
}

// ---- functors: iw inputs (32-bit engine words) -> ow outputs of T ----
// Naming follows the reference entry point they serve.

struct FnUint // uniform_distribution<uint> (uniform.hpp:42-53)
{
    using T                      = uint32_t;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const uint32_t* in, T* out) const { out[0] = in[0]; }
};

struct FnUchar // uniform_distribution<uchar> (uniform.hpp:55-66): the word's 4 bytes
{
    using T                      = uint8_t;
    static constexpr unsigned iw = 1, ow = 4;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = (uint8_t)in[0];
        out[1] = (uint8_t)(in[0] >> 8);
        out[2] = (uint8_t)(in[0] >> 16);
        out[3] = (uint8_t)(in[0] >> 24);
    }
};

struct FnUshort // uniform_distribution<ushort> (uniform.hpp:68-79): the word's 2 halves
{
    using T                      = uint16_t;
    static constexpr unsigned iw = 1, ow = 2;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = (uint16_t)in[0];
        out[1] = (uint16_t)(in[0] >> 16);
    }
};

struct FnFloat // uniform_distribution<float> (uniform.hpp:81-91)
{
    using T                      = float;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = u32_to_f32(in[0]);
    }
};

struct FnDouble // uniform_distribution<double> (uniform.hpp:93-103)
{
    using T                      = double;
    static constexpr unsigned iw = 2, ow = 1;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = u32x2_to_f64(in[0], in[1]);
    }
};

struct FnHalf // uniform_distribution<half> (uniform.hpp:105-117)
{
    using T                      = __half;
    static constexpr unsigned iw = 1, ow = 2;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = u16_to_f16(in[0] & 0xffffu);
        out[1] = u16_to_f16(in[0] >> 16);
    }
};

// normal_distribution<float, uint, 4> (normal.hpp:49-69) and log_normal_distribution<float,
// uint, 4> (log_normal.hpp:51-71)
template<bool kLog>
struct FnBoxMullerF
{
    using T                      = float;
    static constexpr unsigned iw = 2, ow = 2;
    static constexpr bool     kPair = true;
    float                     mean, stddev;
    RB_HD static constexpr bool exponential() { return kLog; }
    RB_HD nm::F2 uniforms(const uint32_t* a, const uint32_t* b) const { return uniform_pair(a[0], b[0]); }
    RB_HD nm::F2 angles(const uint32_t* a, const uint32_t* b) const { return angle_pair(a[1], b[1]); }
    RB_HD void   pair(const uint32_t* in0, const uint32_t* in1, T* out0, T* out1) const
    {
        normal_pair(*this, in0, in1, out0, out1);
    }
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        normal_unit(*this, in, out);
    }
};
using FnNormalF    = FnBoxMullerF<false>;
using FnLogNormalF = FnBoxMullerF<true>;

struct FnNormalD // normal_distribution<double, uint, 4> (normal.hpp:90-111)
{
    using T                      = double;
    static constexpr unsigned iw = 4, ow = 2;
    double                    mean, stddev;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        const double2 v = box_muller_f64(in[0], in[1], in[2], in[3]);
        out[0]          = scaled_f64(v.x, stddev, mean);
        out[1]          = scaled_f64(v.y, stddev, mean);
    }
};

struct FnLogNormalD // log_normal_distribution<double, uint, 4> (log_normal.hpp:92-113)
{
    using T                      = double;
    static constexpr unsigned iw = 4, ow = 2;
    double                    mean, stddev;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        const double2 v = box_muller_f64(in[0], in[1], in[2], in[3]);
        out[0]          = ieee::exp_(scaled_f64(v.x, stddev, mean));
        out[1]          = ieee::exp_(scaled_f64(v.y, stddev, mean));
    }
};

// normal_distribution<half, uint, 4> (normal.hpp:113-136) and log_normal_distribution<half,
// uint, 4> (log_normal.hpp:115-139), float branch
template<bool kLog>
struct FnBoxMullerH
{
    using T                      = __half;
    static constexpr unsigned iw = 1, ow = 2;
    static constexpr bool     kPair = true;
    float                     mean, stddev; // the half parameters widened to float
    RB_HD static constexpr bool exponential() { return kLog; }
    RB_HD nm::F2 uniforms(const uint32_t* a, const uint32_t* b) const
    {
        return uniform_pair_f16(a[0] & 0xffffu, b[0] & 0xffffu);
    }
    RB_HD nm::F2 angles(const uint32_t* a, const uint32_t* b) const
    {
        return angle_pair_f16(a[0] >> 16, b[0] >> 16);
    }
    RB_HD void pair(const uint32_t* in0, const uint32_t* in1, T* out0, T* out1) const
    {
        normal_pair(*this, in0, in1, out0, out1);
    }
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        normal_unit(*this, in, out);
    }
};
using FnNormalH    = FnBoxMullerH<false>;
using FnLogNormalH = FnBoxMullerH<true>;

// poisson_distribution<ALIAS> (poisson.hpp:49-76).  The table is staged in shared memory
// by the kernel; prob/alias then point there.
struct FnPoisson
{
    using T                      = uint32_t;
    static constexpr unsigned iw = 1, ow = 1;
    static constexpr bool     kTable = true;
    const unsigned long long* prob;  // packed entries (alias_entry), not probabilities
    const uint32_t*           alias; // unused: the aliases are packed with the thresholds
    uint32_t                  size, offset;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = alias_lookup_packed(in[0], size, offset, prob);
    }
};

// poisson_distribution_huge (poisson.hpp:80-108), lambda > 4000.
struct FnPoissonHuge
{
    using T                      = uint32_t;
    static constexpr unsigned iw = 1, ow = 1;
    double                    sqrt_lambda, lambda;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = poisson_huge(in[0], sqrt_lambda, lambda);
    }
};

// ---- functors over 64-bit engine words (ThreeFry 2x64/4x64) ----
// uniform.hpp:119-200, normal.hpp:138-200, log_normal.hpp:138-200, and the 64-bit input
// overloads of rocrand_uniform.h / rocrand_normal.h / rocrand_discrete.h.

struct Fn64Ulonglong // uniform_distribution<ull, ull>
{
    using T                      = unsigned long long;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        out[0] = in[0];
    }
};

template<class U, unsigned N>
struct Fn64Split // uchar (ow 8), ushort (ow 4), uint (ow 2): the word's bytes in order
{
    using T                      = U;
    static constexpr unsigned iw = 1, ow = N;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
#pragma unroll
        for(unsigned k = 0; k < N; k++)
            out[k] = static_cast<U>(in[0] >> (k * 8 * sizeof(U)));
    }
};

struct Fn64Float // rocrand_uniform.h:66-69: 2^-32 + (v >> 32) * 2^-32
{
    using T                      = float;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        out[0] = u32_to_f32(static_cast<uint32_t>(in[0] >> 32));
    }
};

struct Fn64Double // rocrand_uniform.h:109-116: 2^-53 + (v >> 11) * 2^-53
{
    using T                      = double;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        out[0] = ieee::dfma(ieee::ull2d(in[0] >> 11), RB_2POW53_INV_DOUBLE, RB_2POW53_INV_DOUBLE);
    }
};

struct Fn64Half // uniform_distribution<half, ull>: four 16-bit fields
{
    using T                      = __half;
    static constexpr unsigned iw = 1, ow = 4;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
#pragma unroll
        for(unsigned k = 0; k < 4; k++)
            out[k] = u16_to_f16(static_cast<uint32_t>(in[0] >> (16 * k)) & 0xffffu);
    }
};

struct Fn64NormalF // box_muller(unsigned long long): x = low word, y = high word
{
    using T                      = float;
    static constexpr unsigned iw = 1, ow = 2;
    static constexpr bool     kPair = true;
    float                     mean, stddev;
    bool                      log_normal;
    RB_HD bool   exponential() const { return log_normal; }
    RB_HD nm::F2 uniforms(const unsigned long long* a, const unsigned long long* b) const
    {
        return uniform_pair(static_cast<uint32_t>(a[0]), static_cast<uint32_t>(b[0]));
    }
    RB_HD nm::F2 angles(const unsigned long long* a, const unsigned long long* b) const
    {
        return angle_pair(static_cast<uint32_t>(a[0] >> 32), static_cast<uint32_t>(b[0] >> 32));
    }
    RB_HD void pair(const unsigned long long* in0, const unsigned long long* in1, T* out0, T* out1) const
    {
        normal_pair(*this, in0, in1, out0, out1);
    }
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        normal_unit(*this, in, out);
    }
};

struct Fn64NormalD // box_muller_double(ulonglong2)
{
    using T                      = double;
    static constexpr unsigned iw = 2, ow = 2;
    double                    mean, stddev;
    bool                      log_normal;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        const double2 v = box_muller_f64(static_cast<uint32_t>(in[0]), static_cast<uint32_t>(in[0] >> 32),
                                         static_cast<uint32_t>(in[1]), static_cast<uint32_t>(in[1] >> 32));
        const double  a = scaled_f64(v.x, stddev, mean);
        const double  b = scaled_f64(v.y, stddev, mean);
        out[0]          = log_normal ? ieee::exp_(a) : a;
        out[1]          = log_normal ? ieee::exp_(b) : b;
    }
};

struct Fn64NormalH // normal_distribution_half2(ull): (ushort)v and (ushort)(v >> 32)
{
    using T                      = __half;
    static constexpr unsigned iw = 1, ow = 2;
    static constexpr bool     kPair = true;
    float                     mean, stddev;
    bool                      log_normal;
    RB_HD bool   exponential() const { return log_normal; }
    RB_HD nm::F2 uniforms(const unsigned long long* a, const unsigned long long* b) const
    {
        return uniform_pair_f16(static_cast<uint32_t>(a[0]) & 0xffffu, static_cast<uint32_t>(b[0]) & 0xffffu);
    }
    RB_HD nm::F2 angles(const unsigned long long* a, const unsigned long long* b) const
    {
        return angle_pair_f16(static_cast<uint32_t>(a[0] >> 32) & 0xffffu,
                              static_cast<uint32_t>(b[0] >> 32) & 0xffffu);
    }
    RB_HD void pair(const unsigned long long* in0, const unsigned long long* in1, T* out0, T* out1) const
    {
        normal_pair(*this, in0, in1, out0, out1);
    }
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        normal_unit(*this, in, out);
    }
};

// discrete_alias(unsigned long long) (rocrand_discrete.h:75-81): x = r * 2^-64 after the
// round-to-nearest conversion of r to double.  When r rounds up to 2^64 the reference reads
// one entry past the table; here the index is clamped to the last entry instead.
struct Fn64Poisson
{
    using T                      = uint32_t;
    static constexpr unsigned iw = 1, ow = 1;
    const double*             prob;
    const uint32_t*           alias;
    uint32_t                  size, offset;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        const double x   = ieee::dmul(ieee::ull2d(in[0]), 5.4210108624275221700372640043497e-20);
        const double nx  = ieee::dmul(ieee::u2d(size), x);
        const double fnx = floor(nx);
        const double y   = ieee::dsub(nx, fnx);
        uint32_t     i   = ieee::d2u_rz(fnx);
        i                = i < size ? i : size - 1;
        out[0]           = offset + (y < prob[i] ? i : alias[i]);
    }
};

struct Fn64PoissonHuge // normal_distribution_double(ull) then round(sqrt(l) * N + l)
{
    using T                      = uint32_t;
    static constexpr unsigned iw = 1, ow = 1;
    double                    sqrt_lambda, lambda;
    RB_HD void operator()(const unsigned long long* in, T* out) const
    {
        const double p  = ieee::dfma(ieee::ull2d(in[0] >> 11), RB_2POW53_INV_DOUBLE, RB_2POW53_INV_DOUBLE);
        const double nd = ieee::dmul((double)RB_SQRT2, erfinv_d(ieee::dsub(ieee::dmul(2.0, p), 1.0)));
        out[0]          = (uint32_t)(long long)round(ieee::dadd(ieee::dmul(sqrt_lambda, nd), lambda));
    }
};

// normal_distribution<double, uint, 2> / log_normal_distribution<double, uint, 2>
// (normal.hpp:71-88): the inverse-erf normal, one word per value; used by ThreeFry2x32.
struct FnNormalD1
{
    using T                      = double;
    static constexpr unsigned iw = 1, ow = 1;
    double                    mean, stddev;
    bool                      log_normal;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        const double z = ieee::dadd(mean, ieee::dmul(normal_from_u32_f64(in[0]), stddev));
        out[0]         = log_normal ? ieee::exp_(z) : z;
    }
};

// ---- MRG functors (uniform.hpp:224-314, normal.hpp:200-270, log_normal.hpp:200-276,
//      poisson.hpp:416-441): the raw MRG output lies in [1, m1] and is normalised by the
//      engine's own constants (rocrand_uniform.h:161-219, rocrand_normal.h:138-172). ----

struct Mrg31k3pNorm // rocrand_mrg31k3p.h:32-34
{
    static constexpr double kNorm     = 4.656612875245796923e-10;
    static constexpr double kUintNorm = 2.000000001396983862;
};
struct Mrg32k3aNorm // rocrand_mrg32k3a.h:38-39
{
    static constexpr double kNorm     = 2.3283065498378288e-10;
    static constexpr double kUintNorm = 1.000000048661607;
};

// (v - 1) * UINT_NORM, truncated.  On the device both conversions are fp64 sums with 2^52 (the
// integer in the low word): the conversion instructions take eight cycles each, a sum two.
template<class N>
RB_HD uint32_t mrg_to_u32(uint32_t v)
{
#if defined(__CUDA_ARCH__)
    const double x = __dsub_rn(__hiloint2double(0x43300000, static_cast<int>(v - 1u)), 0x1p52);
    return static_cast<uint32_t>(__double2loint(__dadd_rz(__dmul_rn(x, N::kUintNorm), 0x1p52)));
#else
    return ieee::d2u_rz(ieee::dmul(ieee::u2d(v - 1u), N::kUintNorm));
#endif
}
template<class N>
RB_HD float mrg_to_f32(uint32_t v)
{
    return ieee::d2f(ieee::dmul(ieee::u2d(v), N::kNorm));
}
template<class N>
RB_HD double mrg_to_f64(uint32_t v)
{
    return ieee::dmul(ieee::u2d(v), N::kNorm);
}

template<class N, class Inner>
struct FnMrgRemap // uint/uchar/ushort/half/Poisson: remap to [0, 2^32) then the plain functor
{
    using T                      = typename Inner::T;
    static constexpr unsigned iw = 1, ow = Inner::ow;
    static constexpr bool     kPair = has_pair<Inner>::value;
    Inner                     inner;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        const uint32_t v = mrg_to_u32<N>(in[0]);
        inner(&v, out);
    }
    RB_HD void pair(const uint32_t* in0, const uint32_t* in1, T* out0, T* out1) const
    {
        const uint32_t v[2] = {mrg_to_u32<N>(in0[0]), mrg_to_u32<N>(in1[0])};
        apply_pair(inner, v, v + 1, out0, out1);
    }
};

template<class N>
struct FnMrgFloat
{
    using T                      = float;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = mrg_to_f32<N>(in[0]);
    }
};

template<class N>
struct FnMrgDouble
{
    using T                      = double;
    static constexpr unsigned iw = 1, ow = 1;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = mrg_to_f64<N>(in[0]);
    }
};

template<class N>
struct FnMrgNormalF // mrg_box_muller (rocrand_normal.h:138-152)
{
    using T                      = float;
    static constexpr unsigned iw = 2, ow = 2;
    static constexpr bool     kPair = true;
    float                     mean, stddev;
    bool                      log_normal;
    RB_HD bool   exponential() const { return log_normal; }
    RB_HD nm::F2 uniforms(const uint32_t* a, const uint32_t* b) const
    {
        return nm::pack(mrg_to_f32<N>(a[0]), mrg_to_f32<N>(b[0]));
    }
    RB_HD nm::F2 angles(const uint32_t* a, const uint32_t* b) const
    {
        return nm::mul(nm::pack(mrg_to_f32<N>(a[1]), mrg_to_f32<N>(b[1])), nm::rep(6.2831855f));
    }
    RB_HD void pair(const uint32_t* in0, const uint32_t* in1, T* out0, T* out1) const
    {
        normal_pair(*this, in0, in1, out0, out1);
    }
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        normal_unit(*this, in, out);
    }
};

template<class N>
struct FnMrgNormalD // mrg_box_muller_double (rocrand_normal.h:154-172): float uniforms widened
{
    using T                      = double;
    static constexpr unsigned iw = 2, ow = 2;
    double                    mean, stddev;
    bool                      log_normal;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        const double u = (double)mrg_to_f32<N>(in[0]);
        const double v = (double)mrg_to_f32<N>(in[1]) * 2.0;
        const double s = pm::sqrt_inner(ieee::dmul(-2.0, pm::log_uniform(u)));
        double       sv, cv;
        pm::sincos(ieee::dmul(v, RB_PI_DOUBLE), sv, cv);
        const double a = scaled_f64(ieee::dmul(sv, s), stddev, mean);
        const double b = scaled_f64(ieee::dmul(cv, s), stddev, mean);
        out[0]         = log_normal ? ieee::exp_(a) : a;
        out[1]         = log_normal ? ieee::exp_(b) : b;
    }
};

template<class N>
struct FnMrgPoissonHuge
{
    using T                      = uint32_t;
    static constexpr unsigned iw = 1, ow = 1;
    double                    sqrt_lambda, lambda;
    RB_HD void operator()(const uint32_t* in, T* out) const
    {
        out[0] = poisson_huge(mrg_to_u32<N>(in[0]), sqrt_lambda, lambda);
    }
};

// Transforms that a thread runs several units of side by side: the packed fp32 / half pairs,
// and the fp64 Box-Muller (a logarithm, a square root and a sine / cosine per unit).
template<class F>
struct long_transform : has_pair<F>
{
};
template<>
struct long_transform<FnNormalD> : std::true_type
{
};
template<>
struct long_transform<FnLogNormalD> : std::true_type
{
};

template<class F>
struct has_table
{
    static constexpr bool value = false;
};
template<>
struct has_table<FnPoisson>
{
    static constexpr bool value = true;
};
template<>
struct has_table<Fn64Poisson>
{
    static constexpr bool value = true;
};
template<class N>
struct has_table<FnMrgRemap<N, FnPoisson>>
{
    static constexpr bool value = true;
};

// Stages a Poisson alias table into shared memory (all threads of the block take part)
// and returns a functor reading it there.  smem holds size doubles then size uints.
template<class F>
struct table_of
{
    __host__ __device__ static F& get(F& f) { return f; }
    __host__ __device__ static const F& get(const F& f) { return f; }
};
template<class N>
struct table_of<FnMrgRemap<N, FnPoisson>>
{
    using W = FnMrgRemap<N, FnPoisson>;
    __host__ __device__ static FnPoisson& get(W& f) { return f.inner; }
    __host__ __device__ static const FnPoisson& get(const W& f) { return f.inner; }
};

template<class F>
__device__ __forceinline__ F stage_table(const F& fw, unsigned char* smem)
{
    if constexpr(has_table<F>::value)
    {
        const auto& f = table_of<F>::get(fw);
        using E       = typename std::remove_cv<typename std::remove_pointer<decltype(f.prob)>::type>::type;
        static_assert(sizeof(E) == 8, "8-byte table entries");
        // packed entries (FnPoisson) carry their aliases; Fn64Poisson has a separate array
        constexpr bool packed = std::is_same<E, unsigned long long>::value;
        E*        p = reinterpret_cast<E*>(smem);
        uint32_t* a = reinterpret_cast<uint32_t*>(smem + sizeof(E) * f.size);
        for(uint32_t i = threadIdx.x; i < f.size; i += blockDim.x)
        {
            p[i] = f.prob[i];
            if constexpr(!packed)
                a[i] = f.alias[i];
        }
        __syncthreads();
        F     g  = fw;
        auto& gt = table_of<F>::get(g);
        gt.prob  = p;
        if constexpr(!packed)
            gt.alias = a;
        return g;
    }
    else
    {
        return fw;
    }
}

template<class F>
inline size_t table_smem_bytes(const F& f)
{
    if constexpr(has_table<F>::value)
    {
        const auto& t = table_of<F>::get(f);
        using E       = typename std::remove_cv<typename std::remove_pointer<decltype(t.prob)>::type>::type;
        constexpr bool packed = std::is_same<E, unsigned long long>::value;
        return (size_t)t.size * (sizeof(E) + (packed ? 0 : sizeof(uint32_t)));
    }
    else
        return 0;
}

// Calls `body(functor)` with the functor that serves distribution d.  Used by every
// generator family to instantiate its kernel once per distribution.
template<class Body>
inline rocrand_status with_functor(Dist d, const DistParams& p, Body&& body)
{
    switch(d)
    {
        case Dist::U32: return body(FnUint{});
        case Dist::U8: return body(FnUchar{});
        case Dist::U16: return body(FnUshort{});
        case Dist::F32: return body(FnFloat{});
        case Dist::F64: return body(FnDouble{});
        case Dist::F16: return body(FnHalf{});
        case Dist::NORMAL_F32: return body(FnNormalF{p.mean_f, p.std_f});
        case Dist::LOGNORMAL_F32: return body(FnLogNormalF{p.mean_f, p.std_f});
        case Dist::NORMAL_F64: return body(FnNormalD{p.mean_d, p.std_d});
        case Dist::LOGNORMAL_F64: return body(FnLogNormalD{p.mean_d, p.std_d});
        case Dist::NORMAL_F16:
            return body(FnNormalH{__half2float(__ushort_as_half(p.mean_h)),
                                  __half2float(__ushort_as_half(p.std_h))});
        case Dist::LOGNORMAL_F16:
            return body(FnLogNormalH{__half2float(__ushort_as_half(p.mean_h)),
                                     __half2float(__ushort_as_half(p.std_h))});
        case Dist::POISSON:
            if(p.huge)
                return body(FnPoissonHuge{p.sqrt_lambda, p.lambda});
            return body(FnPoisson{p.thr, p.alias, p.size, p.offset});
        default: return ROCRAND_STATUS_TYPE_ERROR;
    }
}

// Functor selection for the MRG engines (raw output in [1, m1]).
template<class N, class Body>
inline rocrand_status with_functor_mrg(Dist d, const DistParams& p, Body&& body)
{
    const float mh = __half2float(__ushort_as_half(p.mean_h));
    const float sh = __half2float(__ushort_as_half(p.std_h));
    switch(d)
    {
        case Dist::U32: return body(FnMrgRemap<N, FnUint>{FnUint{}});
        case Dist::U8: return body(FnMrgRemap<N, FnUchar>{FnUchar{}});
        case Dist::U16: return body(FnMrgRemap<N, FnUshort>{FnUshort{}});
        case Dist::F32: return body(FnMrgFloat<N>{});
        case Dist::F64: return body(FnMrgDouble<N>{});
        case Dist::F16: return body(FnMrgRemap<N, FnHalf>{FnHalf{}});
        case Dist::NORMAL_F32: return body(FnMrgNormalF<N>{p.mean_f, p.std_f, false});
        case Dist::LOGNORMAL_F32: return body(FnMrgNormalF<N>{p.mean_f, p.std_f, true});
        case Dist::NORMAL_F64: return body(FnMrgNormalD<N>{p.mean_d, p.std_d, false});
        case Dist::LOGNORMAL_F64: return body(FnMrgNormalD<N>{p.mean_d, p.std_d, true});
        case Dist::NORMAL_F16: return body(FnMrgRemap<N, FnNormalH>{FnNormalH{mh, sh}});
        case Dist::LOGNORMAL_F16: return body(FnMrgRemap<N, FnLogNormalH>{FnLogNormalH{mh, sh}});
        case Dist::POISSON:
            if(p.huge)
                return body(FnMrgPoissonHuge<N>{p.sqrt_lambda, p.lambda});
            return body(FnMrgRemap<N, FnPoisson>{FnPoisson{p.thr, p.alias, p.size, p.offset}});
        default: return ROCRAND_STATUS_TYPE_ERROR;
    }
}

// Functor selection for engines producing 64-bit words.
template<class Body>
inline rocrand_status with_functor64(Dist d, const DistParams& p, Body&& body)
{
    const float mh = __half2float(__ushort_as_half(p.mean_h));
    const float sh = __half2float(__ushort_as_half(p.std_h));
    switch(d)
    {
        case Dist::U64: return body(Fn64Ulonglong{});
        case Dist::U32: return body(Fn64Split<uint32_t, 2>{});
        case Dist::U8: return body(Fn64Split<uint8_t, 8>{});
        case Dist::U16: return body(Fn64Split<uint16_t, 4>{});
        case Dist::F32: return body(Fn64Float{});
        case Dist::F64: return body(Fn64Double{});
        case Dist::F16: return body(Fn64Half{});
        case Dist::NORMAL_F32: return body(Fn64NormalF{p.mean_f, p.std_f, false});
        case Dist::LOGNORMAL_F32: return body(Fn64NormalF{p.mean_f, p.std_f, true});
        case Dist::NORMAL_F64: return body(Fn64NormalD{p.mean_d, p.std_d, false});
        case Dist::LOGNORMAL_F64: return body(Fn64NormalD{p.mean_d, p.std_d, true});
        case Dist::NORMAL_F16: return body(Fn64NormalH{mh, sh, false});
        case Dist::LOGNORMAL_F16: return body(Fn64NormalH{mh, sh, true});
        case Dist::POISSON:
            if(p.huge)
                return body(Fn64PoissonHuge{p.sqrt_lambda, p.lambda});
            return body(Fn64Poisson{p.prob, p.alias, p.size, p.offset});
        default: return ROCRAND_STATUS_TYPE_ERROR;
    }
}

} // namespace rb200
