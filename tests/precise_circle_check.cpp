// Edges of pm::sincos's table and of pm::log_uniform (host build of precise_math.cuh) against
// binary128: the doubles at and beside the multiples of pi/2, both sides of every boundary
// between two table cells, the smallest angles and 2 pi; the uniforms of 53 bits at every
// table row of the logarithm, where log_uniform and log must agree bit for bit.
#include "precise_math.cuh"

#include <quadmath.h>

#include <cmath>
#include <cstdio>
#include <cstring>

static double worst = 0.0;
static long   miss = 0, count = 0;

static void check(double got, __float128 exact)
{
    const double e = static_cast<double>(exact);
    const double u = std::nextafter(std::fabs(e), INFINITY) - std::fabs(e);
    worst          = std::fmax(worst, std::fabs(static_cast<double>(((__float128)got - exact) / (__float128)u)));
    miss += got != e;
    count++;
}

static void angle(double a)
{
    if(!(a >= 0.0) || a > 6.283185307179586)
        return;
    double s, c;
    rb200::pm::sincos(a, s, c);
    check(s, sinq((__float128)a));
    check(c, cosq((__float128)a));
}

int main()
{
    for(int k = 0; k <= 4; k++)
    {
        double up = k * 1.5707963267948966, down = up;
        for(int d = 0; d < 2000; d++)
        {
            angle(up);
            angle(down);
            up   = std::nextafter(up, 10.0);
            down = std::nextafter(down, -1.0);
        }
        for(int e = -50; e < -6; e++)
        {
            angle(k * 1.5707963267948966 + std::ldexp(1.2345, e));
            angle(k * 1.5707963267948966 - std::ldexp(1.2345, e));
        }
    }
    for(int m = 0; m < RB_SC_TABLE_ROWS; m++)
    {
        double up = (m + 0.5) * RB_SC_STEP, down = up;
        for(int d = 0; d < 20; d++)
        {
            angle(up);
            angle(down);
            up   = std::nextafter(up, 10.0);
            down = std::nextafter(down, -1.0);
        }
    }
    angle(0x1p-51 * 3.141592653589793 / 2.0);
    long differ = 0;
    for(uint64_t i = 0; i < RB_LOG_ROWS; i++)
        for(int e = 0; e < 53; e++)
        {
            double         z;
            const uint64_t b = RB_LOG_OFF + (i << 44) + i * 977u;
            std::memcpy(&z, &b, 8);
            z = std::ldexp(z, -e - 1);
            differ += rb200::pm::log_uniform(z) != rb200::pm::log(z);
        }
    differ += rb200::pm::log_uniform(1.0) != 0.0;
    std::printf("%.6f %ld %ld %ld\n", worst, miss, count, differ);
    return 0;
}
