// Accuracy of rocrand_b200/csrc/normal_math.cuh (host build of the device header: the same
// operations with a rounded reciprocal square root as the seed) against double precision.
// Prints the largest error in ulp of 2 log u and of the products, the products' relative
// error in the 2-norm, and the products at u = 1.
#include "normal_math.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace rb200;

static double ulps(float got, double exact)
{
    const float  e = static_cast<float>(std::fabs(exact));
    const double u = std::nextafter(e, INFINITY) - e;
    return std::fabs(got - exact) / u;
}

int main(int argc, char** argv)
{
    const long   n = argc > 1 ? std::atol(argv[1]) : 1000000;
    std::mt19937 rng(7);
    double       log_max = 0, prod_max = 0, num = 0, den = 0;
    const float  pi_half[] = {1.5707964f, 3.1415927f, 4.712389f, 6.2831855f};
    for(long t = 0; t < n; t++)
    {
        float u[2], a[2];
        for(int k = 0; k < 2; k++)
        {
            uint32_t x = rng(), y = rng();
            if((t & 15) == 0)
                x = 0xffffffffu - (x >> (8 + (t / 16) % 24)); // near 1
            if((t & 15) == 1)
                x >>= (t / 16) % 32; // small
            u[k] = std::fma(static_cast<float>(x), 0x1p-32f, 0x1p-32f);
            a[k] = 1.46291807e-09f + static_cast<float>(y) * 1.46291807e-09f;
            if((t & 15) == 2) // the floats around the multiples of pi / 2
                a[k] = std::nextafter(pi_half[(t / 16) % 4], (t / 64) % 2 ? 0.0f : 4.0f);
            if((t & 15) == 3)
                a[k] = pi_half[(t / 16) % 4];
        }
        float        l[2], s[2], c[2];
        nm::F2       ps, pc;
        nm::unpack(nm::log_squared(nm::pack(u[0], u[1])), l[0], l[1]);
        nm::box_muller(nm::pack(u[0], u[1]), nm::pack(a[0], a[1]), ps, pc);
        nm::unpack(ps, s[0], s[1]);
        nm::unpack(pc, c[0], c[1]);
        for(int k = 0; k < 2; k++)
        {
            const double m = 2.0 * std::log(static_cast<double>(u[k]));
            if(m != 0.0)
                log_max = std::fmax(log_max, ulps(l[k], m));
            const double r = std::sqrt(-m);
            const double x[2] = {r * std::sin(static_cast<double>(a[k])), r * std::cos(static_cast<double>(a[k]))};
            const float  g[2] = {s[k], c[k]};
            for(int j = 0; j < 2; j++)
            {
                if(x[j] != 0.0)
                    prod_max = std::fmax(prod_max, ulps(g[j], x[j]));
                num += (g[j] - x[j]) * (g[j] - x[j]);
                den += x[j] * x[j];
            }
        }
    }
    nm::F2 ps, pc;
    float  s0, s1, c0, c1;
    nm::box_muller(nm::pack(1.0f, 1.0f), nm::pack(1.0f, 4.0f), ps, pc);
    nm::unpack(ps, s0, s1);
    nm::unpack(pc, c0, c1);
    std::printf("log %.4f\nproduct %.4f\nnorm %.4g\none %g %g %g %g\n", log_max, prod_max, std::sqrt(num / den), s0,
                s1, c0, c1);
    return 0;
}
