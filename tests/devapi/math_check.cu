// math_check.cu -- the kernels' device-only square roots and packed Box-Muller (sqrt_mid of
// sobol_dist.cuh, sqrt_inner of precise_math.cuh, normal_math.cuh), run by themselves for
// tests/test_device_math_gpu.py.  Test infrastructure.
#include "normal_math.cuh"
#include "precise_math.cuh"
#include "sobol_dist.cuh"

#include <cstddef>
#include <cstdint>

using namespace rb200;

namespace
{

__global__ void sqrt_mid_kernel(uint32_t first, uint32_t count, unsigned long long* differ)
{
    for(uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
    {
        const float x = __uint_as_float(first + i);
        if(__float_as_uint(sqrt_mid(x)) != __float_as_uint(__fsqrt_rn(x)))
            atomicAdd(differ, 1ull);
    }
}

__global__ void sqrt_inner_kernel(const double* t, size_t n, double* ours, double* rounded, double* seed)
{
    for(size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        ours[i]    = pm::sqrt_inner(t[i]);
        rounded[i] = __dsqrt_rn(t[i]);
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(t[i]));
        seed[i] = y;
    }
}

__global__ void box_muller_kernel(const float* u, const float* a, size_t pairs, float* l, float* s, float* c)
{
    for(size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        const nm::F2 uu = nm::pack(u[2 * i], u[2 * i + 1]), aa = nm::pack(a[2 * i], a[2 * i + 1]);
        nm::F2       ps, pc;
        nm::unpack(nm::log_squared(uu), l[2 * i], l[2 * i + 1]);
        nm::box_muller(uu, aa, ps, pc);
        nm::unpack(ps, s[2 * i], s[2 * i + 1]);
        nm::unpack(pc, c[2 * i], c[2 * i + 1]);
    }
}

int done()
{
    return static_cast<int>(cudaGetLastError()) | static_cast<int>(cudaDeviceSynchronize());
}

} // namespace

// Every pointer is device memory.
extern "C" __attribute__((visibility("default"))) int math_sqrt_mid(uint32_t first, uint32_t count,
                                                                    unsigned long long* differ)
{
    sqrt_mid_kernel<<<1024, 256>>>(first, count, differ);
    return done();
}

extern "C" __attribute__((visibility("default"))) int math_sqrt_inner(const double* t, size_t n, double* ours,
                                                                      double* rounded, double* seed)
{
    sqrt_inner_kernel<<<1024, 256>>>(t, n, ours, rounded, seed);
    return done();
}

extern "C" __attribute__((visibility("default"))) int math_box_muller(const float* u, const float* a, size_t pairs,
                                                                      float* l, float* s, float* c)
{
    box_muller_kernel<<<1024, 256>>>(u, a, pairs, l, s, c);
    return done();
}
