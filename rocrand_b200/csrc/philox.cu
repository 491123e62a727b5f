// philox.cu -- Philox4x32-10 generator: host object and fused sm_100a kernels.
//
// Output contract (what the reference's generate_philox, library/src/rng/philox4x32_10.hpp
// :107-214, produces on its default 1024x256 grid), restated position by position so any
// grid gives identical bytes:
//   * the output is split into a head of `head` elements (up to the first 16-byte
//     boundary), vec_n 16-byte vectors and a tail;
//   * vector j holds the distribution applied to the 4 stream values starting at
//     p(j) = 4*j + (j % 262144 == 0 ? start0 : head), where start0 = ceil(head/ow)*iw is
//     how far the head moved thread 0 of the reference grid;
//   * the head is produced sequentially from stream position 0, the tail sequentially
//     from p(vec_n);
//   * positions are relative to the generator's engine position, which advances by
//     ceil(n/ow)*iw per call (philox4x32_10.hpp:349-354).
// The common case (start0 == head and a block-aligned start) needs one Philox block per
// vector; otherwise a vector straddles two blocks.
#include "common.hpp"
#include "counter_engines.cuh"
#include "dist.cuh"
#include "generators.hpp"
#include "launch.cuh"
#include "batch.hpp"
#include "host_exec.hpp"
#include "philox.cuh"
#include "poisson.hpp"

#include <cstring>

namespace rb200
{

// A call with a head or tail has one block more, which makes them alone: a unit to a thread,
// the head's in the first warp and the tail's in the second.  (As one thread's sequential runs
// behind block 0's vectors they were up to 1.5 us of every such call.)
template<class F>
__device__ __forceinline__ bool philox_edges(const PhiloxCall& a, const F& g)
{
    if(a.head + a.tail == 0 || blockIdx.x + 1 != gridDim.x)
        return false;
    using T                        = typename F::T;
    const bool               tail  = threadIdx.x >= 32;
    const uint32_t           unit  = threadIdx.x & 31u;
    const uint32_t           count = threadIdx.x >= 64 ? 0u : (tail ? a.tail : a.head);
    const unsigned long long pos
        = tail ? 4 * a.vec_n + ((a.vec_n % kPhiloxRefStride) == 0 ? a.start0 : a.head) : 0ull;
    T* out = reinterpret_cast<T*>(a.data) + (tail ? a.n - a.tail : 0ull);
    if(unit * F::ow < count)
        philox_scalar_run(a, g, pos + unit * F::iw, out + unit * F::ow,
                          count - unit * F::ow < F::ow ? count - unit * F::ow : F::ow);
    return true;
}

// Blocks that take vectors.
__device__ __forceinline__ uint32_t philox_blocks(const PhiloxCall& a)
{
    return gridDim.x - (a.head + a.tail == 0 ? 0u : 1u);
}

// kAligned: start0 == head and (s0 + head) % 4 == 0, so vector j is exactly block
// c0 + (s0 + head)/4 + j.
template<class F, bool kAligned>
__global__ void __launch_bounds__(kBlock) philox_fill(PhiloxCall a, F f)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const F g = stage_table(f, smem);
    if(philox_edges(a, g))
        return;

    const unsigned long long tid    = static_cast<unsigned long long>(blockIdx.x) * kBlock + threadIdx.x;
    const unsigned long long stride = static_cast<unsigned long long>(philox_blocks(a)) * kBlock;

    if(kAligned)
    {
        const uint4 cbase = ctr_add(a.c0, (a.s0 + a.head) >> 2);
        for(unsigned long long j = tid; j < a.vec_n; j += stride)
        {
            const uint4 b = philox_block(ctr_add(cbase, j), a.keys);
            store16_cs(a.vec + j * 16, philox_vec(g, b));
        }
    }
    else
    {
        for(unsigned long long j = tid; j < a.vec_n; j += stride)
        {
            const uint32_t adj = (j & (kPhiloxRefStride - 1)) == 0 ? a.start0 : a.head;
            const unsigned long long q = a.s0 + adj + 4 * j;
            const uint4 c  = ctr_add(a.c0, q >> 2);
            const uint32_t s = static_cast<uint32_t>(q & 3);
            uint4 b = philox_block(c, a.keys);
            if(s != 0)
                b = interleave4(b, philox_block(ctr_add(c, 1), a.keys), s);
            store16_cs(a.vec + j * 16, philox_vec(g, b));
        }
    }

}

// Fast path: aligned vectors whose counters (x0 + j, y, z, w) share the upper words for the
// whole launch (x0 + vec_n <= 2^32, checked by the host).  Each thread produces two
// independent vectors per iteration so the two multiply chains interleave.
// (Its head and tail stay behind block 0's vectors: a block of their own, as the other kernels
// have, changes the schedule of this loop, 2^26 uniform fp64 91.6 -> 95.7 us on one B200.)
template<class F>
__global__ void __launch_bounds__(kBlock)
    philox_fill_fast(PhiloxCall a, PhiloxLane lane, uint32_t x0, F f)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const F g = stage_table(f, smem);

    const uint32_t vec_n  = static_cast<uint32_t>(a.vec_n);
    const uint32_t stride = gridDim.x * kBlock;
    uint32_t       j      = blockIdx.x * kBlock + threadIdx.x;
    for(; j + stride < vec_n; j += 2 * stride)
    {
        const uint4 b0 = philox_block_lane(x0 + j, lane, a.keys);
        const uint4 b1 = philox_block_lane(x0 + j + stride, lane, a.keys);
        // both transforms before either store, so that their chains can interleave
        const uint4 v0 = philox_vec(g, b0);
        const uint4 v1 = philox_vec(g, b1);
        store16_cs(a.vec + static_cast<size_t>(j) * 16, v0);
        store16_cs(a.vec + static_cast<size_t>(j + stride) * 16, v1);
    }
    if(j < vec_n)
        store16_cs(a.vec + static_cast<size_t>(j) * 16, philox_vec(g, philox_block_lane(x0 + j, lane, a.keys)));

    if(blockIdx.x == 0 && threadIdx.x == 0)
    {
        using T = typename F::T;
        if(a.head > 0)
            philox_scalar_run(a, g, 0, reinterpret_cast<T*>(a.data), a.head);
        if(a.tail > 0)
            philox_scalar_run(a, g, 4 * a.vec_n + a.head, reinterpret_cast<T*>(a.data) + (a.n - a.tail),
                              a.tail);
    }
}

// Shifted path: vectors whose words begin s = 1, 2 or 3 into a block (a misaligned buffer, or an
// earlier call that ended inside a block), the upper counter words fixed as in the fast path
// (x0 + vec_n + 1 <= 2^32, checked by the host).  A vector needs the last words of its block and
// the first s of the next: a warp evaluates the blocks of kRows rows of 32 vectors and one more,
// and every lane takes its neighbour's words by shuffle, so a vector costs 1 + 1/kRows
// evaluations and s shuffles instead of two evaluations.  Vectors j % 262144 == 0 that begin
// elsewhere (start0 != head) go through the general rule.  2^26 values one element off on one
// B200, both blocks evaluated -> this: uint 115.9 -> 61.5 us, uniform fp64 230.7 -> 126.8, normal
// fp32 170.4 -> 116.3.
template<unsigned kRows, class F>
__global__ void __launch_bounds__(kBlock)
    philox_fill_shifted(PhiloxCall a, PhiloxLane lane, uint32_t x0, F f)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const F g = stage_table(f, smem);
    if(philox_edges(a, g))
        return;

    const uint32_t vec_n = static_cast<uint32_t>(a.vec_n);
    const uint32_t s     = (a.s0 + a.head) & 3u;
    const uint32_t l     = threadIdx.x & 31u;
    const uint32_t step  = philox_blocks(a) * (kBlock / 32) * (32 * kRows);
    const bool     odd   = a.start0 != a.head;
    // `base` is the same in the whole warp: every lane takes part in the shuffles
    for(uint32_t base = (blockIdx.x * (kBlock / 32) + threadIdx.x / 32) * (32 * kRows); base < vec_n; base += step)
    {
        uint4 b[kRows + 1];
#pragma unroll
        for(unsigned k = 0; k < kRows; k++)
            b[k] = philox_block_lane(x0 + base + 32 * k + l, lane, a.keys);
        b[kRows] = philox_block_lane(x0 + base + 32 * kRows, lane, a.keys); // lane 0's of the next row
#pragma unroll
        for(unsigned k = 0; k < kRows; k++)
        {
            // lane 31's neighbour is lane 0 one row on
            const uint4    from = l == 0 ? b[k + 1] : b[k];
            const unsigned src  = (l + 1) & 31u;
            uint4          next = make_uint4(0u, 0u, 0u, 0u);
            next.x              = __shfl_sync(0xffffffffu, from.x, src);
            if(s > 1)
                next.y = __shfl_sync(0xffffffffu, from.y, src);
            if(s > 2)
                next.z = __shfl_sync(0xffffffffu, from.z, src);
            b[k] = interleave4(b[k], next, s);
        }
#pragma unroll
        for(unsigned k = 0; k < kRows; k++)
        {
            const uint32_t j = base + 32 * k + l;
            if(j >= vec_n)
                break;
            uint4 w = b[k];
            if(odd && (j & (kPhiloxRefStride - 1)) == 0)
            {
                const unsigned long long q = a.s0 + a.start0 + 4ull * j;
                const uint4              c = ctr_add(a.c0, q >> 2);
                w                          = philox_block(c, a.keys);
                if((q & 3) != 0)
                    w = interleave4(w, philox_block(ctr_add(c, 1), a.keys), static_cast<uint32_t>(q & 3));
            }
            store16_cs(a.vec + static_cast<size_t>(j) * 16, philox_vec(g, w));
        }
    }

}

// The same output contract on the host (host generators without a GPU): every vector by
// the general rule of philox_fill, the head and tail by the same sequential run.
template<class F>
static rocrand_status philox_run_host(const PhiloxCall& a, const F& f)
{
    host_parallel_for(a.vec_n, [&](unsigned long long j0, unsigned long long j1) {
        for(unsigned long long j = j0; j < j1; j++)
        {
            const uint32_t           adj = (j & (kPhiloxRefStride - 1)) == 0 ? a.start0 : a.head;
            const unsigned long long q   = a.s0 + adj + 4 * j;
            const uint4              c   = ctr_add(a.c0, q >> 2);
            const uint32_t           s   = static_cast<uint32_t>(q & 3);
            uint4                    b   = philox_block(c, a.keys);
            if(s != 0)
                b = interleave4(b, philox_block(ctr_add(c, 1), a.keys), s);
            const uint4 v = philox_vec(f, b);
            std::memcpy(a.vec + j * 16, &v, 16);
        }
    });
    using T = typename F::T;
    if(a.head > 0)
        philox_scalar_run(a, f, 0, reinterpret_cast<T*>(a.data), a.head);
    if(a.tail > 0)
    {
        const unsigned long long pos = 4 * a.vec_n + ((a.vec_n % kPhiloxRefStride) == 0 ? a.start0 : a.head);
        philox_scalar_run(a, f, pos, reinterpret_cast<T*>(a.data) + (a.n - a.tail), a.tail);
    }
    return ROCRAND_STATUS_SUCCESS;
}

// Grid of a kernel over `work` threads' items, and the edges' block where there are any; all
// resident at once.
template<class Kernel>
static unsigned philox_grid(Kernel k, const PhiloxCall& a, unsigned long long work, size_t smem)
{
    const unsigned edges = a.head + a.tail == 0 ? 0u : 1u;
    const unsigned main  = grid_for(k, work > 0 ? work : 1, smem, edges);
    return main + edges;
}

template<class F>
static rocrand_status launch_philox(PhiloxCall a, const F& f, cudaStream_t stream)
{
    const size_t   smem  = table_smem_bytes(f);
    const uint32_t s     = (a.s0 + a.head) & 3u;
    const uint4    cbase = ctr_add(a.c0, (a.s0 + a.head) >> 2);
    // 32-bit indices in the fast kernels: keep j + 2*stride below 2^32 too.
    const bool small = a.vec_n < (1ull << 31);
    if(s == 0 && a.start0 == a.head)
    {
        if(static_cast<unsigned long long>(cbase.x) + a.vec_n <= (1ull << 32) && small)
        {
            const PhiloxLane lane = philox_lane(cbase, a.keys);
            auto             k    = philox_fill_fast<F>;
            k<<<grid_for(k, a.vec_n > 0 ? (a.vec_n + 1) / 2 : 1, smem), kBlock, smem, stream>>>(a, lane, cbase.x, f);
            return launch_status();
        }
        auto k = philox_fill<F, true>;
        k<<<philox_grid(k, a, a.vec_n, smem), kBlock, smem, stream>>>(a, f);
        return launch_status();
    }
    // Rows per warp of the shifted kernel, on one B200: from 2^20 vectors four fill the GPU (2^24
    // values of normal fp32: 45.7 us evaluating every block twice, 35.7 with two rows, 31.4 with
    // four); below that two (10^6 values of uniform fp32: 5.1, 4.1, 4.5); below 2^17 a thread's
    // longer chain costs more than the evaluations saved (2^14 normal fp32: 4.1, 4.4, 6.2).
    if(s != 0 && static_cast<unsigned long long>(cbase.x) + a.vec_n + 1 <= (1ull << 32) && small
       && a.vec_n >= (1ull << 17))
    {
        const PhiloxLane lane = philox_lane(cbase, a.keys);
        if(a.vec_n >= (1ull << 20))
        {
            auto k = philox_fill_shifted<4, F>;
            k<<<philox_grid(k, a, (a.vec_n + 3) / 4, smem), kBlock, smem, stream>>>(a, lane, cbase.x, f);
        }
        else
        {
            auto k = philox_fill_shifted<2, F>;
            k<<<philox_grid(k, a, (a.vec_n + 1) / 2, smem), kBlock, smem, stream>>>(a, lane, cbase.x, f);
        }
        return launch_status();
    }
    auto k = philox_fill<F, false>;
    k<<<philox_grid(k, a, a.vec_n, smem), kBlock, smem, stream>>>(a, f);
    return launch_status();
}

// ---------------------------------------------------------------------------------------

PhiloxGenerator::PhiloxGenerator() = default;
PhiloxGenerator::~PhiloxGenerator() = default;

// Output `index` of distribution d comes from stream value index * iw / ow (index a multiple
// of ow, output aligned to the distribution's vector), so the position is that offset.
rocrand_status PhiloxGenerator::set_output_position(Dist d, unsigned long long index)
{
    if(d == Dist::U64)
        return ROCRAND_STATUS_TYPE_ERROR;
    DistParams p;
    return with_functor(d, p, [&](auto f) -> rocrand_status {
        using F = decltype(f);
        if(index % F::ow != 0)
            return ROCRAND_STATUS_LENGTH_NOT_MULTIPLE;
        return set_offset(index / F::ow * F::iw);
    });
}

rocrand_status PhiloxGenerator::init()
{
    if(m_initialized)
        return ROCRAND_STATUS_SUCCESS;
    // the Poisson tables are allocated here, as the reference's generators do in init(), so
    // that a generate call recorded by a stream capture allocates nothing
    const rocrand_status st = m_poisson.reserve();
    if(st != ROCRAND_STATUS_SUCCESS)
        return st;
    // seed(seed, subsequence 0, offset) (philox4x32_10.hpp:291-306, engine seed :134-141)
    m_pos = CounterPos{};
    m_pos.advance(m_offset);
    m_initialized = true;
    return ROCRAND_STATUS_SUCCESS;
}

rocrand_status PhiloxGenerator::set_order(rocrand_ordering order)
{
    // philox4x32_10.hpp:258-278: DEFAULT, DYNAMIC, BEST, LEGACY.  All give the same
    // output on this build.
    switch(order)
    {
        case ROCRAND_ORDERING_PSEUDO_DEFAULT:
        case ROCRAND_ORDERING_PSEUDO_DYNAMIC:
        case ROCRAND_ORDERING_PSEUDO_BEST:
        case ROCRAND_ORDERING_PSEUDO_LEGACY:
            m_order       = order;
            m_initialized = false;
            return ROCRAND_STATUS_SUCCESS;
        default: return ROCRAND_STATUS_OUT_OF_RANGE;
    }
}

rocrand_status PhiloxGenerator::generate(void* data, size_t n, Dist d, const DistParams& p)
{
    if(d == Dist::U64)
        return ROCRAND_STATUS_TYPE_ERROR; // 32-bit engine (philox4x32_10.hpp:359-375)
    rocrand_status st = init();
    if(st != ROCRAND_STATUS_SUCCESS)
        return st;
    if(data == nullptr)
        return ROCRAND_STATUS_SUCCESS;
    const size_t tsize = dist_elem_size(d);
    if(reinterpret_cast<uintptr_t>(data) % tsize != 0)
        return ROCRAND_STATUS_LENGTH_NOT_MULTIPLE; // not even element-aligned

    st = with_functor(d, p, [&](auto f) -> rocrand_status {
        using F                    = decltype(f);
        constexpr unsigned iw      = F::iw;
        constexpr unsigned ow      = F::ow;
        constexpr unsigned fow     = (4 / iw) * ow; // elements per 16-byte vector
        const uintptr_t    addr    = reinterpret_cast<uintptr_t>(data);
        const size_t       mis     = (fow - addr / tsize % fow) % fow;
        PhiloxCall         a;
        a.keys   = philox_keys(m_seed);
        a.c0     = m_pos.counter;
        a.s0     = m_pos.sub;
        a.head   = static_cast<uint32_t>(n < mis ? n : mis);
        a.tail   = static_cast<uint32_t>((n - a.head) % fow);
        a.vec_n  = (n - a.head) / fow;
        a.start0 = a.head > 0 ? (a.head + ow - 1) / ow * iw : 0;
        a.n      = n;
        a.data   = static_cast<unsigned char*>(data);
        a.vec    = a.data + mis * tsize;
        if(n == 0)
            return ROCRAND_STATUS_SUCCESS;
        const rocrand_status s = m_host_exec ? philox_run_host(a, f) : launch_philox(a, f, m_stream);
        if(s == ROCRAND_STATUS_SUCCESS)
            m_pos.advance(static_cast<unsigned long long>((n + ow - 1) / ow) * iw);
        return s;
    });
    return st;
}

// Poisson values of a fresh Philox4x32-10 stream (seed, offset) with a caller-supplied
// table: used by the entry point that allocates nothing (noalloc.cu).
rocrand_status philox_poisson_with_table(unsigned long long seed, unsigned long long offset,
                                         unsigned int* data, size_t n, const DistParams& p,
                                         cudaStream_t stream)
{
    if(data == nullptr || n == 0)
        return ROCRAND_STATUS_SUCCESS;
    CounterPos pos;
    pos.advance(offset);
    const uintptr_t addr = reinterpret_cast<uintptr_t>(data);
    if(addr % sizeof(unsigned int) != 0)
        return ROCRAND_STATUS_LENGTH_NOT_MULTIPLE;
    const size_t mis = (4 - addr / sizeof(unsigned int) % 4) % 4;
    PhiloxCall   a;
    a.keys   = philox_keys(seed);
    a.c0     = pos.counter;
    a.s0     = pos.sub;
    a.head   = static_cast<uint32_t>(n < mis ? n : mis);
    a.tail   = static_cast<uint32_t>((n - a.head) % 4);
    a.vec_n  = (n - a.head) / 4;
    a.start0 = a.head; // iw = ow = 1
    a.n      = n;
    a.data   = reinterpret_cast<unsigned char*>(data);
    a.vec    = a.data + mis * sizeof(unsigned int);
    if(p.huge)
        return launch_philox(a, FnPoissonHuge{p.sqrt_lambda, p.lambda}, stream);
    return launch_philox(a, FnPoisson{p.thr, p.alias, p.size, p.offset}, stream);
}

rocrand_status PhiloxGenerator::batch_descriptor(uint32_t dist, double p0, double p1, void* data,
                                                size_t n, BatchReq& r, cudaStream_t stream)
{
    rocrand_status st = init();
    if(st != ROCRAND_STATUS_SUCCESS)
        return st;
    r             = BatchReq{};
    r.kind        = BK_PHILOX;
    r.philox.keys = philox_keys(m_seed);
    r.philox.c0   = m_pos.counter;
    r.philox.s0   = m_pos.sub;
    st            = batch_set_dist(r, dist, p0, p1, stream);
    if(st == ROCRAND_STATUS_SUCCESS)
        st = batch_layout(r, data, n);
    if(st != ROCRAND_STATUS_SUCCESS)
        return st;
    unsigned iw, ow;
    batch_widths(BK_PHILOX, dist, iw, ow);
    m_pos.advance(static_cast<unsigned long long>((n + ow - 1) / ow) * iw);
    return ROCRAND_STATUS_SUCCESS;
}

rocrand_status PhiloxGenerator::generate_poisson(unsigned int* data, size_t n, double lambda)
{
    rocrand_status st = init();
    if(st != ROCRAND_STATUS_SUCCESS)
        return st;
    DistParams p;
    st = m_poisson.get(lambda, m_stream, false, p);
    if(st != ROCRAND_STATUS_SUCCESS)
        return st;
    return generate(data, n, Dist::POISSON, p);
}

} // namespace rb200
