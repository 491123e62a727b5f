// sobol.cu -- Sobol32, scrambled Sobol32, Sobol64 and scrambled Sobol64 quasi-random
// generators.
//
// Output contract of the reference (library/src/rng/sobol.hpp:72-256, 618-717): the output is
// dimension-major, out[d * N + i] = dist(x_d(offset + i)) with N = n / dims, where x_d(k) is
// the XOR of the direction vectors of dimension d selected by the bits of the Gray code
// k ^ (k >> 1) (rocrand_sobol32.h:122-170); the scrambled variants XOR the result with a
// per-dimension constant which, as the reference's generator is written (sobol.hpp:514),
// is word d of the scrambled direction-vector table.  The point counter is 32-bit and
// advances by N per call.
//
// B200 kernel: grid.y = dimension (its 32/64 vectors staged in shared memory), each thread
// produces a run of consecutive points by Gray-code steps (one XOR each) and leaps ahead by a
// power-of-two stride with two XORs (the leap-frog of rocrand_sobol32.h:140-159), writing
// 16-byte vectors where the row is aligned.  Distributions are applied in registers.
#include "common.hpp"
#include "dist.cuh"
#include "generators.hpp"
#include "launch.cuh"
#include "poisson.hpp"
#include "batch.hpp"
#include "sobol_dist.cuh"
#include "host_exec.hpp"
#include "sobol_tables.hpp"

#include <algorithm>
#include <type_traits>

namespace rb200
{

template<class W>
struct SobolCall
{
    const W*           vectors; // dims x B
    const W*           scramble; // scrambled table, read at flat index dim (nullptr: plain)
    unsigned char*     data;
    unsigned long long n;       // points per dimension
    unsigned long long chunk;   // points per block: a multiple of PPT * kBlock
    uint32_t           offset;
    SobolParams        p;
};

// Points per block for `dims` dimensions of n points each, blocks taking whole groups of
// `group` points, on a GPU holding `wave` resident blocks: among the block counts per
// dimension that fill k = 1 .. 64 waves (floor(k wave / dims) and one more), the one whose
// grid leaves the least of its last wave idle, the fewest blocks on ties.
inline unsigned long long sobol_chunk(unsigned long long n, unsigned long long dims, unsigned long long group,
                                      unsigned long long wave)
{
    if(wave == 0)
        wave = 1;
    const unsigned long long groups     = (n + group - 1) / group;
    unsigned long long       best_chunk = groups * group;
    unsigned long long       best_nb    = 1;
    double                   best_use   = 0.0;
    auto                     consider   = [&](unsigned long long b) {
        b                              = b < 1 ? 1 : (b > groups ? groups : b);
        const unsigned long long chunk = (groups + b - 1) / b * group;
        const unsigned long long nb    = (n + chunk - 1) / chunk;
        const unsigned long long waves = (nb * dims + wave - 1) / wave;
        const double             use   = static_cast<double>(nb * dims) / static_cast<double>(waves * wave);
        if(use > best_use + 1e-3 || (use > best_use - 1e-3 && nb < best_nb))
        {
            best_chunk = chunk;
            best_nb    = nb;
            best_use   = use > best_use ? use : best_use;
        }
    };
    for(unsigned long long k = 1; k <= 64; k++)
    {
        consider(k * wave / dims);
        consider(k * wave / dims + 1);
    }
    return best_chunk;
}

// Points per block of the 8-byte kinds that only store: 32 KiB of output, less where that
// leaves blocks out of the first wave.  Many short blocks in the order of memory keep the writes
// of the moment together: plain stores of 1 GiB run at 7.2-7.4 TB/s in blocks of 28 to 112 KiB
// and at 6.0-6.3 TB/s in one wave of long runs or grid strides, whose blocks drift apart.  64
// dimensions, 2^26 uniform fp64 on one B200, by whole waves -> by 32 KiB: Sobol32 150 -> 126 us,
// scrambled Sobol64 157 -> 116 (2^24: 62.8 -> 34.6).  The 4-byte kinds gain nothing or lose
// (uniform fp32 44.6 -> 49.3: a block's start costs them more) and keep whole waves.
inline unsigned long long sobol_store_chunk(unsigned long long group, unsigned long long spread, size_t size)
{
    const unsigned long long full = 32768 / (group * size);
    return std::max<unsigned long long>(1, std::min(full, spread)) * group;
}

template<SobolKind K>
constexpr bool kSobolStores = K == SobolKind::UINT || K == SobolKind::ULL || K == SobolKind::UCHAR
                              || K == SobolKind::USHORT || K == SobolKind::FLOAT || K == SobolKind::DOUBLE
                              || K == SobolKind::HALF;

// Forms of the kernel: whether a thread looks every step's direction vector up or keeps three of
// four in registers, and the blocks that an SM has to hold (0: as many as the registers leave).
// Registers pay for the 64-bit sequences, whose lookups are 8 bytes; the 32-bit kinds lose
// residency by them.  Measured on one B200, look up -> registers, the output buffer another one
// each call:
//  * Sobol32, 64 dimensions: 2^25 Poisson 97 -> 132 us, 2^24 half normals 70 -> 83; 1000
//    dimensions of 272 normals 6.2 -> 8.2;
//  * Sobol64, 64 dimensions x 2^20: normal fp32 289 -> 245 us, uint32 64 -> 56, uint8 77 -> 44.
// The kinds that are little more than a store need all eight blocks (with seven, 64 dimensions x
// 2^20 uint32 were cut into 16 long runs a row, 1024 streams of one wave, and took 86 us instead
// of 45), except Sobol32's uniform fp64, which the cap costs more than a block (2^21 values 8.4
// -> 6.6 us, 2^27 267 -> 246).  Poisson searches its table in shared memory, which residency
// hides (Sobol64, 2^24 values: 87 us with the transforms' registers, 58 without).  The fp64
// normals gain as much as they lose (Sobol32, 64 dimensions: 2^25 values 222 -> 205 us, 2^22 31.3
// -> 33.2) and keep the registers.
template<class W, SobolKind K>
constexpr bool kSobolLook = sizeof(W) == 4 && K != SobolKind::NORMAL_D && K != SobolKind::LOGNORMAL_D;
template<class W, SobolKind K>
constexpr unsigned kSobolBlocks = kSobolStores<K> ? (sizeof(W) == 4 && K == SobolKind::DOUBLE ? 0u : 8u)
                                                  : (kSobolLook<W, K> || K == SobolKind::POISSON ? 0u : 1u);

// The 8-byte kinds have the other form too (the lookup of Sobol64 with free registers, Sobol32's
// at eight blocks), for the calls that are not cut into short blocks of whole vectors.
template<class W, SobolKind K>
constexpr bool kSobolTwoForms = K == SobolKind::DOUBLE || (sizeof(W) == 8 && K == SobolKind::ULL);
template<class W, SobolKind K>
constexpr unsigned kSobolOtherBlocks = sizeof(W) == 4 ? 8u : 0u;

template<class W, SobolKind K, bool kLook, unsigned kBlocks>
__global__ void __launch_bounds__(kBlock, kBlocks) sobol_fill(SobolCall<W> a)
{
    using T                = typename SobolOut<K, W>::T;
    constexpr int      B   = 8 * sizeof(W);
    constexpr unsigned PPT = sizeof(T) >= 4 ? 4u : 16u / sizeof(T);
    // 64-bit index for Sobol64 (its engine counter is 64-bit), 32-bit for Sobol32.
    using I = W;

    __shared__ W v[B];
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t dim = blockIdx.y;
    if(threadIdx.x < B)
        v[threadIdx.x] = a.vectors[static_cast<size_t>(dim) * B + threadIdx.x];
    const double* cdf = nullptr;
    if constexpr(K == SobolKind::POISSON)
    {
        double* s = reinterpret_cast<double*>(smem);
        for(uint32_t k = threadIdx.x; k < a.p.size; k += blockDim.x)
            s[k] = a.p.cdf[k];
        cdf = s;
    }
    __syncthreads();

    const W            c      = a.scramble ? a.scramble[dim] : W(0);
    T*                 row    = reinterpret_cast<T*>(a.data) + static_cast<size_t>(dim) * a.n;
    // block x covers points [x chunk, (x + 1) chunk) of its dimension, its threads leap-frog
    // through them by the power-of-two stride PPT * kBlock
    constexpr unsigned long long stride = static_cast<unsigned long long>(PPT) * kBlock;
    constexpr uint32_t           lg     = PPT == 4 ? 10u : (PPT == 8 ? 11u : 12u); // log2(stride)
    static_assert((1ull << lg) == stride, "stride is a power of two");
    const unsigned long long begin = static_cast<unsigned long long>(blockIdx.x) * a.chunk;
    const unsigned long long end   = a.n < begin + a.chunk ? a.n : begin + a.chunk;
    unsigned long long       p     = begin + static_cast<unsigned long long>(threadIdx.x) * PPT;
    if(p >= end)
        return;
    const bool         vec_ok = (reinterpret_cast<uintptr_t>(row) % (PPT * sizeof(T))) == 0;

    // The engine starts at the 32-bit sum offset + p (sobol.hpp:191-196) and then counts in
    // its own width.
    I i = static_cast<I>(static_cast<uint32_t>(a.offset + static_cast<uint32_t>(p)));
    W x = 0;
    {
        const I g = i ^ (i >> 1);
#pragma unroll
        for(int b = 0; b < B; b++)
            if((g >> b) & 1)
                x ^= v[b];
    }
    // Point i to i + 1 flips the direction vector of i's lowest zero bit: number 0, 1, 0 after
    // i = 0, 1, 2 (mod 4), and one to look up after i = 3 (mod 4).  A thread's points start at the
    // same residue every time (strides are multiples of 4), so of four steps three have their
    // vector in a register unless kLook has every one looked up.
    const unsigned residue  = static_cast<unsigned>(i) & 3u;
    const W        v0 = v[0], v1 = v[1], vl = v[lg - 1];
    for(; p < end; p += stride)
    {
        T out[PPT];
        W look[PPT / 4];
        if constexpr(!kLook)
        {
#pragma unroll
            for(unsigned j = 0; j < PPT / 4; j++)
                look[j] = v[rzb(static_cast<I>((i + 4 * j) | 3u))];
        }
        W xx = x;
#pragma unroll
        for(unsigned k = 0; k < PPT; k++)
        {
            out[k] = sobol_apply<K, W>(xx ^ c, a.p, cdf);
            if constexpr(kLook)
            {
                xx ^= v[rzb(static_cast<I>(i + k))];
            }
            else
            {
                const unsigned at = (residue + k) & 3u;
                xx ^= at == 3u ? look[k / 4] : (at == 1u ? v1 : v0);
            }
        }
        if(vec_ok && p + PPT <= a.n)
        {
            constexpr unsigned VB = PPT * sizeof(T);
            if constexpr(VB == 16)
            {
                uint4 w;
                memcpy(&w, out, 16);
                __stcs(reinterpret_cast<uint4*>(row + p), w);
            }
            else
            {
                static_assert(VB == 32, "vector");
                uint4 w[2];
                memcpy(w, out, 32);
                __stcs(reinterpret_cast<uint4*>(row + p), w[0]);
                __stcs(reinterpret_cast<uint4*>(row + p) + 1, w[1]);
            }
        }
        else
        {
            for(unsigned k = 0; k < PPT && p + k < a.n; k++)
                row[p + k] = out[k];
        }
        // leap-frog by the power-of-two stride 2^lg: Gray-code bit lg-1 flips, and the bit of
        // the lowest zero of i above the low lg bits (rocrand_sobol32.h:140-159)
        x ^= vl;
        x ^= v[rzb(static_cast<I>(i | static_cast<I>(stride - 1)))];
        i += static_cast<I>(stride);
    }
}

// ---------------------------------------------------------------------------------------

template<bool kIs64, bool kScrambled>
class SobolGenerator final : public rocrand_generator_base_type
{
    using W = std::conditional_t<kIs64, unsigned long long, uint32_t>;

public:
    bool set_host_execution() override
    {
        m_host_exec = true;
        m_poisson.set_host();
        return true;
    }
    rocrand_rng_type type() const override
    {
        if(kIs64)
            return kScrambled ? ROCRAND_RNG_QUASI_SCRAMBLED_SOBOL64 : ROCRAND_RNG_QUASI_SOBOL64;
        return kScrambled ? ROCRAND_RNG_QUASI_SCRAMBLED_SOBOL32 : ROCRAND_RNG_QUASI_SOBOL32;
    }
    rocrand_status init() override
    {
        if(!m_initialized)
        {
            // the Poisson tables are allocated here, as the reference's generators do in init(), so
            // that a generate call recorded by a stream capture allocates nothing
            const rocrand_status st = m_poisson.reserve();
            if(st != ROCRAND_STATUS_SUCCESS)
                return st;
            // likewise the device tables every generate call reads (uploaded once per device)
            lr::Table lt;
            if(!m_host_exec
               && (sobol_device_vectors(kIs64, kScrambled) == nullptr || !logf_replay_device(lt)))
                return ROCRAND_STATUS_ALLOCATION_FAILED;
            m_current     = static_cast<uint32_t>(m_offset); // 32-bit counter (sobol.hpp:604)
            m_initialized = true;
        }
        return ROCRAND_STATUS_SUCCESS;
    }
    rocrand_status set_seed(unsigned long long) override { return ROCRAND_STATUS_SUCCESS; }
    rocrand_status set_offset(unsigned long long offset) override
    {
        m_offset      = offset;
        m_initialized = false;
        return ROCRAND_STATUS_SUCCESS;
    }
    rocrand_status set_order(rocrand_ordering order) override
    {
        if(order != ROCRAND_ORDERING_QUASI_DEFAULT)
            return ROCRAND_STATUS_OUT_OF_RANGE;
        m_initialized = false;
        return ROCRAND_STATUS_SUCCESS;
    }
    rocrand_status set_dimensions(unsigned int dims) override
    {
        if(dims < 1 || dims > kSobolDims)
            return ROCRAND_STATUS_OUT_OF_RANGE;
        m_dims        = dims;
        m_initialized = false;
        return ROCRAND_STATUS_SUCCESS;
    }

    rocrand_status batch_descriptor(uint32_t dist, double p0, double p1, void* data, size_t n,
                                    BatchReq& r, cudaStream_t stream) override
    {
        if(kIs64 || kScrambled || m_dims != 1)
            return ROCRAND_STATUS_TYPE_ERROR;
        rocrand_status st = init();
        if(st != ROCRAND_STATUS_SUCCESS)
            return st;
        r              = BatchReq{};
        r.kind         = BK_SOBOL32;
        r.sobol_offset = m_current;
        r.sobol_v      = static_cast<const uint32_t*>(sobol_device_vectors(false, false));
        if(r.sobol_v == nullptr)
            return ROCRAND_STATUS_ALLOCATION_FAILED;
        st = batch_set_dist(r, dist, p0, p1, stream);
        if(st == ROCRAND_STATUS_SUCCESS)
            st = batch_layout(r, data, n);
        if(st != ROCRAND_STATUS_SUCCESS)
            return st;
        m_current += static_cast<uint32_t>(n);
        return ROCRAND_STATUS_SUCCESS;
    }

    rocrand_status generate(void* data, size_t n, Dist d, const DistParams& dp) override
    {
        if(!kIs64 && d == Dist::U64)
            return ROCRAND_STATUS_TYPE_ERROR;
        if(n % m_dims != 0)
            return ROCRAND_STATUS_LENGTH_NOT_MULTIPLE;
        rocrand_status st = init();
        if(st != ROCRAND_STATUS_SUCCESS)
            return st;
        if(data == nullptr)
            return ROCRAND_STATUS_SUCCESS;
        if(reinterpret_cast<uintptr_t>(data) % dist_elem_size(d) != 0)
            return ROCRAND_STATUS_LENGTH_NOT_MULTIPLE;
        SobolParams p{};
        p.mean_f = dp.mean_f;
        p.std_f  = dp.std_f;
        p.mean_d = dp.mean_d;
        p.std_d  = dp.std_d;
        if(d == Dist::NORMAL_F16 || d == Dist::LOGNORMAL_F16)
        {
            p.mean_f = __half2float(__ushort_as_half(dp.mean_h));
            p.std_f  = __half2float(__ushort_as_half(dp.std_h));
        }
        p.cdf         = dp.cdf;
        p.size        = dp.size;
        p.offset      = dp.offset;
        p.lambda      = dp.lambda;
        p.sqrt_lambda = dp.sqrt_lambda;
        if(!m_host_exec
           && (d == Dist::NORMAL_F32 || d == Dist::LOGNORMAL_F32 || d == Dist::NORMAL_F16
               || d == Dist::LOGNORMAL_F16)
           && !logf_replay_device(p.logf))
            return ROCRAND_STATUS_INTERNAL_ERROR;
        switch(d)
        {
            case Dist::U32: st = launch<SobolKind::UINT>(data, n, p); break;
            case Dist::U64: st = launch<SobolKind::ULL>(data, n, p); break;
            case Dist::U8: st = launch<SobolKind::UCHAR>(data, n, p); break;
            case Dist::U16: st = launch<SobolKind::USHORT>(data, n, p); break;
            case Dist::F32: st = launch<SobolKind::FLOAT>(data, n, p); break;
            case Dist::F64: st = launch<SobolKind::DOUBLE>(data, n, p); break;
            case Dist::F16: st = launch<SobolKind::HALF>(data, n, p); break;
            case Dist::NORMAL_F32: st = launch<SobolKind::NORMAL_F>(data, n, p); break;
            case Dist::NORMAL_F64: st = launch<SobolKind::NORMAL_D>(data, n, p); break;
            case Dist::NORMAL_F16: st = launch<SobolKind::NORMAL_H>(data, n, p); break;
            case Dist::LOGNORMAL_F32: st = launch<SobolKind::LOGNORMAL_F>(data, n, p); break;
            case Dist::LOGNORMAL_F64: st = launch<SobolKind::LOGNORMAL_D>(data, n, p); break;
            case Dist::LOGNORMAL_F16: st = launch<SobolKind::LOGNORMAL_H>(data, n, p); break;
            case Dist::POISSON:
                st = dp.huge ? launch<SobolKind::POISSON_HUGE>(data, n, p)
                             : launch<SobolKind::POISSON>(data, n, p);
                break;
            default: return ROCRAND_STATUS_TYPE_ERROR;
        }
        if(st == ROCRAND_STATUS_SUCCESS)
            m_current += static_cast<uint32_t>(n / m_dims);
        return st;
    }

    rocrand_status generate_poisson(unsigned int* data, size_t n, double lambda) override
    {
        DistParams p;
        // The quasi-random generators use the CDF form of the table (sobol.hpp:498-499).
        const rocrand_status st = m_poisson.get(lambda, m_stream, true, p);
        if(st != ROCRAND_STATUS_SUCCESS)
            return st;
        return generate(data, n, Dist::POISSON, p);
    }

private:
    // A launch shape (kind, points per dimension, shared memory, dimensions, rows of whole
    // vectors) and what serves it, chosen once per shape.
    using Kernel = void (*)(SobolCall<W>);
    struct Plan
    {
        Kernel             kind   = nullptr;
        unsigned long long n      = 0;
        size_t             smem   = 0;
        unsigned int       dims   = 0;
        bool               whole  = false;
        Kernel             kernel = nullptr;
        unsigned long long chunk  = 0; // points per block
    };

    template<SobolKind K>
    Plan plan(Kernel kind, unsigned long long n, size_t smem, bool whole) const
    {
        using T                            = typename SobolOut<K, W>::T;
        constexpr unsigned           PPT   = sizeof(T) >= 4 ? 4u : 16u / sizeof(T);
        constexpr unsigned long long group = static_cast<unsigned long long>(PPT) * kBlock;
        const auto wave_of = [&](Kernel k) {
            return static_cast<unsigned long long>(device_info().sm_count)
                   * blocks_per_sm(reinterpret_cast<const void*>(k), smem);
        };
        Plan r{kind, n, smem, m_dims, whole, kind, 0};
        if constexpr(kSobolTwoForms<W, K>)
        {
            // Short blocks, unless one group a block would be one wave and a part of the next
            // (Sobol64, 2^21 uint64: 10.4 us that way, 7.2 by whole waves of the other form; 2^22:
            // 10.6, 11.1), or the rows are not made of whole vectors and there are many (1000
            // dimensions x 8389 points of Sobol64 uniform fp64: 37 us, 29; 3 dimensions of as many
            // points in all: 33, 40).  Sobol32 keeps short blocks in the first case (6.6 us,
            // 8.4); its other form is the faster one where vectors are split (64 dimensions x
            // 32769 points of uniform fp64: 12.4 us, 10.5).
            constexpr auto           other  = sobol_fill<W, K, true, kSobolOtherBlocks<W, K>>;
            if(sizeof(W) == 4 && !whole)
                r.kernel = other;
            const unsigned long long spread = (n + group - 1) / group * m_dims / wave_of(r.kernel);
            const bool               waves  = whole ? sizeof(W) == 8 && spread == 1 : m_dims >= 128 && spread >= 2;
            if(sizeof(W) == 8 && waves)
                r.kernel = other;
            r.chunk = waves ? sobol_chunk(n, m_dims, group, wave_of(r.kernel))
                            : sobol_store_chunk(group, spread, sizeof(T));
        }
        else
        {
            r.chunk = sobol_chunk(n, m_dims, group, wave_of(kind));
        }
        return r;
    }

    template<SobolKind K>
    rocrand_status launch(void* data, size_t n, const SobolParams& p)
    {
        using T                = typename SobolOut<K, W>::T;
        constexpr unsigned PPT = sizeof(T) >= 4 ? 4u : 16u / sizeof(T);
        if(m_host_exec)
            return run_host<K>(data, n, p);
        const W*           vec = static_cast<const W*>(sobol_device_vectors(kIs64, kScrambled));
        if(vec == nullptr)
            return ROCRAND_STATUS_ALLOCATION_FAILED;
        const unsigned long long N = n / m_dims;
        if(N == 0)
            return ROCRAND_STATUS_SUCCESS;
        SobolCall<W> a;
        a.vectors  = vec;
        a.scramble = kScrambled ? vec : nullptr;
        a.data     = static_cast<unsigned char*>(data);
        a.n        = N;
        a.offset   = m_current;
        a.p        = p;
        // blocks per dimension: whole groups of PPT * kBlock points each, as many as fill the
        // GPU's resident blocks in nearly whole waves, or short blocks (the 8-byte kinds that
        // only store)
        const size_t   smem   = K == SobolKind::POISSON ? p.size * sizeof(double) : 0;
        constexpr auto kernel = sobol_fill<W, K, kSobolLook<W, K>, kSobolBlocks<W, K>>;
        const bool     whole  = reinterpret_cast<uintptr_t>(data) % (PPT * sizeof(T)) == 0
                           && (m_dims == 1 || N * sizeof(T) % (PPT * sizeof(T)) == 0);
        if(m_plan.kind != kernel || m_plan.n != N || m_plan.smem != smem || m_plan.dims != m_dims
           || m_plan.whole != whole)
            m_plan = plan<K>(kernel, N, smem, whole);
        a.chunk                     = m_plan.chunk;
        const unsigned long long nb = (N + a.chunk - 1) / a.chunk;
        m_plan.kernel<<<dim3(static_cast<unsigned>(nb), m_dims), kBlock, smem, m_stream>>>(a);
        return launch_status();
    }

    // The same output on the host (host generators without a GPU): point i of dimension d is
    // the XOR of d's direction vectors over the set bits of Gray(i), with i counted from the
    // 32-bit start as the kernel counts it, and the distribution applied to it.
    template<SobolKind K>
    rocrand_status run_host(void* data, size_t n, const SobolParams& p)
    {
        using T                     = typename SobolOut<K, W>::T;
        using I                     = W;
        constexpr int         B     = 8 * sizeof(W);
        const SobolTables&    t     = sobol_tables();
        if(!t.ok)
            return ROCRAND_STATUS_INTERNAL_ERROR;
        const W* const vec = reinterpret_cast<const W*>(
            kIs64 ? static_cast<const void*>(kScrambled ? t.sv64.data() : t.v64.data())
                  : static_cast<const void*>(kScrambled ? t.sv32.data() : t.v32.data()));
        const unsigned long long N = n / m_dims;
        const uint32_t           offset = m_current;
        host_parallel_for(static_cast<unsigned long long>(m_dims) * N,
                          [&](unsigned long long b0, unsigned long long b1) {
            while(b0 < b1)
            {
                const unsigned long long dim = b0 / N, p0 = b0 % N;
                const unsigned long long p1  = std::min<unsigned long long>(N, p0 + (b1 - b0));
                const W* const v   = vec + dim * B;
                const W        c   = kScrambled ? vec[dim] : W(0);
                T* const       row = static_cast<T*>(data) + dim * N;
                I              i   = static_cast<I>(static_cast<uint32_t>(offset + static_cast<uint32_t>(p0)));
                W              x   = 0;
                const I        g   = i ^ (i >> 1);
                for(int bit = 0; bit < B; bit++)
                    if((g >> bit) & 1)
                        x ^= v[bit];
                for(unsigned long long q = p0; q < p1; q++)
                {
                    row[q] = sobol_apply<K, W>(x ^ c, p, p.cdf);
                    x ^= v[rzb(i)];
                    i++;
                }
                b0 += p1 - p0;
            }
        });
        return ROCRAND_STATUS_SUCCESS;
    }

    unsigned long long m_offset      = 0;
    uint32_t           m_current     = 0;
    unsigned int       m_dims        = 1;
    bool               m_initialized = false;
    PoissonCache       m_poisson;
    Plan               m_plan;
};

rocrand_generator_base_type* make_sobol(rocrand_rng_type t)
{
    switch(t)
    {
        case ROCRAND_RNG_QUASI_DEFAULT:
        case ROCRAND_RNG_QUASI_SOBOL32: return new SobolGenerator<false, false>();
        case ROCRAND_RNG_QUASI_SCRAMBLED_SOBOL32: return new SobolGenerator<false, true>();
        case ROCRAND_RNG_QUASI_SOBOL64: return new SobolGenerator<true, false>();
        case ROCRAND_RNG_QUASI_SCRAMBLED_SOBOL64: return new SobolGenerator<true, true>();
        default: return nullptr;
    }
}

} // namespace rb200
