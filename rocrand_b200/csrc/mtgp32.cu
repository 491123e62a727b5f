// mtgp32.cu -- MTGP32: 512 block generators, each its own published recurrence.
//
// Output contract (library/src/rng/mtgp32.hpp:232-305, rocrand_mtgp32.h): generator b
// (one of 512, config/config_defaults.hpp:48-52) belongs to block b of 256 threads.  One
// block step advances the generator by 256 values: thread t computes
//   r = para_rec(s[k+t], s[k+t+1], s[k+t+pos]),  s[k+t+351] = r,  out = temper(r, s[k+t+pos-1])
// on a 1024-word state ring (k = the ring offset, then k += 256).  Output vector j is thread
// j % 256 of generator (j / 256) % 512 in round j / 131072; a distribution call takes its iw
// inputs from iw successive steps.  After the full rounds every generator steps once more
// when the last round is partial (writing only the vectors that exist), and once more when
// the call has a head or tail, which the threads at vector indices vec_n_up and
// vec_n_up + 1 write.  State and offset carry over to the next call.
//
// B200 layout: the rings and offsets of the 512 generators live in HBM (2 MiB); each block
// keeps its ring in shared memory for the whole call (one __syncthreads per step: a step's
// reads stop short of its first write, the next step reads what it wrote), its parameter
// set in registers and shared memory.  The parameter sets are the published MTGP32 11213
// dynamic-creator sets (rocrand_b200/data/mtgp32_params.bin, embedded by mtgp32_data.S).
#include "common.hpp"
#include "dist.cuh"
#include "generators.hpp"
#include "host_exec.hpp"
#include "launch.cuh"
#include "mtgp32_params.hpp"
#include "stateful_engines.cuh"

#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

extern "C" const unsigned char rb200_mtgp32_params_begin[];
extern "C" const unsigned char rb200_mtgp32_params_end[];

namespace rb200
{
namespace
{

constexpr int      kMtgpState = 1024;
constexpr int      kMtgpMask  = 1023;

struct MtgpArgs
{
    uint32_t*          rings;   // [512][1024]
    int*               offsets; // [512]
    const uint32_t*    params;  // [512][36]
    unsigned char*     data;
    unsigned char*     vec;
    unsigned long long n, vec_n, vec_n_down, vec_n_up;
    uint32_t           head, tail;
};

// Units a thread takes in one iteration of the main loop: whole turns of four block steps, and
// for the long transforms the units they run side by side (four fp64 Box-Muller chains, packed
// pairs of fp32 or half ones).
template<class F>
constexpr unsigned kMtgpUnits = F::iw == 1 ? 4u : F::iw == 2 ? 2u : 4u;

// Words after the ring that repeat its first ones: a step reads up to pos + 255 words ahead of
// its offset, pos <= kMtgpReach, the last of the four offsets being 768.
constexpr int kMtgpMirror = kMtgpReach + 1;

// The ring in shared memory starts at the call's offset, so that the four block steps of a turn
// work at the constant offsets 0, 256, 512 and 768 and every address is the thread's base plus
// an immediate.  Only step 2 writes across the ring's end: its last 95 words go to the mirror,
// where step 3 reads them, and to the start.
//
// Bound: shared memory and the step's own latency.  A value takes seven 4-byte accesses (four
// ring words, two tables, one store) and one global store, 8 of the SM's memory cycles per 32
// values: 66.7 us for 2^26 values on an SM with four of the 512 generators; the rest is the
// chain of a step (load, table, store, barrier), which four blocks overlap only in part.  With
// the offsets wrapped by masks at run time, each step was 36 instructions a value.  2^26 values
// on one B200, before -> now (the transforms' own changes included): uniform fp32 113 -> 97..101
// us, uniform fp64 273 -> 197, normal fp32 202 -> 151, fp64 541 -> 467, Poisson 167 -> 130.
template<class F>
__global__ void __launch_bounds__(kMtgpBlock, 4) mtgp_fill(MtgpArgs a, F fw)
{
    // 4 blocks of 256 threads per SM (at most 64 registers): all 512 block generators resident
    // at once on 148 SMs
    __shared__ uint32_t        s[kMtgpState + kMtgpMirror];
    __shared__ uint32_t        tbl[16], tmp[16];
    extern __shared__ unsigned char smem[];
    const F                    f = stage_table(fw, smem);
    const uint32_t             b = blockIdx.x, t = threadIdx.x;
    const uint32_t*            p = a.params + b * kMtgpWords;
    // The ring's words and its offset are read side by side: reading the words at the offset
    // made every call wait for memory twice (2^18 values on one B200: uniform half 6.15 -> 4.11
    // us, uint 5.13 -> 4.12, Poisson 6.16 -> 4.13).
    constexpr int              kLoads = kMtgpState / static_cast<int>(kMtgpBlock);
    uint32_t                   ring[kLoads];
#pragma unroll
    for(int i = 0; i < kLoads; i++)
        ring[i] = a.rings[b * kMtgpState + i * kMtgpBlock + t];
    const int k = a.offsets[b];
#pragma unroll
    for(int i = 0; i < kLoads; i++)
        s[(i * static_cast<int>(kMtgpBlock) + static_cast<int>(t) - k) & kMtgpMask] = ring[i];
    if(t < 16)
    {
        tbl[t] = p[3 + t];
        tmp[t] = p[19 + t];
    }
    const int      pos = static_cast<int>(p[0]);
    const uint32_t sh1 = p[1], sh2 = p[2], mask = p[35];
    uint32_t*      at  = s + t;           // this thread's word of the step at offset 0
    uint32_t*      far = s + t + pos - 1; // and its pos - 1 (tempering) and pos words
    __syncthreads();

    // entry (v & 15) of a 16-word table
    auto entry = [](const uint32_t* table, uint32_t v) {
        return *reinterpret_cast<const uint32_t*>(reinterpret_cast<const unsigned char*>(table) + ((v << 2) & 60u));
    };
    // one block step at ring offset 256 ph: this thread's value, then every thread's writes
    // become visible
    auto step = [&](int ph) -> uint32_t {
        const int o  = static_cast<int>(kMtgpBlock) * ph;
        uint32_t  x  = (at[o] & mask) ^ at[o + 1];
        uint32_t  tt = far[o];
        uint32_t  y  = far[o + 1];
        y            = x ^ (x << sh1) ^ (y >> sh2);
        const uint32_t r = y ^ entry(tbl, y);
        if(ph == 2)
        {
            at[o + kMtgpN] = r; // the last 95 threads': words of the mirror
            if(t >= kMtgpState - (2 * kMtgpBlock + kMtgpN))
                at[o + kMtgpN - kMtgpState] = r;
        }
        else
        {
            at[ph == 3 ? o + kMtgpN - kMtgpState : o + kMtgpN] = r;
        }
        tt ^= tt >> 16;
        tt ^= tt >> 8;
        __syncthreads();
        return r ^ entry(tmp, tt);
    };

    using T                      = typename F::T;
    constexpr unsigned ow        = F::ow;
    constexpr unsigned VB        = ow * sizeof(T);
    constexpr unsigned long long str = static_cast<unsigned long long>(kMtgpGens) * kMtgpBlock;
    unsigned long long index     = static_cast<unsigned long long>(b) * kMtgpBlock + t;
    constexpr unsigned U         = kMtgpUnits<F>;
    static_assert(U * F::iw % 4 == 0, "whole turns");
    // index < vec_n_down and index < vec_n_up are the same in the whole block (both are
    // multiples of 256), so every thread takes every step
    unsigned char* dst = a.vec + index * VB;
    for(; index + (U - 1) * str < a.vec_n_down; index += U * str, dst += U * str * VB)
    {
        uint32_t in[U][F::iw];
        T        o[U][ow];
        // a long transform after all steps, with no branch between its units, so that their
        // chains interleave instead of each waiting out its own latency
#pragma unroll
        for(unsigned u = 0; u < U; u++)
        {
#pragma unroll
            for(unsigned i = 0; i < F::iw; i++)
                in[u][i] = step((u * F::iw + i) % 4);
            if constexpr(!long_transform<F>::value)
            {
                f(in[u], o[u]);
                store_small(dst + u * str * VB, o[u]);
            }
        }
        if constexpr(long_transform<F>::value)
        {
#pragma unroll
            for(unsigned u = 0; u < U; u += 2)
                apply_pair(f, in[u], in[u + 1], o[u], o[u + 1]);
#pragma unroll
            for(unsigned u = 0; u < U; u++)
                store_small(dst + u * str * VB, o[u]);
        }
    }
    // the rest of the rounds, the round that is not whole, and the head and tail: a step's
    // offset at run time, the next turn's first step on
    uint32_t in[F::iw];
    T        out[ow];
    int      ph  = 0;
    auto     gen = [&]() {
#pragma unroll 1
        for(unsigned i = 0; i < F::iw; i++)
        {
            const uint32_t v = step(ph);
            ph               = (ph + 1) & 3;
#pragma unroll
            for(unsigned j = 0; j < F::iw; j++)
                in[j] = i == j ? v : in[j];
        }
        f(in, out);
    };
    while(index < a.vec_n_down)
    {
        gen();
        store_small(a.vec + index * VB, out);
        index += str;
    }
    if(index < a.vec_n_up)
    {
        gen();
        if(index < a.vec_n)
            store_small(a.vec + index * VB, out);
        index += str;
    }
    if(ow > 1 && (a.head > 0 || a.tail > 0))
    {
        gen();
        T* data = reinterpret_cast<T*>(a.data);
        if(index == a.vec_n_up)
            for(unsigned o = 0; o < a.head; o++)
                data[o] = out[o];
        if(index == a.vec_n_up + 1)
            for(unsigned o = 0; o < a.tail; o++)
                data[a.n - a.tail + o] = out[o];
    }
    // whole turns leave the offset where it was
    for(int i = static_cast<int>(t); i < kMtgpState; i += kMtgpBlock)
        a.rings[b * kMtgpState + ((k + i) & kMtgpMask)] = s[i];
    if(t == 0)
        a.offsets[b] = (k + static_cast<int>(kMtgpBlock) * ph) & kMtgpMask;
}

// mtgp_fill on the host (CPU path of the host generators): generator b's 256 threads take
// each block step in thread order -- a step's reads end before its first written word, so
// the order within a step does not change a value -- then every thread applies the
// distribution to its inputs and writes by mtgp_fill's rules.  Generators are independent.
template<class F>
void mtgp_fill_host(const MtgpArgs& a, const F& f)
{
    using T                      = typename F::T;
    constexpr unsigned iw        = F::iw;
    constexpr unsigned ow        = F::ow;
    constexpr unsigned VB        = ow * sizeof(T);
    const unsigned long long str = static_cast<unsigned long long>(kMtgpGens) * kMtgpBlock;
    host_parallel_for(
        kMtgpGens,
        [&](unsigned long long b0, unsigned long long b1) {
            std::vector<uint32_t> vals(static_cast<size_t>(iw) * kMtgpBlock);
            std::vector<T>        outs(static_cast<size_t>(ow) * kMtgpBlock);
            for(unsigned long long b = b0; b < b1; b++)
            {
                uint32_t*       s    = a.rings + b * kMtgpState;
                const uint32_t* p    = a.params + b * kMtgpWords;
                const int       pos  = static_cast<int>(p[0]);
                const uint32_t  sh1 = p[1], sh2 = p[2], mask = p[35];
                const uint32_t* tbl  = p + 3;
                const uint32_t* tmp  = p + 19;
                int             k    = a.offsets[b];
                // iw block steps, then the distribution on each thread's inputs
                auto gen = [&]() {
                    for(unsigned i = 0; i < iw; i++)
                    {
                        for(uint32_t t = 0; t < kMtgpBlock; t++)
                        {
                            uint32_t x = (s[(k + t) & kMtgpMask] & mask) ^ s[(k + t + 1) & kMtgpMask];
                            uint32_t y = s[(k + t + pos) & kMtgpMask];
                            x ^= x << sh1;
                            y                               = x ^ (y >> sh2);
                            const uint32_t r                = y ^ tbl[y & 0x0f];
                            s[(k + t + kMtgpN) & kMtgpMask] = r;
                            uint32_t tt                     = s[(k + t + pos - 1) & kMtgpMask];
                            tt ^= tt >> 16;
                            tt ^= tt >> 8;
                            vals[t * iw + i] = r ^ tmp[tt & 0x0f];
                        }
                        k = (k + kMtgpBlock) & kMtgpMask;
                    }
                    for(uint32_t t = 0; t < kMtgpBlock; t++)
                        f(&vals[t * iw], &outs[t * ow]);
                };
                unsigned long long index = b * kMtgpBlock; // thread 0's vector index
                while(index < a.vec_n_down)
                {
                    gen();
                    std::memcpy(a.vec + index * VB, outs.data(), VB * kMtgpBlock);
                    index += str;
                }
                if(index < a.vec_n_up)
                {
                    gen();
                    for(uint32_t t = 0; t < kMtgpBlock; t++)
                        if(index + t < a.vec_n)
                            std::memcpy(a.vec + (index + t) * VB, &outs[t * ow], VB);
                    index += str;
                }
                if(ow > 1 && (a.head > 0 || a.tail > 0))
                {
                    gen();
                    T* data = reinterpret_cast<T*>(a.data);
                    for(uint32_t t = 0; t < kMtgpBlock; t++)
                    {
                        if(index + t == a.vec_n_up)
                            for(unsigned o = 0; o < a.head; o++)
                                data[o] = outs[t * ow + o];
                        if(index + t == a.vec_n_up + 1)
                            for(unsigned o = 0; o < a.tail; o++)
                                data[a.n - a.tail + o] = outs[t * ow + o];
                    }
                }
                a.offsets[b] = k;
            }
        },
        2);
}

// Parameter sets on each device, uploaded once.
const uint32_t* device_params(const uint32_t* host_params)
{
    static std::mutex                   mu;
    static std::vector<const uint32_t*> ptr(64, nullptr);
    const int                           dev = device_info().device;
    std::lock_guard<std::mutex>         lock(mu);
    if(ptr[dev])
        return ptr[dev];
    constexpr size_t bytes = sizeof(uint32_t) * kMtgpWords * kMtgpGens;
    void*            d     = nullptr;
    if(cudaMalloc(&d, bytes) != cudaSuccess)
        return nullptr;
    if(cudaMemcpy(d, host_params, bytes, cudaMemcpyHostToDevice) != cudaSuccess)
    {
        cudaFree(d);
        return nullptr;
    }
    ptr[dev] = static_cast<const uint32_t*>(d);
    return ptr[dev];
}

class Mtgp32Generator final : public PseudoGeneratorBase
{
public:
    ~Mtgp32Generator() override
    {
        if(m_rings != nullptr)
            cudaFree(m_rings);
    }

    bool set_host_execution() override { return enable_host(); }

    rocrand_rng_type type() const override { return ROCRAND_RNG_PSEUDO_MTGP32; }

    // mtgp32.hpp:389-393: MTGP32 has no offset
    rocrand_status set_offset(unsigned long long offset) override
    {
        (void)offset;
        return ROCRAND_STATUS_TYPE_ERROR;
    }

    // mtgp32.hpp:395-416 (device generator: DYNAMIC accepted)
    rocrand_status set_order(rocrand_ordering order) override
    {
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

    rocrand_status init() override
    {
        if(m_initialized)
            return ROCRAND_STATUS_SUCCESS;
        // the Poisson tables are allocated here, as the reference's generators do in init(), so
        // that a generate call recorded by a stream capture allocates nothing
        if(m_poisson.reserve() != ROCRAND_STATUS_SUCCESS)
            return ROCRAND_STATUS_ALLOCATION_FAILED;
        const uint32_t* const host_params = mtgp_parameter_sets(
            rb200_mtgp32_params_begin, static_cast<size_t>(rb200_mtgp32_params_end - rb200_mtgp32_params_begin));
        if(host_params == nullptr)
            return ROCRAND_STATUS_INTERNAL_ERROR;
        m_params = m_host_exec ? host_params : device_params(host_params);
        if(m_params == nullptr)
            return ROCRAND_STATUS_ALLOCATION_FAILED;
        constexpr size_t kRingWords = static_cast<size_t>(kMtgpGens) * kMtgpState;
        if(m_rings == nullptr && !m_host_exec)
        {
            if(cudaMalloc(&m_rings, sizeof(uint32_t) * kRingWords + sizeof(int) * kMtgpGens)
               != cudaSuccess)
            {
                m_rings = nullptr;
                return ROCRAND_STATUS_ALLOCATION_FAILED;
            }
        }
        // rocrand_make_state_mtgp32 / rocrand_mtgp32_init_state on the host (2 MiB)
        std::vector<uint32_t>    rings(kRingWords, 0u);
        const unsigned long long seed = m_seed ^ (m_seed >> 32);
        for(uint32_t i = 0; i < kMtgpGens; i++)
        {
            const uint32_t* tbl    = host_params + i * kMtgpWords + 3;
            const uint32_t  hidden = tbl[4] ^ (tbl[8] << 16);
            uint32_t        tmp    = hidden;
            tmp += tmp >> 16;
            tmp += tmp >> 8;
            uint32_t* s = rings.data() + static_cast<size_t>(i) * kMtgpState;
            for(int k = 0; k < kMtgpN; k++)
                s[k] = (tmp & 0xffu) * 0x01010101u;
            s[0] = static_cast<uint32_t>(seed) + i + 1u;
            s[1] = hidden;
            for(uint32_t k = 1; k < static_cast<uint32_t>(kMtgpN); k++)
                s[k] ^= 1812433253u * (s[k - 1] ^ (s[k - 1] >> 30)) + k;
        }
        if(m_host_exec)
        {
            // the host copy: rings, then the 512 ring offsets
            m_hrings.assign(kRingWords + kMtgpGens, 0u);
            std::memcpy(m_hrings.data(), rings.data(), sizeof(uint32_t) * kRingWords);
            m_initialized = true;
            return ROCRAND_STATUS_SUCCESS;
        }
        // pageable sources: the copies have read them when cudaMemcpyAsync returns
        if(cudaMemcpyAsync(m_rings, rings.data(), sizeof(uint32_t) * kRingWords,
                           cudaMemcpyHostToDevice, m_stream)
               != cudaSuccess
           || cudaMemsetAsync(m_rings + kRingWords, 0, sizeof(int) * kMtgpGens, m_stream)
                  != cudaSuccess)
            return ROCRAND_STATUS_INTERNAL_ERROR;
        m_initialized = true;
        return ROCRAND_STATUS_SUCCESS;
    }

    rocrand_status generate(void* data, size_t n, Dist d, const DistParams& p) override
    {
        if(d == Dist::U64)
            return ROCRAND_STATUS_TYPE_ERROR;
        rocrand_status st = init();
        if(st != ROCRAND_STATUS_SUCCESS)
            return st;
        if(data == nullptr)
            return ROCRAND_STATUS_SUCCESS;
        const size_t tsize = dist_elem_size(d);
        if(reinterpret_cast<uintptr_t>(data) % tsize != 0)
            return ROCRAND_STATUS_LENGTH_NOT_MULTIPLE;
        return with_functor(d, p, [&](auto f) -> rocrand_status { return run(f, data, n, tsize); });
    }

    rocrand_status generate_poisson(unsigned int* data, size_t n, double lambda) override
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

private:
    template<class F>
    rocrand_status run(const F& f, void* data, size_t n, size_t tsize)
    {
        constexpr unsigned ow   = F::ow;
        const uintptr_t    addr = reinterpret_cast<uintptr_t>(data);
        const size_t       mis  = (ow - addr / tsize % ow) % ow;
        MtgpArgs           a;
        uint32_t*          rings = m_host_exec ? m_hrings.data() : m_rings;
        a.rings      = rings;
        a.offsets    = reinterpret_cast<int*>(rings + static_cast<size_t>(kMtgpGens) * kMtgpState);
        a.params     = m_params;
        a.head       = static_cast<uint32_t>(n < mis ? n : mis);
        a.tail       = static_cast<uint32_t>((n - a.head) % ow);
        a.vec_n      = (n - a.head) / ow;
        a.n          = n;
        a.data       = static_cast<unsigned char*>(data);
        a.vec        = a.data + mis * tsize;
        const unsigned long long rem = a.vec_n % kMtgpBlock;
        a.vec_n_down = a.vec_n - rem;
        a.vec_n_up   = rem == 0 ? a.vec_n_down : a.vec_n_down + kMtgpBlock;
        // every call steps every generator (mtgp32.hpp:268-305), even with nothing to write
        if(m_host_exec)
        {
            mtgp_fill_host(a, f);
            return ROCRAND_STATUS_SUCCESS;
        }
        const size_t smem = table_smem_bytes(f);
        mtgp_fill<F><<<kMtgpGens, kMtgpBlock, smem, m_stream>>>(a, f);
        return launch_status();
    }

    uint32_t*       m_rings  = nullptr;
    const uint32_t* m_params = nullptr;
    // rings and offsets of the CPU path (the device layout, in host memory)
    std::vector<uint32_t> m_hrings;
};

} // namespace

rocrand_generator_base_type* make_mtgp32()
{
    return new Mtgp32Generator();
}

} // namespace rb200
