// MRG32k3a's step (stateful_engines.cuh, host build) against remainders taken by %, over states
// of edge words -- 0, 1, around each modulus, the largest word (an unskipped engine starts from
// unreduced seed words) -- and random ones.  Prints the number of differences and of steps.
#include "stateful_engines.cuh"

#include <cstdio>
#include <random>
#include <vector>

using rb200::Mrg32k3aEngine;

int main()
{
    const uint64_t m1 = 4294967087ull, m2 = 4294944443ull;
    std::mt19937   rng(5);
    std::vector<uint32_t> edge = {0u, 1u, 2u, 208u, 209u, 210u, 22852u, 22853u, 22854u, 0x80000000u, 0xffffffffu};
    for(uint64_t m : {m1, m2})
        for(int d = -2; d <= 2; d++)
            edge.push_back(static_cast<uint32_t>(m + d));
    for(int k = 0; k < 12; k++)
        edge.push_back(rng());
    long bad = 0, count = 0;
    auto check = [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
        Mrg32k3aEngine e;
        const uint32_t w[6] = {a, b, 7u, c, 9u, d};
        for(int k = 0; k < 6; k++)
            e.w[k] = w[k];
        const uint32_t got = e.next();
        const uint64_t n1  = static_cast<uint32_t>(static_cast<uint32_t>(m1) - a);
        const uint64_t n2  = static_cast<uint32_t>(static_cast<uint32_t>(m2) - c);
        const uint32_t p1  = static_cast<uint32_t>((1403580ull * b + 810728ull * n1) % m1);
        const uint32_t p2  = static_cast<uint32_t>((527612ull * d + 1370589ull * n2) % m2);
        const uint32_t want = (p1 - p2) + (p1 <= p2 ? static_cast<uint32_t>(m1) : 0u);
        bad += got != want || e.w[2] != p1 || e.w[5] != p2;
        count++;
    };
    for(uint32_t a : edge)
        for(uint32_t b : edge)
            for(uint32_t c : edge)
                for(uint32_t d : edge)
                    check(a, b, c, d);
    // sums next to a multiple of a modulus: b (or d) solved for with a = m (so n = 0)
    for(long k = 0; k < 3000000; k++)
    {
        const uint64_t t1 = (static_cast<uint64_t>(rng()) % 1403580ull) * m1, t2 = (static_cast<uint64_t>(rng()) % 527612ull) * m2;
        const int      s  = static_cast<int>(rng() % 3);
        check(static_cast<uint32_t>(m1), static_cast<uint32_t>(t1 / 1403580ull + s), static_cast<uint32_t>(m2),
              static_cast<uint32_t>(t2 / 527612ull + s));
    }
    std::printf("%ld %ld\n", bad, count);
    return 0;
}
