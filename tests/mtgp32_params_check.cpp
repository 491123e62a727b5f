// mtgp_parameter_sets (mtgp32_params.hpp) on the embedded blob and on spoiled copies of it.  Prints
// the smallest and largest pos, then 1 for each spoiled copy that is refused.
#include "mtgp32_params.hpp"

#include <algorithm>
#include <cstdio>
#include <fstream>
#include <iterator>
#include <vector>

using namespace rb200;

int main(int, char** argv)
{
    std::ifstream                    f(argv[1], std::ios::binary);
    const std::vector<unsigned char> blob((std::istreambuf_iterator<char>(f)), std::istreambuf_iterator<char>());
    const uint32_t* const            words = mtgp_parameter_sets(blob.data(), blob.size());
    if(words == nullptr)
        return 1;
    uint32_t low = ~0u, high = 0;
    for(uint32_t i = 0; i < kMtgpGens; i++)
    {
        low  = std::min(low, words[i * kMtgpWords]);
        high = std::max(high, words[i * kMtgpWords]);
    }
    std::printf("%u %u", low, high);
    for(uint32_t set : {0u, kMtgpGens - 1})
        for(uint32_t pos : {0u, static_cast<uint32_t>(kMtgpReach) + 1, ~0u})
        {
            std::vector<unsigned char> bad(blob);
            std::memcpy(bad.data() + 12 + sizeof(uint32_t) * kMtgpWords * set, &pos, sizeof(pos));
            std::printf(" %d", mtgp_parameter_sets(bad.data(), bad.size()) == nullptr);
        }
    std::printf(" %d\n", mtgp_parameter_sets(blob.data(), blob.size() - 1) == nullptr);
    return 0;
}
