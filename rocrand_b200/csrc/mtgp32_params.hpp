// mtgp32_params.hpp -- layout of the embedded MTGP32 parameter sets and what the fill kernel takes
// for granted about them.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>

namespace rb200
{

constexpr int      kMtgpN     = 351;
constexpr uint32_t kMtgpGens  = 512;
constexpr uint32_t kMtgpBlock = 256;
constexpr int      kMtgpWords = 36; // pos, sh1, sh2, tbl[16], tmp_tbl[16], mask

// The largest pos: a block step reads up to pos + 255 words ahead of its offset, and the words that
// the kernel repeats behind its ring are one more than that reaches.
constexpr int kMtgpReach = 95;
static_assert(kMtgpBlock + kMtgpReach <= kMtgpN, "a step reads no word that it writes");

// The sets' words in a blob ("RBMTGP01", the count, then 36 words a set), or nullptr where it is not
// such a blob or a pos is outside 1 .. kMtgpReach (the kernel would read outside its ring).
inline const uint32_t* mtgp_parameter_sets(const unsigned char* blob, size_t bytes)
{
    if(bytes != 12 + sizeof(uint32_t) * kMtgpWords * kMtgpGens || std::memcmp(blob, "RBMTGP01", 8) != 0)
        return nullptr;
    const uint32_t* words = reinterpret_cast<const uint32_t*>(blob + 12);
    for(uint32_t i = 0; i < kMtgpGens; i++)
        if(words[i * kMtgpWords] - 1u >= static_cast<uint32_t>(kMtgpReach))
            return nullptr;
    return words;
}

} // namespace rb200
