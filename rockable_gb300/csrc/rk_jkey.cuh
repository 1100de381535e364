// rk_jkey.cuh -- keys that order the neighbour list's entries by their second
// body (the j-side list): the body above, the entry's index below, so that a
// stable sort on the body's bits keeps the entries of a body in list order.
// The functions also compile for the host (tests check them there).
#pragma once
#include "rk_bits.cuh"

namespace rk {

constexpr int kJkeyBody = 32;                          // first bit of the body (21 bits)
constexpr int64_t kMaxEntries = ((int64_t)1 << 31) - 1;  // the lists hold entries as int

RK_BITS_FN uint64_t jkey(int j, int64_t e) { return ((uint64_t)(uint32_t)j << kJkeyBody) | (uint64_t)e; }
RK_BITS_FN int jkey_entry(uint64_t k) { return (int)(k & (((uint64_t)1 << kJkeyBody) - 1)); }

}  // namespace rk
