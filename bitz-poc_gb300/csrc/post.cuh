// Field elements posted to mapped host memory.  An element is three words of 44
// bits, each with the low 20 bits of the post's number above them.  A 64-bit
// store is one access, so a word whose tag is right holds this post's bits: the
// host needs no flag that is ordered behind them, and the device no
// system-scope release.
#pragma once
#include <stdint.h>

#include "gf128.cuh"

namespace bz {

__device__ __forceinline__ void post_element(uint64_t *words, uint32_t seq, uint4 v) {
    const uint64_t lo = lo64(v), hi = hi64(v), tag = (uint64_t)seq << 44;
    const uint64_t m = ((uint64_t)1 << 44) - 1;
    volatile uint64_t *o = words;
    o[0] = (lo & m) | tag;
    o[1] = (((lo >> 44) | (hi << 20)) & m) | tag;
    o[2] = (hi >> 24) | tag;
}

}  // namespace bz
