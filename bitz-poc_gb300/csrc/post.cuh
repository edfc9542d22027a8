// Field elements posted to mapped host memory.  An element is four 64-bit words,
// each with 32 bits of it below the post's number.  A 64-bit store is one access,
// so a word whose number is right holds this post's bits: the host needs no flag
// that is ordered behind them, and the device no system-scope release.  That
// orders the posted bits alone: where the host may let another stream read
// arrays written beside them, the posting thread calls post_release first.
#pragma once
#include <stdint.h>

#include "gf128.cuh"

namespace bz {

__device__ __forceinline__ void post_element(uint64_t *words, uint32_t seq, uint4 v) {
    const uint64_t tag = (uint64_t)seq << 32;
    volatile uint64_t *o = words;
    o[0] = tag | v.x;
    o[1] = tag | v.y;
    o[2] = tag | v.z;
    o[3] = tag | v.w;
}

// Before a post that ends a synchronous call: what this thread has seen written
// (its CTA's arrays behind a barrier, earlier kernels' behind chain_wait, other
// CTAs' behind their ticket) precedes the post at system scope, so whatever the
// host starts after it, on any stream, reads the arrays.  (2^10-element commit
// 64.3 us, 64.8 without it.)
__device__ __forceinline__ void post_release() { __threadfence_system(); }

}  // namespace bz
