// Kernels around the group passes of ntt_group.cuh and their launchers.
#include <cuda_runtime.h>

#include <algorithm>

#include "bz_internal.h"
#include "chain.cuh"
#include "gf128.cuh"
#include "ntt_group.cuh"

namespace bz {

// Four layers: one CTA of 512 threads per SM (64 registers of data each).
template <int W0, int W1, int W2, int W3>
__global__ void __launch_bounds__(512, 1) ntt_group16(GroupPassArgs a) {
    extern __shared__ uint4 smem[];
    const uint64_t chunks = a.n_tasks / blockDim.x;
    group_pass_body<4, W0, W1, W2, W3, 0, false>(a, chunks * blockIdx.x / gridDim.x,
                                                 chunks * (blockIdx.x + 1) / gridDim.x,
                                                 reinterpret_cast<char *>(smem));
}

// Three layers: two CTAs of 256 threads per SM, so one builds its tables or
// waits for its loads while the other multiplies (2^23 elements of 32 lanes,
// depths 3-5: 170 us against 186 us with one CTA of 512).  Without block
// offsets (EW = 0) there are registers left to load the next task ahead:
// 2^26 elements of 4096 lanes take 440 us against 496 us, and 508 us for the
// radix-8 pass with a table per twiddle.
template <int W0, int W1, int W2, int EW>
__global__ void __launch_bounds__(256, 2) ntt_group8(GroupPassArgs a) {
    extern __shared__ uint4 smem[];
    const uint64_t chunks = a.n_tasks / blockDim.x;
    group_pass_body<3, W0, W1, W2, 0, EW, EW == 0>(a, chunks * blockIdx.x / gridDim.x,
                                                   chunks * (blockIdx.x + 1) / gridDim.x,
                                                   reinterpret_cast<char *>(smem));
}

constexpr int kGroup16Smem = 2 * kGPairBytes;
constexpr int kGroup8Smem = kGPairBytes + kT8Bytes;

#define BZ_GROUP16_WIDTHS(F) F(2, 2, 1, 1) F(4, 2, 1, 1) F(4, 2, 2, 1) F(4, 4, 2, 1)
#define BZ_GROUP8_WIDTHS(F) F(2, 1, 1) F(2, 2, 1) F(4, 2, 1)

void init_group_kernels() {
    auto big = [](auto *k, int bytes) {
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
#define BZ_G_ATTR(A, B, C, D) big(ntt_group16<A, B, C, D>, kGroup16Smem);
    BZ_GROUP16_WIDTHS(BZ_G_ATTR)
#undef BZ_G_ATTR
#define BZ_G_ATTR(A, B, C)                      \
    big(ntt_group8<A, B, C, 0>, kGroup8Smem);   \
    big(ntt_group8<A, B, C, 2>, kGroup8Smem);
    BZ_GROUP8_WIDTHS(BZ_G_ATTR)
#undef BZ_G_ATTR
    big(ntt_group8<4, 4, 4, 4>, kGroup8Smem);
}

// log2 of the CTA size of a pass over 2^log_tasks tasks: 2^full threads, fewer
// while that leaves SMs without a CTA.
static int group_log_threads(int log_tasks, int num_sms, int full) {
    int t = std::min(full, log_tasks);
    while (t > 6 && ((uint64_t)1 << (log_tasks - t)) < (uint64_t)num_sms) --t;
    return t;
}

bool group16_ok(const Shape &s) {
    return s.k_code() - s.log_inv_rate >= 4 && s.k_code() <= 25 && s.log_lanes >= 9;
}

int launch_group16(const Shape &s, const uint4 *src, int src_bits, uint4 *dst, const uint4 *tw,
                   cudaStream_t st, int num_sms, int waves) {
    const int ell = s.k_code(), L = s.log_lanes;
    const int t = group_log_threads(ell - 4 + L, num_sms, 9);
    GroupPassArgs a{src, dst, tw, ell, 0, L, src_bits, (uint64_t)1 << (ell - 4 + L)};
    const unsigned grid =
        (unsigned)std::min<uint64_t>(a.n_tasks >> t, (uint64_t)num_sms * waves);
    const int w3 = narrow_class(twiddle_bits(ell, ell - 4));
    const int w2 = narrow_class(twiddle_bits(ell, ell - 3));
    const int w1 = narrow_class(twiddle_bits(ell, ell - 2));
#define BZ_G_RUN(A, B, C, D) \
    launch_chained(ntt_group16<A, B, C, D>, grid, 1u << t, kGroup16Smem, st, a)
    if (w3 <= 2) BZ_G_RUN(2, 2, 1, 1);
    else if (w2 <= 2 && w1 == 1) BZ_G_RUN(4, 2, 1, 1);
    else if (w2 <= 2) BZ_G_RUN(4, 2, 2, 1);
    else BZ_G_RUN(4, 4, 2, 1);
#undef BZ_G_RUN
    return 1;
}

// ell <= 25: the deepest layer's twiddles fit a one-word table.
bool group8_ok(const Shape &s) {
    return s.k_code() - s.log_inv_rate >= 3 && s.k_code() <= 25 &&
           s.k_code() + s.log_lanes - 3 >= 5;
}

int launch_group8(const Shape &s, int depth, const uint4 *src, int src_bits, uint4 *dst,
                  const uint4 *tw, cudaStream_t st, int num_sms, int waves) {
    const int ell = s.k_code(), L = s.log_lanes;
    const int t = group_log_threads(ell - 3 + L, num_sms, 8);
    GroupPassArgs a{src, dst, tw, ell, depth, L, src_bits, (uint64_t)1 << (ell - 3 + L)};
    const unsigned grid =
        (unsigned)std::min<uint64_t>(a.n_tasks >> t, (uint64_t)num_sms * 2 * waves);
    if (depth > 0) {
        launch_chained(ntt_group8<4, 4, 4, 4>, grid, 1u << t, kGroup8Smem, st, a);
        return 1;
    }
    const int w2 = narrow_class(twiddle_bits(ell, ell - 3));
    const int w1 = narrow_class(twiddle_bits(ell, ell - 2));
    // the offsets of a block in a chunk of 2^t tasks have t - L bits and their
    // twiddles a degree of up to 4 (t - L) <= 32 at depth 2: 33 bits, two words
#define BZ_G_RUN(A, B, C)                                                                     \
    {                                                                                         \
        if (L >= t) launch_chained(ntt_group8<A, B, C, 0>, grid, 1u << t, kGroup8Smem, st, a);\
        else launch_chained(ntt_group8<A, B, C, 2>, grid, 1u << t, kGroup8Smem, st, a);       \
    }
    if (w2 <= 2 && w1 == 1) BZ_G_RUN(2, 1, 1)
    else if (w2 <= 2) BZ_G_RUN(2, 2, 1)
    else BZ_G_RUN(4, 2, 1)
#undef BZ_G_RUN
    return 1;
}

}  // namespace bz
