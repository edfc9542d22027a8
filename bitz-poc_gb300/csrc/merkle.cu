// Merkle tree over codeword rows (flock-core/src/merkle.rs:558-596,
// commit.rs:283-297): leaf i = the 16 * 2^log_lanes bytes of position i,
// flat layout [leaves .., level k-1 .., root].
//
// BLAKE3 leaves are non-root chaining values with BLAKE3's own chunk tree
// (merkle.rs:160-201).  For a leaf of C = L/64 >= 1 full 1 KiB chunks (C a
// power of two), the leaf CV is a perfect binary tree of PARENT merges over
// the C chunk CVs (chunk counter = chunk index inside the leaf), and the
// Merkle tree above the leaves is the same PARENT merge, so one CTA hashes
// 256 chunks (one per thread) and folds them in shared memory straight into
// leaf CVs.  Leaves shorter than 1 KiB are one partial chunk (counter 0).
// SHA-256 leaves are sha256(row) (merkle.rs:213) and parents sha256(l || r).
#include <cuda_runtime.h>

#include <algorithm>

#include "bz_internal.h"
#include "chain.cuh"
#include "hash.cuh"
#include "merkle_kernels.cuh"

namespace bz {

// ---- kernels around the bodies of merkle_kernels.cuh -----------------------
template <bool LEVELS>
__global__ void __launch_bounds__(256) b3_leaves_chunked(const uint4 *cw, uint64_t n_chunks,
                                                         uint32_t *tree_leaves, int log_c,
                                                         uint64_t chunk0, int levels,
                                                         uint64_t n_leaves) {
    __shared__ uint32_t cvs[256][9];  // padded rows
    chain_wait();
    b3_leaves_chunked_body<LEVELS>(cw, n_chunks, tree_leaves, log_c, chunk0,
                                   (uint64_t)blockIdx.x * blockDim.x, cvs, levels, n_leaves);
}

__global__ void b3_leaves_small(const uint4 *cw, int log_lanes, uint64_t n_leaves,
                                uint32_t *tree_leaves) {
    chain_wait();
    b3_leaves_small_body(cw, log_lanes, n_leaves, tree_leaves,
                         (uint64_t)blockIdx.x * blockDim.x + threadIdx.x,
                         (uint64_t)gridDim.x * blockDim.x);
}

// Short leaves (one per thread, a power of two of them) and the `levels` tree
// levels above the CTA's blockDim.x leaves, level l stored at tree + the sizes
// of the levels below it.
__global__ void __launch_bounds__(256) b3_leaves_small_levels(const uint4 *cw, int log_lanes,
                                                              uint64_t n_leaves, uint32_t *tree,
                                                              int levels) {
    __shared__ uint32_t nodes[256][9];  // padded rows
    chain_wait();
    const uint32_t t = threadIdx.x;
    const uint64_t leaf = (uint64_t)blockIdx.x * blockDim.x + t;
    uint32_t o[8];
    b3_leaf_small(cw + (leaf << log_lanes), log_lanes, o);
    uint64_t off = 0;
    for (int lv = 0;; ++lv) {
        const uint32_t n = blockDim.x >> lv;  // the CTA's nodes of this level
        if (t < n) {
            uint4 *po = reinterpret_cast<uint4 *>(tree + (off + (uint64_t)blockIdx.x * n + t) * 8);
            po[0] = make_uint4(o[0], o[1], o[2], o[3]);
            po[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
        if (lv == levels) break;
        if (t < n) {
#pragma unroll
            for (int i = 0; i < 8; ++i) nodes[t][i] = o[i];
        }
        __syncthreads();
        if (t < n / 2) b3_parent(nodes[2 * t], nodes[2 * t + 1], o);
        __syncthreads();  // every read of this level precedes the overwrite
        off += n_leaves >> lv;
    }
}

__global__ void __launch_bounds__(256) merkle_levels(const __grid_constant__ LevelsArgs a) {
    __shared__ uint32_t nodes[256][9];
    chain_wait();
    merkle_levels_body(a, blockIdx.x, nodes);
}

__global__ void __launch_bounds__(128) sha_leaves(const uint4 *cw, int log_lanes,
                                                  uint64_t n_leaves, uint32_t *tree_leaves,
                                                  const __grid_constant__ ShaWords pad) {
    chain_wait();
    sha_leaves_body(cw, log_lanes, n_leaves, tree_leaves, pad,
                    (uint64_t)blockIdx.x * blockDim.x + threadIdx.x,
                    (uint64_t)gridDim.x * blockDim.x);
}

// A small BLAKE3 tree of short leaves (at most one chunk, log_lanes < 6) in
// one CTA: thread i hashes leaf i, then the CTA builds every level up to the
// root in shared memory, writing leaves and levels to the flat tree as
// merkle_levels does.  256 leaves of 512 B take 18.9 us against 28.7 us for
// b3_leaves_small + merkle_levels.  Full 1 KiB chunks are left to the
// multi-CTA kernels: there one SM's issue rate bounds a single CTA (256
// leaves of 1 KiB: 32.4 against 30.7 us).
constexpr int kTreeSmallMax = 1024;  // leaves (threads)
__global__ void __launch_bounds__(kTreeSmallMax) b3_tree_small(const uint4 *cw, int log_lanes,
                                                               uint32_t n_leaves,
                                                               uint32_t *tree, RootPost post) {
    __shared__ uint32_t nodes[kTreeSmallMax][9];  // padded rows
    chain_wait();
    const uint32_t t = threadIdx.x;
    uint32_t o[8];
    b3_leaf_small(cw + ((uint64_t)t << log_lanes), log_lanes, o);
    uint64_t off = 0;
    for (uint32_t n = n_leaves;; n >>= 1) {
        if (t < n) {
            uint4 *po = reinterpret_cast<uint4 *>(tree + (off + t) * 8);
            po[0] = make_uint4(o[0], o[1], o[2], o[3]);
            po[1] = make_uint4(o[4], o[5], o[6], o[7]);
#pragma unroll
            for (int i = 0; i < 8; ++i) nodes[t][i] = o[i];
        }
        __syncthreads();
        if (n == 1) break;
        if (t < n / 2) b3_parent(nodes[2 * t], nodes[2 * t + 1], o);
        __syncthreads();  // every read of this level precedes the overwrite
        off += n;
    }
    if (t == 0) post_root(post, o);
}

// A small SHA-256 tree in one CTA: thread i of the first half hashes leaf i,
// then the CTA builds every level.  Up to one warp per scheduler hashes, so no
// leaf's chain waits for another's; as many warps again compute message
// schedules: of a row's next block while this one is hashed (rows of 8 blocks
// or more: 64 leaves of 512 bytes 30.4 us against 37; of 4 blocks or fewer the
// hashing warps do it all, as the first block's schedule lies on the chain),
// and of a level's pairs, whose first sixteen rounds need none (64 leaves of
// 256 bytes 27.3 us against 29.3).
constexpr int kShaTreeSmallMax = 128;    // leaves
constexpr int kShaAheadLanes = 5;        // log2
constexpr size_t kShaKwWords = 64 * 32;  // a warp's schedule of one block
constexpr size_t sha_ahead_smem(unsigned warps) { return 2 * warps * kShaKwWords * 4; }
__global__ void __launch_bounds__(2 * kShaTreeSmallMax) sha_tree_small(
    const uint4 *cw, int log_lanes, uint32_t n_leaves, uint32_t *tree,
    const __grid_constant__ ShaWords pad, RootPost post) {
    extern __shared__ uint32_t kws[];  // two blocks' schedules for each hashing warp
    __shared__ uint32_t nodes[kShaTreeSmallMax][9];  // padded rows
    chain_wait();
    const uint32_t half = blockDim.x / 2;
    const bool hasher = threadIdx.x < half;
    // leaf or pair; with four warps a half, those that schedule a level of at
    // most 64 pairs sit on the schedulers that the level's hashes leave idle
    const uint32_t t = hasher ? threadIdx.x : (threadIdx.x - half) ^ (half == 128 ? 64 : 0);
    uint32_t *kw = kws + (t >> 5) * 2 * kShaKwWords + (t & 31);
    uint32_t o[8], w[16];
    if (log_lanes >= kShaAheadLanes) {
        const uint4 *p = cw + ((uint64_t)t << log_lanes);
        const uint32_t blocks = 1u << (log_lanes - 2);
        uint32_t st[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                          0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
#pragma unroll 1
        for (uint32_t blk = 0; blk <= blocks; ++blk) {
            if (hasher) {
                if (blk) {
                    uint32_t v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = st[i];
                    sha_rounds<0, 64>(v, kw + ((blk - 1) & 1) * kShaKwWords);
#pragma unroll
                    for (int i = 0; i < 8; ++i) st[i] += v[i];
                }
            } else if (blk < blocks && t < n_leaves) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint4 x = p[4 * blk + q];
                    w[4 * q] = bswap32(x.x);
                    w[4 * q + 1] = bswap32(x.y);
                    w[4 * q + 2] = bswap32(x.z);
                    w[4 * q + 3] = bswap32(x.w);
                }
                sha_schedule<0, 64>(w, kw + (blk & 1) * kShaKwWords);
            }
            __syncthreads();
        }
        if (hasher) sha256_compress_kw<true>(st, pad);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = bswap32(st[i]);
    } else if (hasher && t < n_leaves) {
        sha_leaf<true>(cw + ((uint64_t)t << log_lanes), log_lanes, pad, o);
    }
    uint64_t off = 0;
    for (uint32_t n = n_leaves;; n >>= 1) {
        if (hasher && t < n) {
            uint4 *po = reinterpret_cast<uint4 *>(tree + (off + t) * 8);
            po[0] = make_uint4(o[0], o[1], o[2], o[3]);
            po[1] = make_uint4(o[4], o[5], o[6], o[7]);
#pragma unroll
            for (int i = 0; i < 8; ++i) nodes[t][i] = bswap32(o[i]);
        }
        __syncthreads();
        if (n == 1) break;
        const bool work = t < n / 2;
        uint32_t v[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                         0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
        if (work) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                w[i] = nodes[2 * t][i];
                w[8 + i] = nodes[2 * t + 1][i];
            }
            if (hasher) {
                const uint32_t one = kOne;
#pragma unroll
                for (int i = 0; i < 16; ++i) BZ_SHA_ROUND_AT(v, i, w[i] * one + kSHA.w[i]);
            } else {
                sha_schedule<16, 32>(w, kw);
            }
        }
        __syncthreads();  // words 16 to 31; every read of this level's nodes
        if (work) {
            if (hasher) sha_rounds<16, 32>(v, kw);
            else sha_schedule<32, 64>(w, kw);
        }
        __syncthreads();
        if (work && hasher) {
            sha_rounds<32, 64>(v, kw);
            uint32_t st[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                              0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
#pragma unroll
            for (int i = 0; i < 8; ++i) st[i] += v[i];
            sha256_compress_kw<true>(st, kShaPairPad);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = bswap32(st[i]);
        }
        off += n;
    }
    if (threadIdx.x == 0 && n_leaves > 1) post_root(post, o);
}

void init_merkle_kernels() {
    cudaFuncSetAttribute(sha_tree_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sha_ahead_smem(kShaTreeSmallMax / 32));
}

// Generic BLAKE3 chunk CVs into scratch (leaves longer than 256 chunks).
__global__ void b3_chunk_cvs(const uint4 *cw, uint64_t n_chunks, int log_c, uint32_t *out,
                             uint64_t chunk0) {
    chain_wait();
    const uint64_t chunk = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (chunk >= n_chunks) return;
    const uint64_t c_in_leaf = chunk0 + (chunk & ((1ull << log_c) - 1));
    uint32_t cv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) cv[i] = kIV[i];
    const uint4 *p = cw + chunk * 64;
#pragma unroll 1
    for (int blk = 0; blk < 16; ++blk) {
        uint32_t m[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint4 v = __ldcs(p + blk * 4 + q);
            m[4 * q] = v.x;
            m[4 * q + 1] = v.y;
            m[4 * q + 2] = v.z;
            m[4 * q + 3] = v.w;
        }
        const uint32_t flags = (blk == 0 ? B3_CHUNK_START : 0) | (blk == 15 ? B3_CHUNK_END : 0);
        b3_compress_cv(cv, m, c_in_leaf, 64, flags);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) out[chunk * 8 + i] = cv[i];
}

size_t merkle_scratch_bytes(const Shape &s) {
    if (s.hash_kind == 1 && s.log_lanes > 14) {
        const size_t chunks = s.cw_words() / 64;
        return chunks * 32 * 2;
    }
    return 0;
}

// Build all parent levels above `n_leaves` leaves stored at tree[0..).
// (or above level `from`, whose nodes are stored).
static int launch_levels(uint32_t *tree, uint64_t n_leaves, int kind, cudaStream_t st,
                         LaunchLog *log, int from = 0, const RootPost *post = nullptr);

// Tree levels that the leaf kernel builds, of at most `most` that its CTAs can:
// the fewest that save a launch of nine levels, below the root, else none.  A
// level costs a CTA more than 1 us behind its leaves, and a launch 4 us or more
// (2^17 leaves of 256 bytes, 17 levels: 49 us with 8 levels and one launch, 51
// with two launches; 2^14 leaves of 64 KiB with the 2 levels that its CTAs
// reach and still two launches: 569 + 20 us against 551 + 20).  For commits that
// a caller waits for (those that post their root): many at once are bound by
// issue slots, of which half-empty levels waste some (16 commits in one plan:
// 1431 us against 1411).
static int leaf_levels(uint64_t n_leaves, int most) {
    int lg = 0;
    while (n_leaves >> (lg + 1)) ++lg;
    const int need = lg % 9 == 0 ? 9 : lg % 9;
    return lg > 9 && need <= most ? need : 0;
}

// CTA size of b3_leaves_chunked: 256 threads, halved (down to 32 and to the
// chunks per leaf) while that leaves fewer than two CTAs per SM.
static unsigned leaf_threads(uint64_t n_chunks, int log_c, int num_sms) {
    unsigned t = 256;
    const unsigned floor = std::max(32u, 1u << log_c);
    while (t > floor && n_chunks / t < 2 * (uint64_t)num_sms) t >>= 1;
    return t;
}

bool leaves_range_supported(const Shape &s) { return !(s.hash_kind == 1 && s.log_lanes > 14); }

int launch_leaves_range(const Shape &s, const uint4 *d_cw, uint8_t *d_tree, uint64_t p0,
                        uint64_t p1, cudaStream_t st, int num_sms) {
    uint32_t *tree = reinterpret_cast<uint32_t *>(d_tree);
    const uint64_t n = p1 - p0;
    const uint4 *cw = d_cw + (p0 << s.log_lanes);
    uint32_t *leaves = tree + p0 * 8;
    if (s.hash_kind == 1) {
        if (s.log_lanes < 6) {
            launch_chained(b3_leaves_small, (unsigned)((n + 255) / 256), 256, 0, st, cw,
                           s.log_lanes, n, leaves);
        } else {
            const int log_c = s.log_lanes - 6;
            const uint64_t n_chunks = n << log_c;
            const unsigned t = leaf_threads(n_chunks, log_c, num_sms);
            launch_chained(b3_leaves_chunked<false>, (unsigned)((n_chunks + t - 1) / t), t, 0, st,
                           cw, n_chunks, leaves, log_c, s.chunk0, 0, n);
        }
    } else {
        launch_chained(sha_leaves, (unsigned)((n + 127) / 128), 128, 0, st, cw, s.log_lanes, n,
                       leaves, sha_pad_kw(s.leaf_bytes() * 8));
    }
    return 1;
}

int launch_merkle_levels(const Shape &s, uint8_t *d_tree, cudaStream_t st, LaunchLog *log) {
    return launch_levels(reinterpret_cast<uint32_t *>(d_tree), s.n_leaves(), s.hash_kind, st,
                         log);
}

static int launch_levels(uint32_t *tree, uint64_t n_leaves, int kind, cudaStream_t st,
                         LaunchLog *log, int from, const RootPost *post) {
    int launches = 0;
    uint64_t in_off = 2 * n_leaves - (2 * n_leaves >> from), n_in = n_leaves >> from;
    while (n_in > 1) {
        int k = 0;
        uint64_t n = n_in;
        while (n > 1 && k < 9) {
            n >>= 1;
            ++k;
        }
        LevelsArgs a;
        a.in = tree + in_off * 8;
        a.n_in = n_in;
        a.k = k;
        a.kind = kind;
        if (post && n_in >> k == 1) a.post = *post;
        uint64_t off = in_off + n_in, cnt = n_in >> 1;
        for (int j = 0; j < k; ++j) {
            a.out[j] = tree + off * 8;
            off += cnt;
            cnt >>= 1;
        }
        const uint64_t ctas = (n_in + 511) / 512;
        launch_chained(merkle_levels, (unsigned)ctas, 256, 0, st, a);
        if (log) log->mark("merkle_levels");
        ++launches;
        // advance: the last produced level becomes the next input
        uint64_t o = in_off + n_in, c = n_in >> 1;
        for (int j = 0; j < k - 1; ++j) {
            o += c;
            c >>= 1;
        }
        in_off = o;
        n_in = c;
    }
    return launches;
}

int launch_merkle(const Shape &s, const uint4 *d_cw, uint8_t *d_tree, uint8_t *d_scratch,
                  cudaStream_t st, int num_sms, LaunchLog *log, const RootPost *post) {
    int from = 0;  // tree levels the leaf kernel has built
    auto mark = [&](const char *n) {
        if (log) log->mark(n);
    };
    const uint64_t n_leaves = s.n_leaves();
    uint32_t *tree = reinterpret_cast<uint32_t *>(d_tree);
    int launches = 0;
    if (s.hash_kind == 1) {
        if (s.log_lanes < 6 && n_leaves <= (uint64_t)kTreeSmallMax && n_leaves >= 2) {
            launch_chained(b3_tree_small, 1, (unsigned)n_leaves, 0, st, d_cw, s.log_lanes,
                           (uint32_t)n_leaves, tree, post ? *post : RootPost{});
            mark("b3_tree_small");
            return 1;
        }
        if (s.log_lanes < 6) {
            // more than kTreeSmallMax leaves: a multiple of the CTA's 256
            from = post ? leaf_levels(n_leaves, 8) : 0;
            if (from)
                launch_chained(b3_leaves_small_levels, (unsigned)(n_leaves / 256), 256, 0, st,
                               d_cw, s.log_lanes, n_leaves, tree, from);
            else
                launch_chained(b3_leaves_small, (unsigned)((n_leaves + 255) / 256), 256, 0, st,
                               d_cw, s.log_lanes, n_leaves, tree);
            mark("b3_leaves_small");
            ++launches;
        } else if (s.log_lanes <= 14) {
            const int log_c = s.log_lanes - 6;
            const uint64_t n_chunks = n_leaves << log_c;
            const unsigned t = leaf_threads(n_chunks, log_c, num_sms);
            // a CTA that is full of chunks has t >> log_c whole leaves
            int most = 0;
            while (n_chunks >= t && (t >> log_c) >> (most + 1)) ++most;
            from = post ? leaf_levels(n_leaves, most) : 0;
            launch_chained(from ? b3_leaves_chunked<true> : b3_leaves_chunked<false>,
                           (unsigned)((n_chunks + t - 1) / t), t, 0, st, d_cw, n_chunks, tree, log_c, s.chunk0, from, n_leaves);
            mark("b3_leaves_chunked");
            ++launches;
        } else {
            const int log_c = s.log_lanes - 6;
            const uint64_t n_chunks = n_leaves << log_c;
            uint32_t *cvs = reinterpret_cast<uint32_t *>(d_scratch);
            launch_chained(b3_chunk_cvs, (unsigned)((n_chunks + 255) / 256), 256, 0, st, d_cw,
                           n_chunks, log_c, cvs, s.chunk0);
            mark("b3_chunk_cvs");
            ++launches;
            // reduce chunk CVs to leaf CVs: levels inside the scratch area,
            // the last one written straight into the tree leaves.
            uint32_t *bufs[2] = {cvs, cvs + n_chunks * 8};
            uint64_t n = n_chunks;
            int cur = 0;
            for (int lv = 0; lv < log_c; ++lv) {
                LevelsArgs a;
                a.in = bufs[cur];
                a.n_in = n;
                a.k = 1;
                a.kind = 1;
                a.out[0] = (lv == log_c - 1) ? tree : bufs[cur ^ 1];
                launch_chained(merkle_levels, (unsigned)((n + 511) / 512), 256, 0, st, a);
                mark("merkle_levels");
                ++launches;
                n >>= 1;
                cur ^= 1;
            }
        }
    } else {
        const ShaWords pad = sha_pad_kw(s.leaf_bytes() * 8);
        if (n_leaves <= (uint64_t)kShaTreeSmallMax) {
            const RootPost rp = post ? *post : RootPost{};
            const unsigned warps = (unsigned)(n_leaves + 31) / 32;  // that hash
            launch_chained(sha_tree_small, 1, 64 * warps, sha_ahead_smem(warps), st, d_cw,
                           s.log_lanes, (uint32_t)n_leaves, tree, pad, rp);
            mark("sha_tree_small");
            return 1;
        }
        launch_chained(sha_leaves, (unsigned)((n_leaves + 127) / 128), 128, 0, st, d_cw,
                       s.log_lanes, n_leaves, tree, pad);
        mark("sha_leaves");
        ++launches;
    }
    launches += launch_levels(tree, n_leaves, s.hash_kind, st, log, from, post);
    return launches;
}

// ---------------------------------------------------------------------------
// Leaves of a lane-sharded BLAKE3 commit: one thread per position merges the
// world ranks' subtree CVs left to right with BLAKE3's CV stack (a subtree of
// 2^j ranks is merged with its left neighbour of the same size), which for a
// power-of-two world is the perfect binary tree of PARENT merges the leaf's
// own chunk tree has above those subtrees (merkle.rs:160-201).
// ---------------------------------------------------------------------------
constexpr int kMaxShardLevels = 11;  // world <= 1024
__global__ void b3_combine_shard_cvs(const uint32_t *cvs, uint32_t world, uint64_t n_leaves,
                                     uint32_t *leaves) {
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_leaves) return;
    uint32_t stack[kMaxShardLevels][8];
    int depth = 0;
    for (uint32_t r = 0; r < world; ++r) {
        uint32_t cv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) cv[i] = cvs[((uint64_t)r * n_leaves + p) * 8 + i];
        // merge while the subtree just completed has a left sibling of equal
        // size: the number of trailing one bits of r
        for (uint32_t m = r; m & 1; m >>= 1) {
            uint32_t o[8];
            b3_parent(stack[--depth], cv, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) cv[i] = o[i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) stack[depth][i] = cv[i];
        ++depth;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) leaves[p * 8 + i] = stack[0][i];
}

int launch_combine_shard_cvs(const uint8_t *d_cvs, uint32_t world, uint64_t n_leaves,
                             uint8_t *d_tree, cudaStream_t st) {
    if (world == 0 || (world & (world - 1)) || world > (1u << (kMaxShardLevels - 1))) return 0;
    b3_combine_shard_cvs<<<(unsigned)((n_leaves + 127) / 128), 128, 0, st>>>(
        reinterpret_cast<const uint32_t *>(d_cvs), world, n_leaves,
        reinterpret_cast<uint32_t *>(d_tree));
    return 1;
}

// ---------------------------------------------------------------------------
// Gathers for openings.
// ---------------------------------------------------------------------------
// Rows `pos` of the codeword to `rows`, nodes `idx` of the tree to `nodes`.  The
// positions and the outputs may lie in mapped host memory.
__global__ void gather_open(const uint4 *cw, int log_lanes, const uint64_t *pos, uint64_t q,
                            uint4 *rows, const uint4 *tree, const uint64_t *idx, uint64_t n,
                            uint4 *nodes) {
    chain_wait();
    const uint64_t L = (uint64_t)1 << log_lanes;
    const uint64_t in_rows = q * L, total = in_rows + 2 * n;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (i < in_rows) {
            rows[i] = cw[(pos[i >> log_lanes] << log_lanes) | (i & (L - 1))];
        } else {
            const uint64_t k = i - in_rows;
            nodes[k] = tree[idx[k >> 1] * 2 + (k & 1)];
        }
    }
}

int launch_gather_open(const uint4 *d_cw, int log_lanes, const uint64_t *d_pos, size_t q,
                       uint4 *d_rows, const uint8_t *d_tree, const uint64_t *d_idx, size_t n,
                       uint8_t *d_nodes, cudaStream_t st) {
    const uint64_t total = ((uint64_t)q << log_lanes) + 2 * (uint64_t)n;
    if (total == 0) return 0;
    const unsigned grid = (unsigned)std::min<uint64_t>((total + 255) / 256, 4096);
    launch_chained(gather_open, grid, 256, 0, st, d_cw, log_lanes, d_pos, (uint64_t)q, d_rows,
                   reinterpret_cast<const uint4 *>(d_tree), d_idx, (uint64_t)n,
                   reinterpret_cast<uint4 *>(d_nodes));
    return 1;
}

}  // namespace bz
