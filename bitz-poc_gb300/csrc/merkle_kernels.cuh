// Device bodies of the Merkle leaf and level kernels (the tree layout and
// hashing rules are described at the top of merkle.cu).  merkle.cu wraps each
// body in a kernel of its own; the persistent batch kernel (persist.cu) calls
// the same bodies for its work items, with its own shared-memory layout.
#pragma once
#include <stdint.h>

#include "bz_internal.h"
#include "hash.cuh"
#include "post.cuh"

namespace bz {

// The root o to mapped host memory: the host reads it there instead of copying
// it and waiting for the stream.  Called behind a barrier that follows the CTA's
// tree stores, so the tree and the codeword are released before the root.
__device__ __forceinline__ void post_root(const RootPost &p, const uint32_t o[8]) {
    if (!p.words) return;
    post_release();
    post_element(p.words, p.seq, make_uint4(o[0], o[1], o[2], o[3]));
    post_element(p.words + 4, p.seq, make_uint4(o[4], o[5], o[6], o[7]));
}

// ---------------------------------------------------------------------------
// BLAKE3 leaves, C >= 1 chunks per leaf, C <= 256.
// Each thread computes one chunk CV; the CTA (T <= 256 threads = T chunks =
// T / C leaves, T a power of two >= C) reduces groups of C CVs to leaf CVs in
// shared memory.  Small trees launch smaller CTAs so the chunks spread over
// the SMs (a chunk's 16 compressions are sequential).
// ---------------------------------------------------------------------------
//
// Body: the CTA's blockDim.x chunks from chunk_base (a multiple of blockDim.x,
// blockDim.x a multiple of C); cvs holds blockDim.x padded rows of 9 words.
//
// LEVELS: the CTA goes on merging its leaves into `levels` levels of the tree
// above them (n_leaves leaves; at most log2 of the CTA's), whose parents are the
// same PARENT merge as those inside a leaf.  A kernel of its own: one loop for
// both cost the leaves alone 1 to 1.5 us.
template <bool LEVELS = false>
__device__ __forceinline__ void b3_leaves_chunked_body(const uint4 *cw, uint64_t n_chunks,
                                                       uint32_t *tree_leaves, int log_c,
                                                       uint64_t chunk0, uint64_t chunk_base,
                                                       uint32_t (*cvs)[9], int levels = 0,
                                                       uint64_t n_leaves = 0) {
    const uint64_t chunk = chunk_base + threadIdx.x;
    const uint64_t c_in_leaf = chunk0 + (chunk & ((1u << log_c) - 1));
    uint32_t cv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) cv[i] = kIV[i];
    if (chunk < n_chunks) {
        const uint4 *p = cw + chunk * 64;  // 64 elements = 1024 bytes
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
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) cvs[threadIdx.x][i] = cv[i];
    __syncthreads();
    // Step s merges nodes (2j, 2j+1) of the CTA.
    const int t = threadIdx.x;
    auto merge = [&](int s) {
        const int stride = 1 << s;
        if ((t & ((stride << 1) - 1)) == 0 && t + stride < (int)blockDim.x) {
            uint32_t out[8];
            b3_parent(cvs[t], cvs[t + stride], out);
#pragma unroll
            for (int i = 0; i < 8; ++i) cvs[t][i] = out[i];
        }
        __syncthreads();
    };
    auto store = [&](int s, uint64_t off) {
        if ((t & ((1 << s) - 1)) == 0 && chunk < n_chunks) {
            const uint64_t node = off + (chunk >> s);
#pragma unroll
            for (int i = 0; i < 8; ++i) tree_leaves[node * 8 + i] = cvs[t][i];
        }
    };
    if constexpr (!LEVELS) {
        for (int s = 0; s < log_c; ++s) merge(s);
        store(log_c, 0);
    } else {
        uint64_t off = 0, cnt = n_leaves;  // the tree level's first node and size
        for (int s = 0;; ++s) {
            if (s >= log_c) {
                store(s, off);
                off += cnt;
                cnt >>= 1;
            }
            if (s == log_c + levels) break;
            merge(s);
        }
    }
}

// One BLAKE3 leaf of at most one chunk (leaf_bytes = 16 * 2^log_lanes <= 1024).
__device__ __forceinline__ void b3_leaf_small(const uint4 *p, int log_lanes, uint32_t cv[8]) {
    const uint32_t elems = 1u << log_lanes;  // 16-byte elements
    const uint32_t bytes = elems * 16;
    const uint32_t nblk = (bytes + 63) / 64;
#pragma unroll
    for (int i = 0; i < 8; ++i) cv[i] = kIV[i];
#pragma unroll 1
    for (uint32_t blk = 0; blk < nblk; ++blk) {
        uint32_t m[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t e = blk * 4 + q;
            const uint4 v = e < elems ? p[e] : make_uint4(0, 0, 0, 0);
            m[4 * q] = v.x;
            m[4 * q + 1] = v.y;
            m[4 * q + 2] = v.z;
            m[4 * q + 3] = v.w;
        }
        const uint32_t len = min(64u, bytes - blk * 64);
        const uint32_t flags =
            (blk == 0 ? B3_CHUNK_START : 0) | (blk == nblk - 1 ? B3_CHUNK_END : 0);
        b3_compress_cv(cv, m, 0, len, flags);
    }
}

// Body: leaves first, first + step, .. below n_leaves.
__device__ __forceinline__ void b3_leaves_small_body(const uint4 *cw, int log_lanes,
                                                     uint64_t n_leaves, uint32_t *tree_leaves,
                                                     uint64_t first, uint64_t step) {
    for (uint64_t leaf = first; leaf < n_leaves; leaf += step) {
        uint32_t cv[8];
        b3_leaf_small(cw + (leaf << log_lanes), log_lanes, cv);
#pragma unroll
        for (int i = 0; i < 8; ++i) tree_leaves[leaf * 8 + i] = cv[i];
    }
}

// ---------------------------------------------------------------------------
// Parent levels.  One CTA takes 2^k consecutive nodes of level `in` and
// writes every node of the k levels above them (each level into its own slot
// of the flat tree), so a 2^20-leaf tree needs 3 launches instead of 20.
// kind: 0 = SHA-256, 1 = BLAKE3.
// ---------------------------------------------------------------------------
// MOVED: by sha256_compress_moved, padding block and all.
template <bool MOVED>
__device__ __forceinline__ void sha256_pair(const uint32_t l[8], const uint32_t r[8],
                                            uint32_t out[8]) {
    uint32_t st[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                      0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        w[i] = bswap32(l[i]);
        w[8 + i] = bswap32(r[i]);
    }
    if constexpr (MOVED) {
        sha256_compress_moved(st, w);
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = 0;
        w[0] = 0x80000000u;
        w[15] = 512;
        sha256_compress_moved(st, w);
    } else {
        sha256_compress<true>(st, w);
        sha256_compress_kw<true>(st, kShaPairPad);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = bswap32(st[i]);
}

template <bool MOVED>
__device__ __forceinline__ void hash_pair(int kind, const uint32_t l[8], const uint32_t r[8],
                                          uint32_t out[8]) {
    if (kind == 1) b3_parent(l, r, out);
    else sha256_pair<MOVED>(l, r, out);
}

// in: n_in nodes (32 B each); outputs levels written at out_levels[0..k-1]
// with level j holding n_in >> (j+1) nodes.  blockDim = 256, each CTA covers
// 512 input nodes (or fewer at the top).
struct LevelsArgs {
    const uint32_t *in;
    uint32_t *out[10];
    uint64_t n_in;
    int k;  // levels to produce (<= 9)
    int kind;
    RootPost post;  // when the last level is the root
};

// Body: unit u (512 input nodes) with threads 0..255; any further threads of
// the CTA only take part in its barriers.  nodes holds 256 padded rows.
template <bool MOVED = false>
__device__ __forceinline__ void merkle_levels_body(const LevelsArgs &a, uint64_t u,
                                                   uint32_t (*nodes)[9]) {
    const int t = threadIdx.x;
    // every level through the same code: the first reads its pairs from
    // global memory, the others from shared memory
    uint64_t cta_nodes = min(a.n_in >> 1, (uint64_t)256);  // nodes of this CTA at the level
    for (int lv = 0; lv < a.k; ++lv) {
        const bool active = (uint64_t)t < cta_nodes &&
                            u * (256 >> lv) + t < (a.n_in >> (lv + 1));
        uint32_t o[8];
        if (active) {
            uint32_t l[8], r[8];
            if (lv == 0) {
                const uint4 *pl = reinterpret_cast<const uint4 *>(a.in + (u * 512 + 2 * t) * 8);
                const uint4 l0 = pl[0], l1 = pl[1], r0 = pl[2], r1 = pl[3];
                l[0] = l0.x; l[1] = l0.y; l[2] = l0.z; l[3] = l0.w;
                l[4] = l1.x; l[5] = l1.y; l[6] = l1.z; l[7] = l1.w;
                r[0] = r0.x; r[1] = r0.y; r[2] = r0.z; r[3] = r0.w;
                r[4] = r1.x; r[5] = r1.y; r[6] = r1.z; r[7] = r1.w;
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    l[i] = nodes[2 * t][i];
                    r[i] = nodes[2 * t + 1][i];
                }
            }
            hash_pair<MOVED>(a.kind, l, r, o);
            uint4 *po = reinterpret_cast<uint4 *>(a.out[lv] + (u * (256 >> lv) + t) * 8);
            po[0] = make_uint4(o[0], o[1], o[2], o[3]);
            po[1] = make_uint4(o[4], o[5], o[6], o[7]);
        }
        __syncthreads();  // every read of this level precedes the overwrite
        if (lv == a.k - 1) {
            if (t == 0) post_root(a.post, o);
            break;
        }
        if (active) {
#pragma unroll
            for (int i = 0; i < 8; ++i) nodes[t][i] = o[i];
        }
        __syncthreads();
        cta_nodes >>= 1;
    }
}

// SHA-256 of one row of 16 * 2^log_lanes bytes; pad: sha_pad_kw of its bit
// length (read from 4 lanes up, where the row ends on a block boundary).
template <bool ROLLED>
__device__ __forceinline__ void sha_leaf(const uint4 *p, int log_lanes, const ShaWords &pad,
                                         uint32_t out[8]) {
    uint32_t st[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                      0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
    if (log_lanes >= 2) {
        const uint64_t blocks = (uint64_t)1 << (log_lanes - 2);
        for (uint64_t blk = 0; blk < blocks; ++blk) {
            uint32_t w[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = p[blk * 4 + q];
                w[4 * q] = bswap32(v.x);
                w[4 * q + 1] = bswap32(v.y);
                w[4 * q + 2] = bswap32(v.z);
                w[4 * q + 3] = bswap32(v.w);
            }
            sha256_compress<ROLLED>(st, w);
        }
        sha256_compress_kw<ROLLED>(st, pad);
    } else {
        // one block: 16 or 32 bytes, 0x80, zeros, the length
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = 0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (e >> log_lanes) break;
            const uint4 v = p[e];
            w[4 * e] = bswap32(v.x);
            w[4 * e + 1] = bswap32(v.y);
            w[4 * e + 2] = bswap32(v.z);
            w[4 * e + 3] = bswap32(v.w);
        }
        if (log_lanes == 0) w[4] = 0x80000000u;
        else w[8] = 0x80000000u;
        w[15] = 128u << log_lanes;
        sha256_compress<ROLLED>(st, w);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = bswap32(st[i]);
}

// SHA-256 leaves: one thread per leaf, sequential over the row.
// Body: leaves first, first + step, .. below n_leaves.
__device__ __forceinline__ void sha_leaves_body(const uint4 *cw, int log_lanes, uint64_t n_leaves,
                                                uint32_t *tree_leaves, const ShaWords &pad,
                                                uint64_t first, uint64_t step) {
    for (uint64_t leaf = first; leaf < n_leaves; leaf += step) {
        uint32_t o[8];
        sha_leaf<false>(cw + (leaf << log_lanes), log_lanes, pad, o);
        uint4 *po = reinterpret_cast<uint4 *>(tree_leaves + leaf * 8);
        po[0] = make_uint4(o[0], o[1], o[2], o[3]);
        po[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

}  // namespace bz
