// NTT passes that keep a group of 2^K positions of one lane in a thread's
// registers and run K layers on it with one table per layer.
//
// twiddle(l, b) is GF(2)-linear in the block index b, so over a chunk of
// tasks whose block indices share their high bits it is s + e: s, the
// twiddle of the chunk's first block, is the same for the whole CTA and
// multiplies through one shared-memory table per layer, whatever the number
// of blocks below; e, the twiddle of the block's offset in the chunk, has
// bits of the offset alone (at depth d an offset bit j contributes a
// polynomial of degree 2^d (j - d)), so it is short and multiplies by
// shifting over its set bits.  A pass that gives every block its own tables
// (seven of 32 KB for three layers) rebuilds them for each block and cannot
// run where a block has fewer tasks than the CTA has threads; these passes
// build K tables per chunk for any block size, so the deepest layers of
// codewords with few lanes run through tables too.
#pragma once
#include "ntt_kernels.cuh"

namespace bz {

struct GroupPassArgs {
    const uint4 *src;  // message (first pass) or codeword
    uint4 *dst;        // codeword
    const uint4 *tw;   // twiddle heap
    int ell;
    int depth;         // of the last layer; groups are positions i << depth, i < 2^K
    int log_lanes;
    int src_pos_bits;
    uint64_t n_tasks;  // 2^(ell - K) * lanes, a multiple of blockDim.x
};

// ---- tables ------------------------------------------------------------------
// The byte tables of t8.cuh and the compact tables of ntt_kernels.cuh with
// rows of 128 bytes at a pitch of 256: two tables share 64 KB.  A byte of the
// operand that stands at bits 8-15 of a word is then a row offset as it is,
// and the other three are brought there by one shift, so a lookup costs one or
// two ALU operations (mask and lane offset in one LOP3) beside its shared-memory
// wavefronts.  Multiplies by powers of two in place of the shifts leave the ALU
// pipe 59 % busy instead of 75, and the four-layer pass takes as long (2^26
// elements of 4096 lanes 496 us, 475 with shifts): the issue slots bound it too.
constexpr int kGPairBytes = 65536;

__device__ __forceinline__ int group_slot(int j) { return (j >> 1) * kGPairBytes + (j & 1) * 128; }
// The third table of a three-layer pass stands alone.
template <int K>
constexpr int group_pitch(int j) { return K == 3 && j == 2 ? 128 : 256; }

// Row offset of byte r of w in a table of row pitch P.
template <int P>
__device__ __forceinline__ uint32_t byte_row(uint32_t w, int r) {
    if constexpr (P == 256)
        return (r == 0 ? w << 8 : w >> (8 * r - 8)) & 0xFF00u;
    else
        return (r == 0 ? w << 7 : w >> (8 * r - 7)) & 0x7F80u;
}

template <int W, int P>
__device__ __forceinline__ void group_build_item(char *tb, uint4 t, int u) {
    if constexpr (W == 4) {
        const int s = u & 7, hi = (u >> 3) & 15;
        uint4 b[8];
        b[0] = gf_mul_xpow(t, (uint32_t)(8 * s));
#pragma unroll
        for (int e = 1; e < 8; ++e) b[e] = gf_mul_x(b[e - 1]);
        uint4 H = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if ((hi >> q) & 1) H = gf_add(H, b[4 + q]);
        uint4 L[16];
        L[0] = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int x = 1; x < 16; ++x) {
            const int low = x & -x;
            L[x] = gf_add(L[x & (x - 1)], b[low == 1 ? 0 : low == 2 ? 1 : low == 4 ? 2 : 3]);
        }
#pragma unroll
        for (int lo = 0; lo < 16; ++lo)
            *reinterpret_cast<uint4 *>(tb + ((hi << 4) | lo) * P + s * 16) = gf_add(H, L[lo]);
    } else {
        // half of row x's copies, rotated by x: a warp's stores cover the banks
        constexpr int copies = W == 1 ? 32 : 16, half = copies / 2;
        const uint64_t t64 = lo64(t);
        const uint32_t x = (uint32_t)u >> 1, h = (uint32_t)u & 1;
        uint64_t p = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if ((x >> i) & 1) p ^= t64 << i;
        char *row = tb + x * P;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const uint32_t c = h * half + ((i + x) & (half - 1));
            if (W == 1)
                reinterpret_cast<uint32_t *>(row)[c] = (uint32_t)p;
            else
                reinterpret_cast<uint2 *>(row)[c] = make_uint2((uint32_t)p, (uint32_t)(p >> 32));
        }
    }
}

// Per-thread lookup order of the byte tables (t8.cuh) or copy of the compact
// ones.
struct GroupLane {
    uint32_t off[8], r;
    __device__ __forceinline__ void init() {
        r = threadIdx.x & 7;
#pragma unroll
        for (int m = 0; m < 8; ++m) off[m] = ((m + r) & 7) << 4;
    }
    __device__ __forceinline__ void rot(uint32_t &a, uint32_t &b) const {
        const uint32_t x = (r & 4) ? b : a, y = (r & 4) ? a : b;
        const uint32_t sh = (r & 3) << 3;
        a = __funnelshift_r(x, y, sh);
        b = __funnelshift_r(y, x, sh);
    }
};

// x[0 .. 5] ^= v * s, unreduced above bit 128 (byte tables: reduced).
template <int W, int P>
__device__ __forceinline__ void group_lookup(const GroupLane &lc, const char *tb, uint4 v,
                                             uint32_t *x) {
    if constexpr (W == 4) {
        uint32_t l0 = v.x, l1 = v.y, h0 = v.z, h1 = v.w;
        lc.rot(l0, l1);
        lc.rot(h0, h1);
        uint4 A = make_uint4(x[0], x[1], x[2], x[3]), B = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const uint32_t xl = byte_row<P>(m < 4 ? l0 : l1, m & 3);
            const uint32_t xh = byte_row<P>(m < 4 ? h0 : h1, m & 3);
            A = gf_add(A, *reinterpret_cast<const uint4 *>(tb + (xl | lc.off[m])));
            B = gf_add(B, *reinterpret_cast<const uint4 *>(tb + (xh | lc.off[m])));
        }
        // A + X^64 B
        const uint64_t g1 = (uint64_t)B.z | ((uint64_t)B.w << 32);
        const uint64_t f_lo = g1 ^ (g1 << 1) ^ (g1 << 2) ^ (g1 << 7);
        const uint64_t f_hi = (g1 >> 63) ^ (g1 >> 62) ^ (g1 >> 57);
        x[0] = A.x ^ (uint32_t)f_lo;
        x[1] = A.y ^ (uint32_t)(f_lo >> 32);
        x[2] = A.z ^ B.x ^ (uint32_t)f_hi;
        x[3] = A.w ^ B.y;
    } else {
        const uint32_t lane_off = W == 1 ? (threadIdx.x & 31) << 2 : (threadIdx.x & 15) << 3;
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        constexpr int NS = W == 1 ? 4 : 5;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            // S = XOR_q u[byte r of word q] << 32 q, then x ^= S << 8 r
            uint32_t S[NS];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t a = byte_row<P>(w[q], r) | lane_off;
                if constexpr (W == 1) {
                    S[q] = *reinterpret_cast<const uint32_t *>(tb + a);
                } else {
                    const uint2 u = *reinterpret_cast<const uint2 *>(tb + a);
                    S[q] = q == 0 ? u.x : S[q] ^ u.x;
                    S[q + 1] = u.y;
                }
            }
#pragma unroll
            for (int k = 0; k <= NS; ++k) {
                const uint32_t hi = k < NS ? S[k] : 0u, lo = k > 0 ? S[k - 1] : 0u;
                if (r == 0) { if (k < NS) x[k] ^= hi; }
                else x[k] ^= __funnelshift_l(lo, hi, 8 * r);
            }
        }
    }
}

// ---- offsets -------------------------------------------------------------------
// x[i][o ..] ^= v[i] * e over the set bits of e, two at a time, for N
// operands: a wide multiply by the bit's power of two gives both halves of
// each shifted word on the FMA pipe.
template <int N, int NX>
__device__ __forceinline__ void mul_bits_into(uint32_t (&x)[N][NX], const uint4 *v, uint32_t e,
                                              int o) {
    while (e) {
        const uint32_t m = e & (0u - e);
        e ^= m;
        const uint32_t n = e & (0u - e);
        e ^= n;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
            uint64_t p[4], q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                p[k] = (uint64_t)w[k] * m;
                q[k] = (uint64_t)w[k] * n;
            }
            x[i][o] ^= (uint32_t)p[0] ^ (uint32_t)q[0];
#pragma unroll
            for (int k = 1; k < 4; ++k)
                x[i][o + k] ^= ((uint32_t)p[k] ^ (uint32_t)(p[k - 1] >> 32)) ^
                               ((uint32_t)q[k] ^ (uint32_t)(q[k - 1] >> 32));
            x[i][o + 4] ^= (uint32_t)(p[3] >> 32) ^ (uint32_t)(q[3] >> 32);
        }
    }
}

// x[0 .. 4] ^= v * e for a compile-time e of at most 5 bits (after unrolling).
BZ_HD void mul_small_into(uint32_t *x, uint4 v, uint32_t e) {
#pragma unroll
    for (int b = 1; b < 5; ++b)
        if ((e >> b) & 1) {
            x[0] ^= v.x << b;
            x[1] ^= __funnelshift_l(v.x, v.y, b);
            x[2] ^= __funnelshift_l(v.y, v.z, b);
            x[3] ^= __funnelshift_l(v.z, v.w, b);
            x[4] ^= v.w >> (32 - b);
        }
}

// Twiddle of sub-block sb at depth d of the zero block, for the deepest four
// layers: XOR over the bits i of sb of the complete homogeneous symmetric
// polynomial of degree i + 1 in X, X^2, .., X^(2^d).
__host__ __device__ constexpr uint32_t group_const(int d, int sb) {
    uint32_t r = 0;
    if (d == 0) r = (uint32_t)sb << 1;
    if (d == 1) r = ((sb & 1) ? 0x6u : 0u) ^ ((sb & 2) ? 0x1Cu : 0u);
    if (d == 2) r = (sb & 1) ? 0x16u : 0u;
    return r;
}

// x mod X^128 + X^7 + X^2 + X + 1.  NX = 5: at most 24 bits above 128;
// NX = 6: at most 56; NX = 8: 128.
template <int NX>
__device__ __forceinline__ uint4 group_reduce(const uint32_t (&x)[NX]) {
    if constexpr (NX == 8) {
        return gf_reduce32(x);
    } else if constexpr (NX == 5) {
        const uint32_t h = x[4];
        return make_uint4(x[0] ^ (h ^ (h << 1) ^ (h << 2) ^ (h << 7)), x[1], x[2], x[3]);
    } else {
        const uint64_t h = (uint64_t)x[4] | ((uint64_t)x[5] << 32);
        const uint64_t f = h ^ (h << 1) ^ (h << 2) ^ (h << 7);
        return make_uint4(x[0] ^ (uint32_t)f, x[1] ^ (uint32_t)(f >> 32), x[2], x[3]);
    }
}

// ---- layers ----------------------------------------------------------------------
// Layer J of K on v.  EW = 0: blocks of at least blockDim.x tasks, the pass
// ends at depth 0, the offset is the sub-block's compile-time constant.
// EW = 2: the same layers with the block's offset twiddle eb (two words, below
// 2^56) added.  EW = 4: any depth; the sub-block's part comes from the heap's
// entries of the zero block.
template <int K, int J, int W, int EW>
__device__ __forceinline__ void group_layer(uint4 (&v)[1 << K], const GroupLane &lc,
                                            const char *tb, const uint32_t *eb,
                                            const uint4 *tw_zero) {
    constexpr int half = 1 << (K - 1 - J);
    constexpr int NX = EW == 4 ? 8 : (EW == 2 || W == 2) ? 6 : 5;
#pragma unroll
    for (int sb = 0; sb < (1 << J); ++sb) {
        const uint32_t c = EW < 4 ? group_const(K - 1 - J, sb) : 0u;
        uint4 *u = &v[sb * 2 * half], *w = u + half;
        if constexpr (EW == 0) {
#pragma unroll
            for (int i = 0; i < half; ++i) {
                uint32_t x[6] = {u[i].x, u[i].y, u[i].z, u[i].w, 0, 0};
                mul_small_into(x, w[i], c);
                group_lookup<W, group_pitch<K>(J)>(lc, tb, w[i], x);
                uint32_t y[NX];
#pragma unroll
                for (int k = 0; k < NX; ++k) y[k] = x[k];
                u[i] = group_reduce<NX>(y);
                w[i] = gf_add(w[i], u[i]);
            }
        } else {
            uint32_t x[half][NX];
#pragma unroll
            for (int i = 0; i < half; ++i) {
                x[i][0] = u[i].x;
                x[i][1] = u[i].y;
                x[i][2] = u[i].z;
                x[i][3] = u[i].w;
#pragma unroll
                for (int k = 4; k < NX; ++k) x[i][k] = 0;
            }
            if constexpr (EW == 2) {
                mul_bits_into(x, w, eb[0] ^ c, 0);
                mul_bits_into(x, w, eb[1], 1);
            } else {
                const uint4 z = __ldg(tw_zero + sb);
                mul_bits_into(x, w, eb[0] ^ z.x, 0);
                mul_bits_into(x, w, eb[1] ^ z.y, 1);
                mul_bits_into(x, w, eb[2] ^ z.z, 2);
                mul_bits_into(x, w, eb[3] ^ z.w, 3);
            }
#pragma unroll
            for (int i = 0; i < half; ++i) {
                group_lookup<W, group_pitch<K>(J)>(lc, tb, w[i], x[i]);
                u[i] = group_reduce<NX>(x[i]);
                w[i] = gf_add(w[i], u[i]);
            }
        }
    }
}

// Body: chunks [c_beg, c_end) of blockDim.x (a power of two) tasks; tbl holds
// K tables.  Task = (block, row below `depth`, lane), lanes fastest.
template <int K, int W0, int W1, int W2, int W3, int EW, bool PF>
__device__ __forceinline__ void group_pass_body(const GroupPassArgs &a, uint64_t c_beg,
                                                uint64_t c_end, char *tbl) {
    GroupLane lc;
    lc.init();
    const int depth = EW < 4 ? 0 : a.depth;
    const int log_task_per_b = depth + a.log_lanes;
    const uint64_t lanes_mask = ((uint64_t)1 << a.log_lanes) - 1;
    const uint64_t row_mask = ((uint64_t)1 << depth) - 1;
    const uint64_t src_mask = ((uint64_t)1 << a.src_pos_bits) - 1;
    const int top = a.ell - depth - K;  // layer of J = 0
    constexpr int NE = EW ? EW : 1;
    uint32_t eb[K][NE];
    if constexpr (EW > 0) {
        // the thread's block offset in its chunk: the same for every chunk
        const uint64_t off = log_task_per_b < 32 ? threadIdx.x >> log_task_per_b : 0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const uint4 t = a.tw[((uint64_t)1 << (top + j)) + (off << j)];
            eb[j][0] = t.x;
            eb[j][1] = t.y;
            if constexpr (EW == 4) {
                eb[j][2] = t.z;
                eb[j][3] = t.w;
            }
        }
    }
    auto load = [&](uint64_t c, uint4 (&v)[1 << K]) {
        const uint64_t task = c * blockDim.x + threadIdx.x;
        const uint64_t pbase = ((task >> log_task_per_b) << (depth + K)) +
                               ((task >> a.log_lanes) & row_mask);
#pragma unroll
        for (int i = 0; i < (1 << K); ++i) {
            const uint64_t p = pbase + ((uint64_t)i << depth);
            v[i] = __ldcs(a.src + (((p & src_mask) << a.log_lanes) | (task & lanes_mask)));
        }
    };
    auto build = [&](uint64_t B0) {
        constexpr int n0 = build_items<W0>(), n1 = build_items<W1>(), n2 = build_items<W2>();
        constexpr int n3 = K > 3 ? build_items<W3>() : 0;
        for (int u = threadIdx.x; u < n0 + n1 + n2 + n3; u += blockDim.x) {
            const int j = u < n0 ? 0 : u < n0 + n1 ? 1 : u < n0 + n1 + n2 ? 2 : 3;
            const uint4 t = __ldg(a.tw + ((uint64_t)1 << (top + j)) + (B0 << j));
            if (j == 0) group_build_item<W0, group_pitch<K>(0)>(tbl + group_slot(0), t, u);
            else if (j == 1)
                group_build_item<W1, group_pitch<K>(1)>(tbl + group_slot(1), t, u - n0);
            else if (j == 2)
                group_build_item<W2, group_pitch<K>(2)>(tbl + group_slot(2), t, u - n0 - n1);
            else if constexpr (K > 3)
                group_build_item<W3, group_pitch<K>(3)>(tbl + group_slot(3), t,
                                                        u - n0 - n1 - n2);
        }
    };
    // the first chunk's tables are built ahead of the wait; its barrier below
    build((c_beg * blockDim.x) >> log_task_per_b);
    chain_wait();
    uint64_t cur = (c_beg * blockDim.x) >> log_task_per_b;
    bool built = true;  // since the last barrier
    uint4 nxt[1 << K];
    if (PF && c_beg < c_end) load(c_beg, nxt);
    for (uint64_t c = c_beg; c < c_end; ++c) {
        const uint64_t task = c * blockDim.x + threadIdx.x;
        const uint64_t B = task >> log_task_per_b;
        const uint64_t pbase = (B << (depth + K)) + ((task >> a.log_lanes) & row_mask);
        const uint64_t ln = task & lanes_mask;
        uint4 v[1 << K];
        if constexpr (PF) {
#pragma unroll
            for (int i = 0; i < (1 << K); ++i) v[i] = nxt[i];
            if (c + 1 < c_end) load(c + 1, nxt);
        } else {
            load(c, v);
        }
        const uint64_t B0 = (c * blockDim.x) >> log_task_per_b;  // uniform
        if (B0 != cur) {
            __syncthreads();  // every lookup into the previous tables is done
            build(B0);
            built = true;
            cur = B0;
        }
        if (built) __syncthreads();
        built = false;
        group_layer<K, 0, W0, EW>(v, lc, tbl + group_slot(0), eb[0],
                                  a.tw + ((uint64_t)1 << top));
        group_layer<K, 1, W1, EW>(v, lc, tbl + group_slot(1), eb[1],
                                  a.tw + ((uint64_t)1 << (top + 1)));
        group_layer<K, 2, W2, EW>(v, lc, tbl + group_slot(2), eb[2],
                                  a.tw + ((uint64_t)1 << (top + 2)));
        if constexpr (K > 3)
            group_layer<K, 3, W3, EW>(v, lc, tbl + group_slot(3), eb[3],
                                      a.tw + ((uint64_t)1 << (top + 3)));
#pragma unroll
        for (int i = 0; i < (1 << K); ++i) {
            const uint64_t p = pbase + ((uint64_t)i << depth);
            __stcs(a.dst + ((p << a.log_lanes) | ln), v[i]);
        }
    }
}

}  // namespace bz
