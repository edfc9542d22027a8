// Opening-time kernels: sumcheck lane folds and messages
// (flock-core/src/pcs/ligerito.rs), the ring-switch passes (BitZ
// src/ligerito.rs), the eq table (src/poly/utils.rs) and the ChaCha20 input
// generator.
//
// Field sums are exact and order independent, so partial sums per CTA are
// XOR-reduced as unreduced 256-bit values and reduced once at the end, which
// is bit-identical to the reference's per-term sums (ligerito.rs:2646-2649).
#include <cuda_runtime.h>

#include <algorithm>

#include "bz_internal.h"
#include "chain.cuh"
#include "gf128.cuh"
#include "post.cuh"
#include "t16.cuh"
#include "t8.cuh"

namespace bz {

__device__ __forceinline__ uint64_t warp_xor64(uint64_t v) {
    const uint32_t lo = __reduce_xor_sync(0xffffffffu, (uint32_t)v);
    const uint32_t hi = __reduce_xor_sync(0xffffffffu, (uint32_t)(v >> 32));
    return (uint64_t)lo | ((uint64_t)hi << 32);
}

// Word w = lane mod 8 of the XOR of n rows of 8 words (one warp; every lane
// returns its word).
template <typename Load>
__device__ __forceinline__ uint64_t rows_xor(int n, Load row_word) {
    const int ln = threadIdx.x & 31, w = ln & 7;
    uint64_t a = 0;
    for (int i = ln >> 3; i < n; i += 4) a ^= row_word(i, w);
    a ^= __shfl_xor_sync(0xffffffffu, a, 8);
    return a ^ __shfl_xor_sync(0xffffffffu, a, 16);
}

// XOR of two wide accumulators over the CTA: lanes of warp 0 return word
// (lane mod 8) of {u0, u2}.
__device__ __forceinline__ uint64_t cta_xor_pair(const gf_wide &u0, const gf_wide &u2) {
    __shared__ uint64_t red[32][8];
    const int w = threadIdx.x >> 5, ln = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint64_t x = warp_xor64(u0.w[i]), y = warp_xor64(u2.w[i]);
        if (ln == 0) {
            red[w][i] = x;
            red[w][4 + i] = y;
        }
    }
    __syncthreads();
    if (w != 0) return 0;
    return rows_xor((int)(blockDim.x >> 5), [&](int i, int k) { return red[i][k]; });
}

// Dynamic shared memory of the kernels that multiply by one challenge r
// through byte tables: the 64 KB table of r and its 128 basis products
// (padded to kT16Bases).
constexpr size_t kRTableSmem = (size_t)kT16Entries * 16 + kT16Bases * 16;

// Build the byte tables of r in shared memory (all threads; syncs inside).
__device__ __forceinline__ const char *build_r_table(uint4 *smem, uint4 r) {
    __shared__ uint4 rs[1];
    if (threadIdx.x == 0) rs[0] = r;
    __syncthreads();
    t16_build(smem, smem + kT16Entries, rs, 1);
    return reinterpret_cast<const char *>(smem);
}

// {u0, u2} from the eight words of their unreduced sums, word i in lane i of
// the calling warp: lane 0 returns u0 and lane 1 u2, reduced.
__device__ __forceinline__ uint4 reduce_pair(uint64_t word) {
    gf_wide x;
    const int t = threadIdx.x & 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) x.w[i] = __shfl_sync(0xffffffffu, word, 4 * t + i);
    return gf_reduce(x);
}

// Where a message goes: a mailbox in mapped host memory, as tagged elements.
// With a system-scope release store of a flag (and the sums reduced by
// shuffles) the end of a one-CTA round took 1.74 us, now 0.45.  Without a
// mailbox (ticket null) the caller launches finish_msg_kernel.
struct MsgMailbox {
    unsigned int *ticket = nullptr;  // device counter, 0 between launches
    uint64_t *words = nullptr;       // mapped host memory: u0, u2
    uint32_t seq_val = 0;
    uint32_t release = 0;            // release the folded arrays before the post
};

// Lanes 0 and 1 of the calling warp post u0 and u2, behind a barrier that
// follows the CTA's stores.  RELEASE is false in the kernels whose arrays only
// the provers read: GKR rounds pay 0.3 us each for the fence's branch and code.
template <bool RELEASE>
__device__ __forceinline__ void post_pair(uint64_t word, const MsgMailbox &mb) {
    const uint4 v = reduce_pair(word);
    const int ln = threadIdx.x & 31;
    if (RELEASE && mb.release) post_release();
    if (ln < 2) post_element(mb.words + 4 * ln, mb.seq_val, v);
}

// XOR of the partials (8 words each) of n CTAs, by all threads; lanes of warp
// 0 return word (lane mod 8).  Partials are read from L2 (other CTAs wrote
// them in this launch or the previous one).
constexpr int kFinishThreads = 256;
__device__ uint64_t partials_xor(const uint64_t *partials, int n) {
    __shared__ uint64_t red[32][8];
    const int nw = blockDim.x >> 5, wp = threadIdx.x >> 5, ln = threadIdx.x & 31;
    const int rows = n > wp * 4 ? (n - wp * 4 + 4 * nw - 1) / (4 * nw) * 4 : 0;
    const uint64_t a = rows_xor(rows, [&](int i, int k) {
        const int row = (i >> 2) * 4 * nw + wp * 4 + (i & 3);
        return row < n ? __ldcg(partials + (uint64_t)row * 8 + k) : 0;
    });
    if (ln < 8) red[wp][ln] = a;
    __syncthreads();
    if (wp != 0) return 0;
    return rows_xor(nw, [&](int i, int k) { return red[i][k]; });
}

// The CTA's sums (word (lane mod 8) in the lanes of warp 0).  With a mailbox
// and up to kMsgPosts CTAs, each posts its own and the host adds them (0.2 us;
// the ticket takes 0.9 to 2.1).  Otherwise every CTA stores its partial, and
// with a mailbox the last one (whose ticket completes the count) reduces them
// all, posts and resets the ticket for the next launch.
template <bool RELEASE>
__device__ __forceinline__ void msg_out(uint64_t word, uint64_t *partials, MsgMailbox mb) {
    if (mb.ticket && msg_posts(gridDim.x) == (int)gridDim.x) {
        mb.words += 8 * blockIdx.x;
        if (threadIdx.x < 32) post_pair<RELEASE>(word, mb);
        return;
    }
    if (threadIdx.x < 8) partials[(uint64_t)blockIdx.x * 8 + threadIdx.x] = word;
    if (!mb.ticket) return;
    __shared__ int last;
    if (threadIdx.x < 32) {
        __threadfence();  // this CTA's partial, by the lanes that wrote it
        __syncwarp();
        if (threadIdx.x == 0) last = atomicAdd(mb.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const uint64_t sum = partials_xor(partials, (int)gridDim.x);
    if (threadIdx.x < 32) post_pair<RELEASE>(sum, mb);
    if (threadIdx.x == 0) *mb.ticket = 0;
}

template <bool RELEASE>
__device__ __forceinline__ void msg_finish(const gf_wide &u0, const gf_wide &u2,
                                           uint64_t *partials, const MsgMailbox &mb) {
    msg_out<RELEASE>(cta_xor_pair(u0, u2), partials, mb);
}

// Out of line for the fold kernel: its loop runs at the 128-register cap, and
// an inlined epilogue adds spills to it.
template <bool RELEASE>
__device__ __noinline__ void msg_finish_call(gf_wide u0, gf_wide u2, uint64_t *partials,
                                             const MsgMailbox &mb) {
    msg_finish<RELEASE>(u0, u2, partials, mb);
}

__device__ __forceinline__ uint64_t ld_relaxed_sys(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Warp 0 of each CTA polls the gate's four words, sleeping between polls,
// until all carry the round's number (open: together they hold r, as
// post_element lays it out, so one access brings both), the first carries the
// number with its top bit set (cancelled) or the time limit passes (bit 0 of
// *err is set).  Returns whether the gate opened; r is then the posted
// challenge.
__device__ bool gate_wait(const RGate &g, uint4 &r) {
    __shared__ uint4 rs;
    __shared__ int open;
    if (threadIdx.x < 32) {
        const uint64_t t0 = globaltimer_ns();
        const int ln = threadIdx.x;
        int st = 0;
        uint64_t v = 0;
        for (;;) {
            if (ln < 4) v = ld_relaxed_sys(g.words + ln);
            const uint32_t tag = (uint32_t)(v >> 32);
            if (__all_sync(0xffffffffu, ln >= 4 || tag == g.seq)) {
                st = 1;
                break;
            }
            if (__any_sync(0xffffffffu, ln == 0 && tag == (g.seq | kGateCancel))) break;
            if (__any_sync(0xffffffffu, ln == 0 && globaltimer_ns() - t0 > g.limit_ns)) {
                if (ln == 0) atomicOr(g.err, 1u);
                break;
            }
            __nanosleep(128);
        }
        const uint32_t x = __shfl_sync(0xffffffffu, (uint32_t)v, 0);
        const uint32_t y = __shfl_sync(0xffffffffu, (uint32_t)v, 1);
        const uint32_t z = __shfl_sync(0xffffffffu, (uint32_t)v, 2);
        const uint32_t w = __shfl_sync(0xffffffffu, (uint32_t)v, 3);
        if (ln == 0) {
            rs = make_uint4(x, y, z, w);
            open = st;
        }
    }
    __syncthreads();
    r = rs;
    return open != 0;
}

// nf[j] = f[2j] + (f[2j] + f[2j+1]) * r (same for b); thread k produces the
// folded pair (2k, 2k+1) and its message terms.  The four multiplies by the
// challenge r use r's byte tables; the two variable products of the message
// use the generic carry-less multiply.  Registers are capped at 128 so two
// CTAs share an SM (a few spilled words cost less than half the warps: the
// 2^24 first fold takes 0.30 ms instead of 0.35 ms).
// GATED: launched before r is known; r comes through the gate instead (a
// cancelled or timed-out CTA returns before touching the arrays or the
// mailbox ticket).
template <bool GATED>
__global__ void __launch_bounds__(256, 2) fold_and_msg_kernel(const uint4 *f, const uint4 *b,
                                                           uint64_t half, uint4 r, uint4 *nf,
                                                           uint4 *nb, uint64_t *partials,
                                                           MsgMailbox mb, RGate gate) {
    chain_wait();
    extern __shared__ uint4 smem[];
    if constexpr (GATED) {
        if (!gate_wait(gate, r)) return;
    }
    const char *T = build_r_table(smem, r);
    T16Lane8 lc;
    lc.init();
    gf_wide u0 = gf_wide_zero(), u2 = gf_wide_zero();
    const uint64_t pairs = half >> 1;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < pairs;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 *fp = f + 4 * k, *bp = b + 4 * k;
        const uint4 f0 = fp[0], f1 = fp[1], f2 = fp[2], f3 = fp[3];
        const uint4 b0 = bp[0], b1 = bp[1], b2 = bp[2], b3 = bp[3];
        const uint4 x0 = gf_add(f0, lc.mul(T, gf_add(f0, f1)));
        const uint4 x1 = gf_add(f2, lc.mul(T, gf_add(f2, f3)));
        const uint4 y0 = gf_add(b0, lc.mul(T, gf_add(b0, b1)));
        const uint4 y1 = gf_add(b2, lc.mul(T, gf_add(b2, b3)));
        nf[2 * k] = x0;
        nf[2 * k + 1] = x1;
        nb[2 * k] = y0;
        nb[2 * k + 1] = y1;
        gf_wide_xor(u0, gf_mul_wide(x0, y0));
        gf_wide_xor(u2, gf_mul_wide(gf_add(x0, x1), gf_add(y0, y1)));
    }
    msg_finish_call<true>(u0, u2, partials, mb);
}

__global__ void __launch_bounds__(256) round_msg_kernel(const uint4 *f, const uint4 *b,
                                                        uint64_t pairs, uint64_t *partials,
                                                        MsgMailbox mb) {
    chain_wait();
    gf_wide u0 = gf_wide_zero(), u2 = gf_wide_zero();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < pairs;
         j += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 f0 = f[2 * j], f1 = f[2 * j + 1], b0 = b[2 * j], b1 = b[2 * j + 1];
        gf_wide_xor(u0, gf_mul_wide(f0, b0));
        gf_wide_xor(u2, gf_mul_wide(gf_add(f0, f1), gf_add(b0, b1)));
    }
    msg_finish<false>(u0, u2, partials, mb);
}

// Final XOR of per-CTA partials and the single reduction: out = {u0, u2}.
__global__ void __launch_bounds__(kFinishThreads) finish_msg_kernel(const uint64_t *partials,
                                                                    int n, uint64_t *out) {
    chain_wait();
    const uint64_t sum = partials_xor(partials, n);
    if (threadIdx.x >= 32) return;
    const uint4 v = reduce_pair(sum);
    if (threadIdx.x < 2) {
        out[2 * threadIdx.x] = lo64(v);
        out[2 * threadIdx.x + 1] = hi64(v);
    }
}

// ---------------------------------------------------------------------------
// Small rounds.  A round over few slots is the latency of its own chain: the
// byte tables of the challenge (0.84 us to build), one lookup product and up
// to three variable products a thread, each of 144 wide multiply-adds one
// after the other (0.6 us).  Here a CTA has nine warps and warp q computes the
// q-th 32x32 product of the Karatsuba tree for 32 products at a time, through
// shared memory: no tables, and a product takes 0.35 to 0.5 us of latency.  The
// message sums need no recombination per product: each warp sums its own part
// and the parts of the total are combined once.  A sumcheck round of one CTA
// takes 1.7 us on the device instead of 4.7, a GKR round 1.6 us behind its
// challenge instead of 6.7.
// ---------------------------------------------------------------------------
constexpr int kCoopThreads = 288;
constexpr int kCoopSlots = 64;  // slots a CTA takes at a time at most (4 elements each)

// Part q = 3 u + v of the operand: u picks the low or high 64-bit half or
// their sum, v the same of its 32-bit halves.
struct CoopPart {
    uint32_t m[4];
    __device__ __forceinline__ explicit CoopPart(int q) {
        const int u = q / 3, v = q - 3 * u;
        const uint32_t lo = u == 1 ? 0u : ~0u, hi = u == 0 ? 0u : ~0u;
        const uint32_t even = v == 1 ? 0u : ~0u, odd = v == 0 ? 0u : ~0u;
        m[0] = lo & even;
        m[1] = lo & odd;
        m[2] = hi & even;
        m[3] = hi & odd;
    }
    __device__ __forceinline__ uint32_t of(uint4 a) const {
        return (a.x & m[0]) ^ (a.y & m[1]) ^ (a.z & m[2]) ^ (a.w & m[3]);
    }
};

// The unreduced product from its nine parts.
template <typename Part>
__device__ __forceinline__ gf_wide coop_combine(Part part) {
    uint64_t lo[3], hi[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
        const uint64_t l = part(3 * u), h = part(3 * u + 1), m = part(3 * u + 2) ^ l ^ h;
        lo[u] = l ^ (m << 32);
        hi[u] = h ^ (m >> 32);
    }
    const uint64_t m0 = lo[2] ^ lo[0] ^ lo[1], m1 = hi[2] ^ hi[0] ^ hi[1];
    gf_wide r;
    r.w[0] = lo[0];
    r.w[1] = hi[0] ^ m0;
    r.w[2] = lo[1] ^ m1;
    r.w[3] = hi[1];
    return r;
}

// f(p, p < n) for p = lane, lane + 32, .. up to n - 1: U at a time where there
// is more than one, so that their latencies overlap (p stays below the next
// multiple of 32 U).
template <int U, typename F>
__device__ __forceinline__ void coop_each(int n, F f) {
    const int ln = threadIdx.x & 31;
    if (n <= 32) {
        f(ln, ln < n);
        return;
    }
    for (int p = ln; p - ln < n; p += 32 * U) {
#pragma unroll
        for (int u = 0; u < U; ++u) f(p + 32 * u, p + 32 * u < n);
    }
}

// A round over h slots.  GKR: the tables a, b hold entry i of slot c at c +
// i h and a fold joins the entries at i h and (i + 2) h; the sums are weighted
// by w.  Otherwise (the sumcheck): entry i of slot c is at 2 c + i and a fold
// joins 2 j and 2 j + 1.  Folded tables go to na, nb, which are not the inputs
// (a gate that runs out in some CTAs leaves the round to be run again).
struct CoopRound {
    const uint4 *a, *b;
    uint4 *na, *nb;
    const uint4 *w;
    uint4 *w_next;
    uint64_t *tail;  // mapped: the round's four entries, 4 tagged words each
    uint64_t h;
    int per;  // slots a CTA takes at a time
    uint4 r;
    int send_one;
    int single;  // a sumcheck fold to one element: no message
    uint64_t *partials;
    MsgMailbox mb;
};

template <bool GKR, bool FOLD, bool GATED>
__global__ void __launch_bounds__(kCoopThreads) coop_round_kernel(
    const __grid_constant__ CoopRound a, const __grid_constant__ RGate gate) {
    __shared__ uint4 mul[4 * kCoopSlots];  // multiplicands: differences, then weighted entries
    __shared__ uint4 ent[4 * kCoopSlots];  // entry 4 slot + 2 table + i
    __shared__ uint4 wgt[kCoopSlots];
    __shared__ uint64_t prod[9][4 * kCoopSlots];
    __shared__ uint64_t sums[9][2];
    const int tid = threadIdx.x, q = tid >> 5, ln = tid & 31;
    const CoopPart part(q);
    const uint64_t h = a.h;
    uint4 r = a.r;
    uint32_t rp = 0;
    uint64_t acc = 0;  // even lanes: the first sum's part, odd lanes: the second's
    chain_wait();
    for (uint64_t c0 = (uint64_t)blockIdx.x * a.per; c0 < h;
         c0 += (uint64_t)gridDim.x * a.per) {
        const int ns = (int)(h - c0 < a.per ? h - c0 : a.per);
        // thread 4 slot + 2 table + i loads its entry (GATED: before the challenge)
        uint64_t dst = 0;
        const int i = tid & 1;
        const bool mine = tid < 4 * ns && !(a.single && i);
        uint4 base = make_uint4(0, 0, 0, 0), diff = base;
        if (mine) {
            const uint64_t c = c0 + (tid >> 2);
            const uint4 *t = (tid & 2) ? a.b : a.a;
            dst = GKR ? c + i * h : 2 * c + i;
            if constexpr (FOLD) {
                base = t[GKR ? dst : 2 * dst];
                diff = gf_add(base, t[GKR ? dst + 2 * h : 2 * dst + 1]);
            } else {
                base = t[dst];
            }
        }
        // the last threads: a slot's weight, and the next round's
        const int sw = tid - (kCoopThreads - kCoopSlots);
        const uint64_t cw = c0 + sw;
        const bool weigh = GKR && sw >= 0 && sw < ns;
        const bool weigh_next = weigh && a.w_next && cw < h / 2;
        uint4 wn = base;
        if (weigh) {
            const uint4 wc = a.w[cw];
            wgt[sw] = wc;
            if (weigh_next) wn = gf_add(wc, a.w[cw + h / 2]);
        }
        if constexpr (FOLD) {
            if (tid < 4 * ns) mul[tid] = diff;
            if (GATED && c0 == (uint64_t)blockIdx.x * a.per) {
                if (!gate_wait(gate, r)) return;
            }
            __syncthreads();
            rp = part.of(r);
            coop_each<4>(4 * ns, [&](int p, bool) { prod[q][p] = clmul32(part.of(mul[p]), rp); });
            __syncthreads();
            if (mine) {
                base = gf_add(base, gf_reduce(coop_combine([&](int k) { return prod[k][tid]; })));
                ((tid & 2) ? a.nb : a.na)[dst] = base;
            }
        }
        // written after the gate, as all of global memory: the round behind one
        // whose gate ran out must leave that round's inputs as they are
        if (weigh_next) a.w_next[cw] = wn;
        if (tid < 4 * ns) ent[tid] = base;
        __syncthreads();
        // products 2 slot + t of the message: t = 0 the end value, 1 the difference
        auto operand = [&](int p, int table) {
            const uint4 *e = ent + 4 * (p >> 1) + 2 * table;
            if (p & 1) return gf_add(e[0], e[1]);
            return e[GKR && a.send_one];
        };
        if constexpr (GKR) {
            if (a.tail && tid < 4) post_element(a.tail + 4 * tid, a.mb.seq_val, base);
            coop_each<2>(2 * ns, [&](int p, bool) {
                prod[q][p] = clmul32(part.of(operand(p, 0)), part.of(wgt[p >> 1]));
            });
            __syncthreads();
            if (tid < 2 * ns)
                mul[tid] = gf_reduce(coop_combine([&](int k) { return prod[k][tid]; }));
            __syncthreads();
        }
        if (!a.single)
            coop_each<2>(2 * ns, [&](int p, bool in) {
                const uint64_t v =
                    clmul32(part.of(GKR ? mul[p] : operand(p, 0)), part.of(operand(p, 1)));
                acc ^= in ? v : 0;
            });
        __syncthreads();
    }
    const uint64_t s0 = warp_xor64((ln & 1) ? 0 : acc), s1 = warp_xor64((ln & 1) ? acc : 0);
    if (ln == 0) {
        sums[q][0] = s0;
        sums[q][1] = s1;
    }
    __syncthreads();
    // word (lane mod 8) of {sum 0, sum 1} in warp 0
    uint64_t word = 0;
    if (tid < 8) {
        const gf_wide x = coop_combine([&](int k) { return sums[k][tid >> 2]; });
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if ((tid & 3) == k) word = x.w[k];
    }
    msg_out<FOLD && !GKR>(word, a.partials, a.mb);
}

// Up to kMsgPosts CTAs while they take at most kCoopSlots each (the host adds
// their sums), at least 8 slots (one step of the fold's products) each; above,
// the ticket is paid for and half the slots a CTA halve its steps.
static int coop_per(uint64_t slots) {
    if (slots <= kMsgPosts * kCoopSlots)
        return (int)std::max<uint64_t>(8, (slots + kMsgPosts - 1) / kMsgPosts);
    return slots <= 4096 ? kCoopSlots / 2 : kCoopSlots;
}

// CTAs of a small round over `slots` slots, 0 above `limit`, where the table
// kernels (or a thread a product) are as fast or faster.  Through the public
// calls: a fold to 2^13 pairs 18.6 us (tables 19.8) and to 2^14 20.8 (20.2); a
// message alone over 2^12 pairs 14.9 (15.0) and over 2^14 16.4 (15.3); GKR
// rounds may be armed below the limit, 2^22 leaves take 2.70 ms at 2^13, 2.65 at
// 2^14 and 2.68 at 2^15.
constexpr uint64_t kCoopFoldSlots = 1 << 13, kCoopMsgSlots = 1 << 12, kCoopGkrSlots = 1 << 14;
static int coop_grid(uint64_t slots, uint64_t limit, int num_sms) {
    if (slots > limit) return 0;
    const int per = coop_per(slots);
    return (int)std::max<uint64_t>(
        1, std::min<uint64_t>((slots + per - 1) / per, 2 * (uint64_t)num_sms));
}

static int msg_grid(uint64_t work, int num_sms) {
    const uint64_t g = (work + 255) / 256;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(g, (uint64_t)num_sms * 4));
}

size_t fold_partials_bytes(size_t n) {
    (void)n;
    return (size_t)1024 * 8 * sizeof(uint64_t);  // up to 1024 CTAs
}

// CTAs of a message kernel over `slots` slots.
static int round_grid(uint64_t slots, uint64_t limit, int num_sms) {
    const int cg = coop_grid(slots, limit, num_sms);
    return cg ? cg : std::min(msg_grid(slots, num_sms), 1024);
}

int fold_grid(size_t n, int num_sms) { return round_grid(n / 4, kCoopFoldSlots, num_sms); }
int fold_posts(size_t n, int num_sms) { return msg_posts(fold_grid(n, num_sms)); }
int round_msg_posts(size_t n, int num_sms) {
    return msg_posts(round_grid(n / 2, kCoopMsgSlots, num_sms));
}

int launch_fold_and_msg(const uint4 *d_f, const uint4 *d_b, size_t n, uint4 r, uint4 *d_nf,
                        uint4 *d_nb, uint64_t *d_partials, uint64_t *d_msg_out, cudaStream_t st,
                        int num_sms, const MsgPost *post, const RGate *gate) {
    const uint64_t half = n / 2;
    const int grid = fold_grid(n, num_sms);
    MsgMailbox mb;
    if (post) mb = {post->ticket, post->words, post->seq_val, post->release};
    if (n / 4 <= kCoopFoldSlots) {
        const CoopRound a = {d_f, d_b, d_nf, d_nb, nullptr, nullptr, nullptr,
                             std::max<uint64_t>(n / 4, 1), coop_per(n / 4), r, 0, n == 2, d_partials, mb};
        if (gate)
            launch_chained(coop_round_kernel<false, true, true>, grid, kCoopThreads, 0, st, a,
                           *gate);
        else
            launch_chained(coop_round_kernel<false, true, false>, grid, kCoopThreads, 0, st, a,
                           RGate{});
    } else if (gate) {
        launch_chained(fold_and_msg_kernel<true>, grid, 256, kRTableSmem, st, d_f, d_b, half, r,
                       d_nf, d_nb, d_partials, mb, *gate);
    } else {
        launch_chained(fold_and_msg_kernel<false>, grid, 256, kRTableSmem, st, d_f, d_b, half, r,
                       d_nf, d_nb, d_partials, mb, RGate{});
    }
    if (post) return 1;
    launch_chained(finish_msg_kernel, 1, kFinishThreads, 0, st, d_partials, grid, d_msg_out);
    return 2;
}

int launch_round_msg(const uint4 *d_f, const uint4 *d_b, size_t n, uint64_t *d_partials,
                     uint64_t *d_msg_out, cudaStream_t st, int num_sms, const MsgPost *post) {
    const uint64_t pairs = n / 2;
    const int grid = round_grid(pairs, kCoopMsgSlots, num_sms);
    MsgMailbox mb;
    if (post) mb = {post->ticket, post->words, post->seq_val, post->release};
    if (pairs <= kCoopMsgSlots) {
        const CoopRound a = {d_f, d_b, nullptr, nullptr, nullptr, nullptr, nullptr, pairs,
                             coop_per(pairs), make_uint4(0, 0, 0, 0), 0, 0, d_partials, mb};
        launch_chained(coop_round_kernel<false, false, false>, grid, kCoopThreads, 0, st, a,
                       RGate{});
    } else {
        launch_chained(round_msg_kernel, grid, 256, 0, st, d_f, d_b, pairs, d_partials, mb);
    }
    if (post) return 1;
    launch_chained(finish_msg_kernel, 1, kFinishThreads, 0, st, d_partials, grid, d_msg_out);
    return 2;
}

// One partial_eval_lsb round: out[i] = in[2i] + (in[2i] + in[2i+1]) * r
// (= in[2i]*(1+r) + in[2i+1]*r exactly, ligerito.rs:1686-1691).
__global__ void __launch_bounds__(256) partial_eval_round_kernel(const uint4 *in, uint64_t half,
                                                                 uint4 r, uint4 *out) {
    chain_wait();
    extern __shared__ uint4 smem[];
    const char *T = build_r_table(smem, r);
    T16Lane8 lc;
    lc.init();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < half;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 v0 = in[2 * i], v1 = in[2 * i + 1];
        out[i] = gf_add(v0, lc.mul(T, gf_add(v0, v1)));
    }
}

int launch_partial_eval_round(const uint4 *d_in, size_t n, uint4 r, uint4 *d_out,
                              cudaStream_t st) {
    const uint64_t half = n / 2;
    const unsigned grid = (unsigned)std::min<uint64_t>((half + 255) / 256, 152 * 3);
    launch_chained(partial_eval_round_kernel, std::max(grid, 1u), 256, kRTableSmem, st, d_in,
                   half, r, d_out);
    return 1;
}

// The point of an eq table is a kernel argument: no upload and no buffer, and
// the small tables are built before chain_wait, while the previous kernel, whose
// CTAs have exited, is retired and its writes are flushed.
constexpr int kEqSplitMaxK = 22;
struct EqPoint {
    uint4 r[kEqSplitMaxK];
};

// eq table rounds: entries [0, half) double into [0, 2 half).
__global__ void eq_round_kernel(uint4 *eq, uint64_t half, uint4 r) {
    chain_wait();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < half;
         j += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 p = eq[j];
        const uint4 one = gf_mul(p, r);
        eq[half + j] = one;
        eq[j] = gf_add(p, one);
    }
}

// The first k rounds in one CTA (global writes of a round are visible to the
// CTA's threads after the barrier).
__global__ void __launch_bounds__(512) eq_small_kernel(uint4 *eq, const __grid_constant__ EqPoint point,
                                                       int k) {
    chain_wait();
    if (threadIdx.x == 0) eq[0] = make_uint4(1, 0, 0, 0);
    __syncthreads();
    for (int i = 0; i < k; ++i) {
        const uint4 r = point.r[i];
        const uint32_t half = 1u << i;
        for (uint32_t j = threadIdx.x; j < half; j += blockDim.x) {
            const uint4 p = eq[j];
            const uint4 one = gf_mul(p, r);
            eq[half + j] = one;
            eq[j] = gf_add(p, one);
        }
        __syncthreads();
    }
}

// eq over k variables in one launch, as the product of two half tables:
// eq[j] = lo[j mod 2^a] * hi[j >> a], lo over point[0..a) and hi over
// point[a..k).  Every factor of an entry is the same field element as in the
// doubling rounds (bit i of j picks r_i or 1 + r_i), so the entries are
// identical.  Each CTA builds both halves in shared memory (their rounds side
// by side), then writes its share of the products.
__global__ void __launch_bounds__(512) eq_split_kernel(uint4 *eq,
                                                       const __grid_constant__ EqPoint point,
                                                       int k, int a) {
    extern __shared__ uint4 halves[];
    const int b = k - a;
    uint4 *lo = halves, *hi = halves + ((size_t)1 << a);
    if (threadIdx.x == 0) {
        lo[0] = make_uint4(1, 0, 0, 0);
        hi[0] = make_uint4(1, 0, 0, 0);
    }
    __syncthreads();
    for (int i = 0; i < (a > b ? a : b); ++i) {
        const uint32_t nlo = i < a ? 1u << i : 0u, nhi = i < b ? 1u << i : 0u;
        for (uint32_t j = threadIdx.x; j < nlo + nhi; j += blockDim.x) {
            const bool in_lo = j < nlo;
            uint4 *t = in_lo ? lo : hi;
            const uint32_t jj = in_lo ? j : j - nlo;
            const uint4 r = point.r[in_lo ? i : a + i];
            const uint4 p = t[jj];
            const uint4 one = gf_mul(p, r);
            t[(1u << i) + jj] = one;
            t[jj] = gf_add(p, one);
        }
        __syncthreads();
    }
    chain_wait();
    const uint64_t n = (uint64_t)1 << k;
    const uint64_t mask = ((uint64_t)1 << a) - 1;
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
         j += (uint64_t)gridDim.x * blockDim.x)
        eq[j] = gf_mul(lo[j & mask], hi[j >> a]);
}

// The same entries from kEqRowsK variables on.  A CTA takes rows of 2^a entries
// with the same hi and multiplies lo by its byte tables: 2 clocks per SM a
// product instead of 7, for a build of 2048 table entries a row.  The half
// tables' rounds (a launch's latency) are split once more: lo and the CTA's
// own hi are products of quarter tables of at most 6 rounds.  2^18 entries: 24
// us against 30 us, 2^20: 34 against 56, 2^22: 67 against 142 (below, the extra
// products make it 2 to 8 us slower).
constexpr int kEqRowsK = 18;
constexpr int kEqThreads = 512;
constexpr int kEqHeadRows = 64;  // rows whose hi a CTA forms at a time
__global__ void __launch_bounds__(kEqThreads) eq_rows_kernel(uint4 *eq,
                                                             const __grid_constant__ EqPoint point,
                                                             int k, int a) {
    extern __shared__ uint4 lo[];  // 2^a, then the row's byte tables
    __shared__ uint4 quarter[4][1 << ((kEqSplitMaxK + 3) / 4)];
    __shared__ uint4 head[kEqHeadRows];
    __shared__ uint4 pt[kEqSplitMaxK];
    const int b = k - a, a0 = a / 2, b0 = b / 2;
    if (threadIdx.x < kEqSplitMaxK) pt[threadIdx.x] = point.r[threadIdx.x];
    {
        const int g = threadIdx.x >> 7, t = threadIdx.x & 127;
        const int first = g == 0 ? 0 : g == 1 ? a0 : g == 2 ? a : a + b0;
        const int nv = g == 0 ? a0 : g == 1 ? a - a0 : g == 2 ? b0 : b - b0;
        const int rounds = max(a - a0, b - b0);
        if (t == 0) quarter[g][0] = make_uint4(1, 0, 0, 0);
        __syncthreads();
        for (int i = 0; i < rounds; ++i) {
            if (i < nv && t < (1 << i)) {
                const uint4 p = quarter[g][t];
                const uint4 one = gf_mul(p, pt[first + i]);
                quarter[g][(1 << i) + t] = one;
                quarter[g][t] = gf_add(p, one);
            }
            __syncthreads();
        }
    }
    char *tbl = reinterpret_cast<char *>(lo + ((size_t)1 << a));
    T8Lane lc;
    lc.init();
    for (uint32_t j = threadIdx.x; j < (1u << a); j += kEqThreads)
        lo[j] = gf_mul(quarter[0][j & ((1u << a0) - 1)], quarter[1][j >> a0]);
    chain_wait();
    const uint32_t rows = 1u << b;
    uint32_t at = kEqHeadRows;  // rows of head[] taken
    for (uint32_t h = blockIdx.x; h < rows; h += gridDim.x, ++at) {
        if (at == kEqHeadRows) {
            __syncthreads();
            const uint64_t hh = h + (uint64_t)threadIdx.x * gridDim.x;
            if (threadIdx.x < kEqHeadRows && hh < rows)
                head[threadIdx.x] = gf_mul(quarter[2][hh & ((1u << b0) - 1)], quarter[3][hh >> b0]);
            at = 0;
        }
        __syncthreads();  // head, lo; the previous row's lookups are done
        t8_build_item<4>(tbl, head[at], threadIdx.x);
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < (1u << a); j += kEqThreads)
            eq[((uint64_t)h << a) | j] = lc.mul(tbl, lo[j]);
    }
}

constexpr size_t kEqSmallRounds = 12;

// Up to 6 variables: the doubling rounds in one CTA.  Up to 22: one split
// launch (2^12 entries: 3 to 4 us of products after 6 half-table rounds,
// against 12 rounds in one CTA; 2^20: one launch instead of nine).  Above:
// 12 rounds in one CTA, then one launch per further round.
int launch_build_eq(const uint64_t *point, size_t k, uint4 *d_out, cudaStream_t st,
                    int num_sms) {
    auto r = [&](size_t i) {
        return make_uint4((uint32_t)point[2 * i], (uint32_t)(point[2 * i] >> 32),
                          (uint32_t)point[2 * i + 1], (uint32_t)(point[2 * i + 1] >> 32));
    };
    EqPoint pt{};
    for (size_t i = 0; i < std::min(k, (size_t)kEqSplitMaxK); ++i) pt.r[i] = r(i);
    if (k > 6 && k <= (size_t)kEqSplitMaxK) {
        const int a = (int)k / 2;
        if ((int)k >= kEqRowsK) {
            const unsigned grid = std::min(1u << (k - a), 2u * (unsigned)num_sms);
            launch_chained(eq_rows_kernel, grid, kEqThreads, (sizeof(uint4) << a) + kT8Bytes, st,
                           d_out, pt, (int)k, a);
            return 1;
        }
        const size_t smem = (((size_t)1 << a) + ((size_t)1 << (k - a))) * sizeof(uint4);
        const uint64_t n = (uint64_t)1 << k;
        const unsigned grid = (unsigned)std::max<uint64_t>(
            1, std::min<uint64_t>((n + 511) / 512, (uint64_t)2 * num_sms));
        launch_chained(eq_split_kernel, grid, 512, smem, st, d_out, pt, (int)k, a);
        return 1;
    }
    const size_t k0 = std::min(k, kEqSmallRounds);
    launch_chained(eq_small_kernel, 1, 512, 0, st, d_out, pt, (int)k0);
    for (size_t i = k0; i < k; ++i) {
        const uint64_t half = (uint64_t)1 << i;
        const unsigned grid = (unsigned)std::min<uint64_t>((half + 255) / 256, 8192);
        launch_chained(eq_round_kernel, std::max(grid, 1u), 256, 0, st, d_out, half, r(i));
    }
    return (int)(k - k0) + 1;
}

// sv[j] = sum_y eq[y] * bit_j(P[y]) (src/ligerito.rs:317-375).  128 threads
// per CTA, one per output bit j, over tiles of 128 y.  Warp w transposes the
// 32 P words of its y by shuffles, so thread j has bit j of 32 words in one
// register and takes four of them as an index into the 16 subset sums of
// their eq entries.  The sums of the 8 groups of 4 of a warp's y stand side by
// side (row x: subset x of each group), and thread j walks the groups in an
// order rotated by j mod 8, so a quarter-warp's lookups fall in 8 bank groups
// as those of the byte tables do: 4 clocks per SM and y, against 17 for lookups
// of one group by every thread.  A CTA runs four such tiles side by side and
// stores its sums; a CTA per output adds them (2^20 words: 80 us before).
constexpr int kSvTile = 128;
// Block swaps of halving size (Warren, Hacker's Delight, 7-3), a row a lane.
__device__ __forceinline__ uint32_t transpose32(uint32_t x) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        const uint32_t m = j == 16 ? 0x0000FFFFu : j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu
                         : j == 2 ? 0x33333333u : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
        x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
    }
    return x;
}

constexpr int kSvGroups = 4;  // groups of 128 threads, each with a tile of its own
__global__ void __launch_bounds__(kSvTile *kSvGroups, 2) sv_fold_kernel(const uint4 *packed,
                                                                         const uint4 *eq,
                                                                         uint64_t n,
                                                                         uint4 *partials) {
    chain_wait();
    __shared__ uint32_t bits[kSvGroups][4][128];
    __shared__ uint4 sub[kSvGroups][4][16][8];
    const int grp = threadIdx.x >> 7, t = threadIdx.x & 127, w = t >> 5, r = t & 7;
    auto sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(kSvTile) : "memory"); };
    uint4 acc = make_uint4(0, 0, 0, 0);
    for (uint64_t base = ((uint64_t)blockIdx.x * kSvGroups + grp) * kSvTile; base < n;
         base += (uint64_t)gridDim.x * kSvGroups * kSvTile) {
        const uint64_t y = base + t;
        const uint4 p = y < n ? packed[y] : make_uint4(0, 0, 0, 0);
        // thread (w, q, g) sums subsets 4q .. 4q + 3 of group g of warp w's y
        const int g = t & 7, q = (t >> 3) & 3;
        uint4 e[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t ye = base + 32 * w + 4 * g + k;
            e[k] = ye < n ? eq[ye] : make_uint4(0, 0, 0, 0);
        }
        sync();  // the previous tile's lookups are done
        bits[grp][w][t & 31] = transpose32(p.x);
        bits[grp][w][32 + (t & 31)] = transpose32(p.y);
        bits[grp][w][64 + (t & 31)] = transpose32(p.z);
        bits[grp][w][96 + (t & 31)] = transpose32(p.w);
        uint4 H = make_uint4(0, 0, 0, 0);
        if (q & 1) H = gf_add(H, e[2]);
        if (q & 2) H = gf_add(H, e[3]);
        sub[grp][w][4 * q][g] = H;
        sub[grp][w][4 * q + 1][g] = gf_add(H, e[0]);
        sub[grp][w][4 * q + 2][g] = gf_add(H, e[1]);
        sub[grp][w][4 * q + 3][g] = gf_add(gf_add(H, e[0]), e[1]);
        sync();
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t b = bits[grp][s][t];
            const uint32_t x = __funnelshift_r(b, b, 4 * r);  // nibble m: group (m + r) mod 8
#pragma unroll
            for (int m = 0; m < 8; ++m)
                acc = gf_add(acc, sub[grp][s][(x >> (4 * m)) & 15][(m + r) & 7]);
        }
    }
    __syncthreads();
    uint4 *red = &sub[0][0][0][0];
    red[threadIdx.x] = acc;
    __syncthreads();
    if (grp == 0) {
#pragma unroll
        for (int k = 1; k < kSvGroups; ++k) acc = gf_add(acc, red[k * kSvTile + t]);
        partials[(uint64_t)blockIdx.x * 128 + t] = acc;
    }
}

// CTA j XORs output j of every partial and posts it.
__global__ void __launch_bounds__(128) sv_finish_kernel(const uint4 *partials, int n_ctas,
                                                        ElementPost post) {
    __shared__ uint4 red[4];
    chain_wait();
    uint4 acc = make_uint4(0, 0, 0, 0);
    for (int c = threadIdx.x; c < n_ctas; c += 128)
        acc = gf_add(acc, partials[(uint64_t)c * 128 + blockIdx.x]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc.x ^= __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y ^= __shfl_xor_sync(0xffffffffu, acc.y, o);
        acc.z ^= __shfl_xor_sync(0xffffffffu, acc.z, o);
        acc.w ^= __shfl_xor_sync(0xffffffffu, acc.w, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0)
        post_element(post.words + 4 * blockIdx.x, post.seq,
                     gf_add(gf_add(red[0], red[1]), gf_add(red[2], red[3])));
}

size_t sv_partials_bytes(int num_sms) { return (size_t)num_sms * 2 * 128 * sizeof(uint4); }

int launch_sv_fold(const uint4 *d_packed, const uint4 *d_eq, size_t n, uint4 *d_partials,
                   const ElementPost &post, cudaStream_t st, int num_sms) {
    const uint64_t tiles = (n + kSvTile - 1) / kSvTile;
    const int grid = (int)std::max<uint64_t>(
        1, std::min<uint64_t>((tiles + kSvGroups - 1) / kSvGroups, (uint64_t)num_sms * 2));
    launch_chained(sv_fold_kernel, grid, kSvTile * kSvGroups, 0, st, d_packed, d_eq, n,
                   d_partials);
    launch_chained(sv_finish_kernel, 128, 128, 0, st, d_partials, grid, post);
    return 2;
}

// n elements of device memory to the mailbox.
__global__ void post_elements_kernel(const uint4 *in, int n, ElementPost post) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) post_element(post.words + 4 * i, post.seq, in[i]);
}

int launch_post_elements(const uint4 *d_in, int n, const ElementPost &post, cudaStream_t st) {
    launch_chained(post_elements_kernel, (unsigned)(n + 127) / 128, 128, 0, st, d_in, n, post);
    return 1;
}

// phi_from_words with phi_byte_tables (src/ligerito.rs:384-427): phi(y) =
// sum over the set bits u of eq_hi[y] of eq_r2[u], a GF(2)-linear map of
// eq_hi[y] whose image of bit u is eq_r2[u].  So it is a byte-table multiply:
// the tables are expanded from those 128 images in the bank-conflict-free
// layout of the NTT's and the folds' tables, and each word is one 16-lookup
// table multiply.
__global__ void __launch_bounds__(256) phi_kernel(const uint4 *eq_hi, uint64_t n,
                                                  const uint4 *eq_r2, uint4 *out) {
    chain_wait();
    extern __shared__ uint4 smem[];
    uint4 *bases = smem + kT16Entries;
    for (int e = threadIdx.x; e < 128; e += blockDim.x)
        bases[(e >> 3) * 9 + (e & 7)] = eq_r2[e];
    __syncthreads();
    t16_expand(smem, bases, 1);
    const char *T = reinterpret_cast<const char *>(smem);
    T16Lane8 lc;
    lc.init();
    for (uint64_t y = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; y < n;
         y += (uint64_t)gridDim.x * blockDim.x)
        out[y] = lc.mul(T, eq_hi[y]);
}

void init_gkr_kernels();

void init_fold_kernels() {
    init_gkr_kernels();
    cudaFuncSetAttribute(phi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kRTableSmem);
    cudaFuncSetAttribute(eq_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(uint4) << (kEqSplitMaxK / 2)) + kT8Bytes);
    cudaFuncSetAttribute(fold_and_msg_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kRTableSmem);
    cudaFuncSetAttribute(fold_and_msg_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kRTableSmem);
    cudaFuncSetAttribute(partial_eval_round_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kRTableSmem);
}

// Two CTAs per SM at most: every CTA builds the 64 KB of tables first, so a
// grid-stride loop over fewer CTAs builds them fewer times.
int launch_phi(const uint4 *d_eq_hi, size_t n, const uint4 *d_eq_r2, uint4 *d_out,
               cudaStream_t st, int num_sms) {
    const unsigned grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((n + 255) / 256, (uint64_t)2 * num_sms));
    launch_chained(phi_kernel, grid, 256, kRTableSmem, st, d_eq_hi, n, d_eq_r2, d_out);
    return 1;
}

// ---------------------------------------------------------------------------
// ChaCha20 (RFC 8439 section 2.3): one 64-byte block per thread = 4 words.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rotl(uint32_t x, int n) { return __funnelshift_l(x, x, n); }
#define BZ_QR(a, b, c, d)                                 \
    do {                                                  \
        x[a] += x[b]; x[d] = rotl(x[d] ^ x[a], 16);       \
        x[c] += x[d]; x[b] = rotl(x[b] ^ x[c], 12);       \
        x[a] += x[b]; x[d] = rotl(x[d] ^ x[a], 8);        \
        x[c] += x[d]; x[b] = rotl(x[b] ^ x[c], 7);        \
    } while (0)

__global__ void chacha_kernel(uint32_t k0, uint32_t k1, uint64_t first_word, uint4 *out,
                              uint64_t n_words) {
    const uint64_t first_blk = first_word >> 2;
    const uint64_t last_blk = (first_word + n_words - 1) >> 2;
    for (uint64_t blk = first_blk + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
         blk <= last_blk; blk += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t st[16] = {0x61707865u, 0x3320646eu, 0x79622d32u, 0x6b206574u, k0, k1, 0, 0,
                           0, 0, 0, 0, (uint32_t)blk, 0, 0, 0};
        uint32_t x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = st[i];
#pragma unroll
        for (int i = 0; i < 10; ++i) {
            BZ_QR(0, 4, 8, 12); BZ_QR(1, 5, 9, 13); BZ_QR(2, 6, 10, 14); BZ_QR(3, 7, 11, 15);
            BZ_QR(0, 5, 10, 15); BZ_QR(1, 6, 11, 12); BZ_QR(2, 7, 8, 13); BZ_QR(3, 4, 9, 14);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] += st[i];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint64_t w = blk * 4 + q;
            if (w >= first_word && w < first_word + n_words)
                out[w - first_word] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
        }
    }
}

int launch_chacha(uint64_t seed, uint64_t first_word, uint4 *d_out, size_t n_words,
                  cudaStream_t st) {
    if (n_words == 0) return 0;
    const uint64_t blocks = ((first_word + n_words - 1) >> 2) - (first_word >> 2) + 1;
    const unsigned grid = (unsigned)std::min<uint64_t>((blocks + 255) / 256, 8192);
    chacha_kernel<<<grid, 256, 0, st>>>((uint32_t)seed, (uint32_t)(seed >> 32), first_word, d_out,
                                        n_words);
    return 1;
}

// ---------------------------------------------------------------------------
// Batched grand-product GKR (BitZ src/bitz/gkr.rs), the dense rounds.
// ---------------------------------------------------------------------------
// One product layer: out[i] = in[i] * in[half + i] (GrandProductCircuit::
// batched_eval, gkr.rs:93-108: the top index bit pairs the factors).
__global__ void __launch_bounds__(256) gkr_product_kernel(const uint4 *in, uint64_t half,
                                                          uint4 *out) {
    chain_wait();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < half;
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = gf_mul(in[i], in[half + i]);
}

// One dense round over h slots (prove_dense_rounds, gkr.rs:188-282, with the
// column-free weights): the tables l and r (the layer's two halves) hold the
// round's lo entries at [0, h) and hi entries at [h, 2h).  With FOLD the
// previous round's challenge rho is applied first, in place: entries q0..q3
// at c, h + c, 2h + c, 3h + c become q0 + rho (q2 - q0) at c and
// q1 + rho (q3 - q1) at h + c (kernels.rs:146-186, 312-348).  Each CTA
// stores its partial sums of w_c l_end r_end and w_c (l_hi - l_lo)(r_hi -
// r_lo) (kernels.rs:248-262; l_end = l_hi when send_one), unreduced; the
// finish kernel reduces them.  With w_next, the next round's weights
// w_next[c] = w[c] + w[c + h/2] (eq over one coordinate fewer: the two
// values of the dropped coordinate's factor sum to 1) are written too.
template <bool FOLD>
__global__ void __launch_bounds__(256, 2) gkr_round_kernel(uint4 *l, uint4 *r, const uint4 *w,
                                                           uint64_t h, uint4 rho, int send_one,
                                                           uint64_t *partials, MsgMailbox mb,
                                                           uint4 *w_next) {
    chain_wait();
    extern __shared__ uint4 smem[];
    const char *T = nullptr;
    T16Lane8 lc;
    if constexpr (FOLD) {
        T = build_r_table(smem, rho);
        lc.init();
    }
    gf_wide e = gf_wide_zero(), f = gf_wide_zero();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < h; c += stride) {
        uint4 l0, l1, r0, r1;
        if constexpr (FOLD) {
            const uint4 a0 = l[c], a1 = l[h + c], a2 = l[2 * h + c], a3 = l[3 * h + c];
            const uint4 b0 = r[c], b1 = r[h + c], b2 = r[2 * h + c], b3 = r[3 * h + c];
            l0 = gf_add(a0, lc.mul(T, gf_add(a2, a0)));
            l1 = gf_add(a1, lc.mul(T, gf_add(a3, a1)));
            r0 = gf_add(b0, lc.mul(T, gf_add(b2, b0)));
            r1 = gf_add(b1, lc.mul(T, gf_add(b3, b1)));
            l[c] = l0;
            l[h + c] = l1;
            r[c] = r0;
            r[h + c] = r1;
        } else {
            l0 = l[c];
            l1 = l[h + c];
            r0 = r[c];
            r1 = r[h + c];
        }
        const uint4 wc = w[c];
        if (w_next && c < h / 2) w_next[c] = gf_add(wc, w[c + h / 2]);
        const uint4 le = send_one ? l1 : l0, re = send_one ? r1 : r0;
        gf_wide_xor(e, gf_mul_wide(gf_mul(wc, le), re));
        gf_wide_xor(f, gf_mul_wide(gf_mul(wc, gf_add(l1, l0)), gf_add(r1, r0)));
    }
    msg_finish_call<false>(e, f, partials, mb);
}

// The leaf grid of the BitZ forest (src/bitz/forest_tests.rs:42-68): leaf
// row * 2^s + column is images[row] when bit (column mod 64) of
// packed[(column / 64) * 2^t + row] is set, else 1.
__global__ void __launch_bounds__(256) gkr_forest_leaves_kernel(const uint64_t *packed,
                                                                const uint4 *images, int t,
                                                                int s, uint4 *out) {
    chain_wait();
    const uint64_t n = (uint64_t)1 << (t + s), rows = (uint64_t)1 << t;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t row = i >> s, col = i & (((uint64_t)1 << s) - 1);
        const uint64_t bit = (packed[(col >> 6) * rows + row] >> (col & 63)) & 1;
        out[i] = bit ? images[row] : make_uint4(1, 0, 0, 0);
    }
}

int launch_gkr_product(const uint4 *d_in, size_t half, uint4 *d_out, cudaStream_t st,
                       int num_sms) {
    const unsigned grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((half + 255) / 256, (uint64_t)num_sms * 8));
    launch_chained(gkr_product_kernel, grid, 256, 0, st, d_in, half, d_out);
    return 1;
}

bool gkr_small_round(size_t h) { return h <= kCoopGkrSlots; }

static int gkr_round_grid(size_t h, int num_sms) { return round_grid(h, kCoopGkrSlots, num_sms); }

int gkr_round_posts(size_t h, int num_sms) { return msg_posts(gkr_round_grid(h, num_sms)); }

int launch_gkr_round(uint4 *d_l, uint4 *d_r, uint4 *d_nl, uint4 *d_nr, const uint4 *d_w, size_t h,
                     bool fold, uint4 rho, bool send_one, uint4 *d_w_next, uint64_t *d_partials,
                     cudaStream_t st, int num_sms, const MsgPost &post, uint64_t *d_tail,
                     const RGate *gate) {
    const MsgMailbox mb = {post.ticket, post.words, post.seq_val, post.release};
    const int grid = gkr_round_grid(h, num_sms);
    if (gkr_small_round(h)) {
        const CoopRound a = {d_l, d_r, d_nl, d_nr, d_w, d_w_next, h == 1 ? d_tail : nullptr, h,
                             coop_per(h), rho, send_one, 0, d_partials, mb};
        if (gate)
            launch_chained(coop_round_kernel<true, true, true>, grid, kCoopThreads, 0, st, a, *gate);
        else if (fold)
            launch_chained(coop_round_kernel<true, true, false>, grid, kCoopThreads, 0, st, a,
                           RGate{});
        else
            launch_chained(coop_round_kernel<true, false, false>, grid, kCoopThreads, 0, st, a,
                           RGate{});
        return 1;
    }
    if (fold)
        launch_chained(gkr_round_kernel<true>, grid, 256, kRTableSmem, st, d_l, d_r, d_w, h, rho,
                       send_one, d_partials, mb, d_w_next);
    else
        launch_chained(gkr_round_kernel<false>, grid, 256, 0, st, d_l, d_r, d_w, h, rho, send_one,
                       d_partials, mb, d_w_next);
    return 1;
}

void init_gkr_kernels() {
    cudaFuncSetAttribute(gkr_round_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kRTableSmem);
}

int launch_gkr_forest_leaves(const uint64_t *d_packed, const uint4 *d_images, int t, int s,
                             uint4 *d_out, cudaStream_t st, int num_sms) {
    const uint64_t n = (uint64_t)1 << (t + s);
    const unsigned grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((n + 255) / 256, (uint64_t)num_sms * 8));
    launch_chained(gkr_forest_leaves_kernel, grid, 256, 0, st, d_packed, d_images, t, s, d_out);
    return 1;
}

}  // namespace bz
