// Host paths that a GPU cannot be made to take at will, over the fake runtime:
// `host_paths CASE` prints what the case found and exits with 0 when it held.
#include <cstdio>
#include <cstring>
#include <vector>

#include "fake_cudart.h"
#include "runtime.h"

#define CHECK(x)                                                    \
    do {                                                            \
        if (!(x)) {                                                 \
            printf("%s:%d: %s\n", __FILE__, __LINE__, #x);          \
            return 1;                                               \
        }                                                           \
    } while (0)

namespace {

bz_ctx *ctx;
const bz_params kSmall = {8, 1, 3, BZ_HASH_BLAKE3};

// A commit whose kernels post nothing: its root is what the tree's memory
// holds, 0xA5 in every byte.
int commit_root_is_the_trees() {
    std::vector<uint64_t> msg(2 << 8);
    bz_commitment *c = nullptr;
    uint8_t root[32] = {0};
    CHECK(bz_commit(ctx, msg.data(), 1 << 8, &kSmall, &c, root) == BZ_OK);
    for (int i = 0; i < 32; ++i) CHECK(root[i] == 0xA5);
    CHECK(bz_commitment_root(c, root) == BZ_OK && root[0] == 0xA5);
    CHECK(bz_commitment_free(c) == BZ_OK);
    return 0;
}

// The stream goes idle and the mailbox has no root.
int root_not_posted() { return commit_root_is_the_trees(); }

// Commits of other threads took the slot before the owner read it: every word
// of the 16 slots carries a later number.
int root_slot_reused() {
    int queries = 0;
    fake::query = [&] {
        uint64_t *w = (uint64_t *)((uint8_t *)ctx->h_mbox + 1024);
        for (int i = 0; i < 16 * 16; ++i) w[i] = (uint64_t)(ctx->root_seq + 16) << 32;
        return ++queries < 100 ? cudaErrorNotReady : cudaSuccess;
    };
    return commit_root_is_the_trees();
}

// The work queued before the commit takes longer than a spinning wait allows.
int root_slow() {
    bool done = false;
    fake::query = [&] {
        fake::clock_skew_s += 61;
        return done ? cudaSuccess : cudaErrorNotReady;
    };
    fake::sync = [&] {
        done = true;
        return cudaSuccess;
    };
    return commit_root_is_the_trees();
}

// A failed stream still fails the commit.
int root_stream_error() {
    fake::query = [] { return cudaErrorLaunchFailure; };
    fake::sync = [] { return cudaErrorLaunchFailure; };
    std::vector<uint64_t> msg(2 << 8);
    bz_commitment *c = nullptr;
    uint8_t root[32];
    CHECK(bz_commit(ctx, msg.data(), 1 << 8, &kSmall, &c, root) == BZ_ERR_CUDA);
    CHECK(!c);
    return 0;
}

// Posted elements behind work that outlasts the spin: the partial evaluations
// come when the stream is synchronised.
int elements_slow() {
    bool done = false;
    fake::query = [&] {
        fake::clock_skew_s += 61;
        return done ? cudaSuccess : cudaErrorNotReady;
    };
    fake::sync = [&] {
        uint64_t *w = (uint64_t *)((uint8_t *)ctx->h_mbox + 4096);
        for (int i = 0; i < 4 * 128; ++i) w[i] = (uint64_t)ctx->mbox_seq << 32 | i;
        done = true;
        return cudaSuccess;
    };
    std::vector<uint64_t> d(2 << 8), sv(256);
    CHECK(bz_sv_fold(ctx, d.data(), d.data(), 1 << 8, sv.data()) == BZ_OK);
    for (uint64_t i = 0; i < 256; ++i) CHECK(sv[i] == ((2 * i) | (2 * i + 1) << 32));
    return 0;
}

// A stream that goes idle, or fails, without the post is an error.
int elements_not_posted() {
    std::vector<uint64_t> d(2 << 8), sv(256);
    CHECK(bz_sv_fold(ctx, d.data(), d.data(), 1 << 8, sv.data()) == BZ_ERR_CUDA);
    fake::query = [] {
        fake::clock_skew_s += 61;
        return cudaErrorNotReady;
    };
    fake::sync = [] { return cudaErrorLaunchFailure; };
    CHECK(bz_sv_fold(ctx, d.data(), d.data(), 1 << 8, sv.data()) == BZ_ERR_CUDA);
    return 0;
}

// Openings through device buffers (the mapped one is held): a refused launch and
// each copy that fails are errors, not rows that were never gathered.
int opening_errors() {
    std::vector<uint64_t> msg(2 << 8);
    bz_commitment *c = nullptr;
    uint8_t root[32];
    CHECK(bz_commit(ctx, msg.data(), 1 << 8, &kSmall, &c, root) == BZ_OK);
    const std::vector<uint64_t> pos = {1, 5, 9};
    std::vector<uint64_t> rows(3 * 8 * 2);
    std::vector<uint8_t> nodes(32 * 64);
    size_t n = 0;
    auto open_rows = [&] { return bz_commitment_rows(c, pos.data(), 3, rows.data()); };
    auto open_nodes = [&] {
        return bz_commitment_multiproof(c, pos.data(), 3, nodes.data(), 64, &n);
    };
    std::lock_guard<std::mutex> held(ctx->open_mu);
    CHECK(open_rows() == BZ_OK && open_nodes() == BZ_OK);
    fake::launch = [] { return cudaErrorInvalidConfiguration; };
    CHECK(open_rows() == BZ_ERR_CUDA && open_nodes() == BZ_ERR_CUDA);
    fake::launch = nullptr;
    for (int bad = 0; bad < 2; ++bad) {  // the indices up, the results down
        int at = 0;
        fake::copy = [&] { return at++ == bad ? cudaErrorInvalidValue : cudaSuccess; };
        CHECK(open_rows() == BZ_ERR_CUDA);
        at = 0;
        CHECK(open_nodes() == BZ_ERR_CUDA);
    }
    fake::copy = nullptr;
    CHECK(open_rows() == BZ_OK && open_nodes() == BZ_OK);
    return 0;
}

// A profile runs the launches of the commit that a caller waits for.
int profile_is_the_commit() {
    const bz_params shapes[] = {kSmall, {12, 1, 1, BZ_HASH_BLAKE3}, {16, 1, 6, BZ_HASH_BLAKE3},
                                {14, 2, 7, BZ_HASH_BLAKE3}, {14, 1, 2, BZ_HASH_SHA256}};
    for (const bz_params &p : shapes) {
        const size_t n = (size_t)1 << p.log_msg_len;
        std::vector<uint64_t> msg(2 * n);
        bz_commitment *c = nullptr;
        uint8_t root[32];
        uint64_t before = bz_kernel_launches(ctx);
        CHECK(bz_commit_device(ctx, msg.data(), n, &p, &c, root) == BZ_OK);
        const uint64_t launches = bz_kernel_launches(ctx) - before;
        size_t count = 0;
        before = bz_kernel_launches(ctx);
        CHECK(bz_commit_profile(ctx, msg.data(), n, &p, 0, nullptr, nullptr, &count, root) == BZ_OK);
        CHECK(count == launches && bz_kernel_launches(ctx) - before == launches);
        CHECK(bz_commitment_free(c) == BZ_OK);
    }
    return 0;
}

const struct {
    const char *name;
    int (*run)();
} kCases[] = {
    {"root_not_posted", root_not_posted},
    {"root_slot_reused", root_slot_reused},
    {"root_slow", root_slow},
    {"root_stream_error", root_stream_error},
    {"elements_slow", elements_slow},
    {"elements_not_posted", elements_not_posted},
    {"opening_errors", opening_errors},
    {"profile_is_the_commit", profile_is_the_commit},
};

}  // namespace

int main(int argc, char **argv) {
    if (bz_ctx_create(0, 0, &ctx) != BZ_OK) return 2;
    for (const auto &c : kCases)
        if (argc == 2 && !strcmp(argv[1], c.name)) return c.run();
    for (const auto &c : kCases) printf("%s\n", c.name);
    return argc == 1 ? 0 : 2;
}
