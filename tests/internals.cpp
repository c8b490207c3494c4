// What the library's host code decides, printed for tests/test_internals.py (built
// there against libsaqg.so).  Without a GPU: `estimate`, `candidates`, `tiles`; with one: `presize`, `chunks`.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "saqg_internal.h"

using namespace saqg;

// Bytes that admission counts for a batch over clusters of `blocks` blocks each.
static void estimate(int S, int64_t blocks, int64_t nq, int64_t k, int64_t np) {
    Index I;
    I.D = 64 * S;
    I.K = 512;
    for (int s = 0; s < S; ++s) {
        Index::SegHost h{};
        h.dim = 64;
        h.bits = 4;
        I.segs.push_back(h);
        I.view.seg[s].dim = 64;
        I.view.seg[s].bits = 4;
    }
    for (int64_t c = 0; c <= I.K; ++c) I.blk_off.push_back(c * blocks);
    finalize_view(I);
    std::printf("%zu\n", search_bytes_estimate(I, nq, k, np));
}

static int presize(const char *path) {
    Index *I = load_index_file(path);
    {
        SearchCtx c;
        presize_tc_ctx(*I, c, 64, 10, 4, 40, 100000);
        std::printf("%d %d %d %d %d %d\n", c.aux != nullptr, c.low != nullptr, c.ev_fork != nullptr,
                    c.ev_join != nullptr, c.ev_qfork != nullptr, c.ev_qjoin != nullptr);
    }
    delete I;
    return 0;
}

int main(int argc, char **argv) {
    const char *what = argc > 1 ? argv[1] : "";
    if (!std::strcmp(what, "estimate") && argc == 7) {
        estimate(std::atoi(argv[2]), std::atoll(argv[3]), std::atoll(argv[4]), std::atoll(argv[5]), std::atoll(argv[6]));
        return 0;
    }
    if (!std::strcmp(what, "candidates")) {
        for (const ScanTune &t : exact_candidates(10))
            std::printf("%d %d %d %d\n", t.mode, t.defer_blocks, t.first_blocks, t.spec_levels);
        return 0;
    }
    if (!std::strcmp(what, "tiles")) {
        for (int mode : {0, 1})
            for (int64_t nq : {1, 16, 17, 4096}) std::printf("%d %d %d\n", mode, (int)nq, spec_tile_blocks(mode, nq));
        return 0;
    }
    if (!std::strcmp(what, "chunks") && argc == 4) {
        const int64_t n = std::atoll(argv[2]), maxd = std::atoll(argv[3]);
        for (int bits = 0; bits <= kMaxBits; ++bits)
            std::printf("%d %lld %lld\n", bits, (long long)encode_chunk(n, bits, maxd), (long long)encoder_vectors(bits));
        return 0;
    }
    if (!std::strcmp(what, "presize") && argc == 3) return presize(argv[2]);
    return 2;
}
