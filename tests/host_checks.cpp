// Checks of the library's host code on the CPU: csrc/slm.cpp, over the fake runtime of
// fake_cuda.h. Each check is a function of its own; `host_checks NAME` runs one
// (tests/test_host_checks.py builds this file and runs them all).
#include "fake_cuda.h"

#include "slm.cpp"

#define REQUIRE(x)                                                                                    \
    do {                                                                                              \
        if (!(x)) return std::printf("%s:%d: %s (last error: %s)\n", __FILE__, __LINE__, #x, slm_last_error()), 1; \
    } while (0)

// Scratch of slm_build_tracks_drop when pairs name the same matches: every pair's
// matches are edges of their own.
int tracks_that_share_matches() {
    slm_ctx *c = nullptr;
    REQUIRE(slm_ctx_create(nullptr, &c) == SLM_OK);
    const uint32_t images = 64, features = 1000, np = images / 2;
    std::vector<uint32_t> nf(images, features);
    std::vector<slm_pair> m(features);
    for (uint32_t k = 0; k < features; ++k) m[k] = slm_pair{k, k};
    std::vector<slm_pair_matches> pairs(np);
    for (uint32_t p = 0; p < np; ++p) pairs[p] = slm_pair_matches{2 * p, 2 * p + 1, 0, features};
    uint64_t nt = 0, no = 0;
    REQUIRE(slm_build_tracks_drop(c, nf.data(), images, pairs.data(), np, m.data(), 2, 100, nullptr, 0, nullptr, 0, &nt, &no,
                                  nullptr) == SLM_OK);
    const slm::TrackArgs &a = fake::tracks;
    const uint64_t edges = uint64_t(np) * features, linked = 2 * edges;  // all distinct, no node shared
    auto room = [](const void *from, const void *to) { return uint64_t(static_cast<const char *>(to) - static_cast<const char *>(from)); };
    REQUIRE(a.table_mask + 1 >= edges);
    REQUIRE(8 * (a.table_mask + 1) >= 8 * linked);  // `sorted` lies over the table
    REQUIRE(room(a.members, a.comps) >= 4 * linked);
    REQUIRE(a.max_comps >= edges);
    REQUIRE(room(a.comps, a.sums) >= 8 * edges);
    REQUIRE(room(a.track_off, a.obs) >= 8 * (edges + 1));
    slm_ctx_destroy(c);
    return 0;
}

// What a call's kernels may read in the caller's memory must be read when it returns,
// also when a later step fails.
size_t last(const char *what) {
    for (size_t k = fake::log.size(); k; --k)
        if (fake::log[k - 1] == what) return k;
    return 0;
}

int sampson_waits_after_a_failure() {
    slm_ctx *c = nullptr;
    REQUIRE(slm_ctx_create(nullptr, &c) == SLM_OK);
    std::vector<double> pts(4 * 10, 0.5), E(9 * 3, 0.25), th(1, 0.1);
    const uint64_t off[2] = {0, 10}, mo[3] = {0, ~0ull, 1};
    const uint32_t hp[3] = {0, 0, 0};
    uint32_t counts[3], masks[2];
    for (int nth = 1; nth <= 2; ++nth) {  // the counts' copy back, then the masks'
        fake::log.clear();
        fake::fail_d2h = nth;
        REQUIRE(slm_sampson_score(c, pts.data(), off, 1, th.data(), E.data(), hp, 3, counts, mo, masks, 2) == SLM_CUDA_ERROR);
        REQUIRE(fake::sampson.E == E.data());  // read where it lies
        REQUIRE(last("sampson") && last("copy failed") > last("sampson"));
        REQUIRE(last("sync") > last("copy failed"));
    }
    REQUIRE(slm_sampson_score(c, pts.data(), off, 1, th.data(), E.data(), hp, 3, counts, mo, masks, 2) == SLM_OK);
    slm_ctx_destroy(c);
    return 0;
}

int single_pair_waits_after_a_failure() {
    slm_ctx *c = nullptr;
    REQUIRE(slm_ctx_create(nullptr, &c) == SLM_OK);
    void *a = nullptr;
    REQUIRE(posix_memalign(&a, 16, 512 * 300) == 0);  // read where it lies
    std::memset(a, 0, 512 * 300);
    std::vector<slm_pair> out(300);
    uint32_t n = 0;
    for (const slm_precision prec : {SLM_PREC_BF16, SLM_PREC_FP8})
        for (int nth = 1; nth <= 2; ++nth) {
            fake::log.clear();
            fake::fail_d2h = nth;
            REQUIRE(slm_ratio_match(c, static_cast<float *>(a), 300, static_cast<float *>(a), 300, 0.8f, 1, prec, out.data(), 300, &n,
                                    nullptr) == SLM_CUDA_ERROR);
            REQUIRE(last("gather rows") && last("copy failed") > last("gather rows"));
            REQUIRE(last("sync") > last("copy failed"));
        }
    // the same by way of the coalescer
    REQUIRE(slm_ctx_set_coalescing(c, 0, 4) == SLM_OK);
    fake::log.clear();
    fake::fail_d2h = 1;
    REQUIRE(slm_ratio_match(c, static_cast<float *>(a), 300, static_cast<float *>(a), 300, 0.8f, 1, SLM_PREC_AUTO, out.data(), 300, &n,
                            nullptr) == SLM_CUDA_ERROR);
    REQUIRE(last("gather rows") && last("sync") > last("copy failed"));
    REQUIRE(slm_ctx_set_coalescing(c, 0, 0) == SLM_OK);
    // and describe, whose image and keypoints are read by copies
    const slm_keypoint kp{5, 5, 2, 0, 0};
    std::vector<float> desc(128);
    fake::log.clear();
    fake::fail_d2h = 1;
    REQUIRE(slm_describe(c, static_cast<float *>(a), 20, 20, &kp, 1, desc.data()) == SLM_CUDA_ERROR);
    REQUIRE(last("sync") > last("copy failed"));
    slm_ctx_destroy(c);
    std::free(a);
    return 0;
}

// Device memory of a detection call: the layers of an octave at a time, every octave's
// gradient tables, the candidates and the images, with the buffers' slack of a quarter,
// whatever parts the batch goes in.
uint64_t detection_bytes(uint64_t n, uint64_t w, uint64_t h) {
    const uint64_t s = 3, ng = s + 3, wh0 = w * h, wh1 = (w / 2) * (h / 2);
    uint64_t grads = 0;
    for (int o = 0; o < 4; ++o) grads += 8 * s * (w >> o) * (h >> o);
    const uint64_t image = 4 * (ng * wh0 + (ng - 1) * wh0 + wh0 + wh1) + grads + 16384 * (sizeof(slm::FeatCand) + 4 * slm::kMaxAngles + 1) + 7 * wh0;
    return (n * image + (64 << 10)) * 5 / 4;
}

int detect(slm_ctx *c, uint32_t n, uint32_t w, uint32_t h) {
    slm_detector_config cfg;
    slm_detector_config_default(&cfg);
    std::vector<uint8_t> img(size_t(3) * n * w * h);
    std::vector<uint64_t> off(n + 1);
    return slm_detect_and_describe_rgb8(c, img.data(), n, w, h, &cfg, nullptr, nullptr, 0, off.data());
}

int detection_within_its_budget() {
    for (const uint32_t n : {1u, 3u, 4u, 8u, 15u, 24u, 31u}) {
        slm_opts o{};
        o.hbm_budget = detection_bytes(n, 960, 540);
        slm_ctx *c = nullptr;
        REQUIRE(slm_ctx_create(&o, &c) == SLM_OK);
        REQUIRE(detect(c, n, 960, 540) == SLM_OK);
        slm_ctx_destroy(c);
        REQUIRE(fake::device_bytes == 0);
    }
    return 0;
}

// A batch leaves its workspaces with memory; a later call of another shape may need it.
int idle_workspaces_give_memory_back() {
    slm_opts o{};
    o.hbm_budget = detection_bytes(24, 960, 540) * 13 / 10;
    slm_ctx *c = nullptr;
    REQUIRE(slm_ctx_create(&o, &c) == SLM_OK);
    for (int k = 0; k < 2; ++k) {
        REQUIRE(detect(c, 24, 960, 540) == SLM_OK);
        REQUIRE(detect(c, 1, 4500, 2700) == SLM_OK);  // as many pixels in one image
    }
    void *a = nullptr;  // and a pair of another kind
    REQUIRE(posix_memalign(&a, 16, 512 * 300) == 0);
    std::memset(a, 0, 512 * 300);
    std::vector<slm_pair> out(300);
    uint32_t n = 0;
    REQUIRE(slm_ratio_match(c, static_cast<float *>(a), 300, static_cast<float *>(a), 300, 0.8f, 1, SLM_PREC_BF16, out.data(), 300, &n,
                            nullptr) == SLM_OK);
    REQUIRE(detect(c, 24, 960, 540) == SLM_OK);
    REQUIRE(detect(c, 60, 960, 540) == SLM_OOM);  // what does not fit at all is refused, and the context stays usable
    REQUIRE(detect(c, 24, 960, 540) == SLM_OK);
    slm_ctx_destroy(c);
    REQUIRE(fake::device_bytes == 0);
    std::free(a);
    return 0;
}

// What a batch is admitted by is what its plan allocates, and slm_plan_bytes counts that.
// (The BF16 pass's parts are bounded, not counted: one more for each of 152 CTAs, of 3 KB
// and the buffers' quarter.)
int plans_hold_what_is_counted() {
    std::vector<uint32_t> bad;
    uint32_t seed = 1;
    auto next = [&](uint32_t n) { return (seed = seed * 1664525u + 1013904223u) / 65536u % n; };
    for (const slm_precision prec : {SLM_PREC_FP32, SLM_PREC_BF16, SLM_PREC_FP8})
        for (int round = 0; round < 40; ++round) {
            slm_ctx *c = nullptr;
            REQUIRE(slm_ctx_create(nullptr, &c) == SLM_OK);
            const uint32_t most = round % 4 == 0 ? 9000 : round % 4 == 1 ? 2000 : round % 4 == 2 ? 300 : 40000;
            const uint32_t nv = 2 + next(most > 3000 ? 4 : 30), np = 1 + next(round % 3 ? 40 : 400);
            std::vector<uint32_t> n(nv);
            for (uint32_t &v : n) v = next(8) ? 1 + next(most) : next(3);
            std::vector<float> rows(size_t(most + 3) * 128);
            slm_store *st = nullptr;
            REQUIRE(slm_store_create(c, size_t(nv) * (most + 3), nv, &st) == SLM_OK);
            for (uint32_t v : n) REQUIRE(slm_store_add_view(st, rows.data(), v, nullptr) == SLM_OK);
            std::vector<slm_pair> pairs(np);
            for (slm_pair &p : pairs) p = slm_pair{next(nv), next(nv)};
            const int mutual = round & 1;
            slm_tune t{};
            t.use_graph = 2;
            slm_plan *warm = nullptr, *p = nullptr;  // the first builds the store's images
            REQUIRE(slm_plan_create(c, st, pairs.data(), np, 0.8f, mutual, prec, &t, &warm) == SLM_OK);
            const uint64_t before = slm_ctx_bytes_in_use(c);
            REQUIRE(slm_plan_create(c, st, pairs.data(), np, 0.8f, mutual, prec, &t, &p) == SLM_OK);
            const uint64_t held = slm_ctx_bytes_in_use(c) - before, counted = batch_bytes(st, n, pairs, prec, mutual);
            REQUIRE(slm_plan_bytes(p) == held);
            if (counted < held || counted > held + held / 4 + (768 << 10)) {
                std::printf("precision %d, %u pairs of up to %u rows, mutual %d: holds %llu, counted %llu\n", (int)prec, np, most, mutual,
                            (unsigned long long)held, (unsigned long long)counted);
                bad.push_back(round);
            }
            slm_plan_destroy(p);
            slm_plan_destroy(warm);
            slm_store_destroy(st);
            slm_ctx_destroy(c);
        }
    REQUIRE(bad.empty());
    return 0;
}

// A server within a small budget: batches of unlike shapes one after the other in one
// slot, whose buffers keep the size of the largest before.
int serving_batches_of_unlike_shapes() {
    for (const slm_precision prec : {SLM_PREC_FP32, SLM_PREC_BF16, SLM_PREC_FP8}) {
        std::vector<float> rows(size_t(20000) * 128);
        std::vector<uint32_t> n(12, 64);  // the first view's many rows now as rows, now as columns
        n[0] = 20000;
        uint64_t largest = 0, images = 0;
        for (int pass = 0; pass < 2; ++pass) {  // the first finds what the batches need
            slm_server_opts o{};
            o.max_descs = 60000, o.max_views = 64, o.slots = 1, o.max_batch_pairs = 4096, o.tick_us = 50;
            o.ratio = 0.8f, o.mutual = 1, o.prec = prec;
            o.hbm_budget = pass ? images + largest + largest / 32 : 0;
            slm_server *srv = nullptr;
            REQUIRE(slm_server_create(&o, &srv) == SLM_OK);
            images = srv->ctx->used.load();
            std::vector<slm_pair> out(1), pairs;
            for (uint32_t v = 0; v < n.size(); ++v) {
                pairs.clear();
                if (v % 2) pairs.assign(v % 3 ? 1 : 2, slm_pair{0, SLM_SELF});
                if (v && v % 2 == 0) pairs.assign(prec == SLM_PREC_FP32 ? 2 : 4, slm_pair{SLM_SELF, 0});
                std::vector<slm_pair> named = pairs;
                for (slm_pair &p : named) p = slm_pair{p.i == SLM_SELF ? v : p.i, p.j == SLM_SELF ? v : p.j};
                if (!pass) {
                    std::vector<uint32_t> seen(n.begin(), n.begin() + v + 1);
                    largest = std::max(largest, batch_bytes(srv->store, seen, named, prec, 1));
                }
                uint64_t ticket = 0;
                std::vector<uint64_t> off(pairs.size() + 1);
                REQUIRE(slm_server_submit(srv, rows.data(), n[v], pairs.data(), (uint32_t)pairs.size(), nullptr, &ticket) == SLM_OK);
                REQUIRE(slm_server_wait(srv, ticket, 20000, out.data(), 0, off.data(), nullptr) == SLM_OK);
            }
            slm_server_destroy(srv);
            REQUIRE(fake::device_bytes == 0);
        }
    }
    return 0;
}

// Items a SM asked for are whole tiles against ranges of whole tiles, four a SM too; only
// the default cuts a batch of few tiles finer.
int items_asked_for() {
    slm_ctx *c = nullptr;
    slm_store *st = nullptr;
    REQUIRE(slm_ctx_create(nullptr, &c) == SLM_OK);
    REQUIRE(slm_store_create(c, 2000, 2, &st) == SLM_OK);
    std::vector<float> rows(size_t(1000) * 128);
    REQUIRE(slm_store_add_view(st, rows.data(), 700, nullptr) == SLM_OK && slm_store_add_view(st, rows.data(), 900, nullptr) == SLM_OK);
    const slm_pair pr{0, 1};
    for (const uint32_t ips : {0u, 1u, 2u, 4u, 8u}) {
        slm_tune t{};
        t.items_per_sm = ips;
        slm_plan *p = nullptr;
        REQUIRE(slm_plan_create(c, st, &pr, 1, 0.8f, 1, SLM_PREC_FP32, &t, &p) == SLM_OK);
        bool whole = true;
        for (const slm::Item &it : p->items) whole &= it.g0 == 0 && it.g1 == 4 && it.q0 % 4 == 0 && (it.q1 % 4 == 0 || it.q1 == 29);
        REQUIRE(whole == (ips != 0));
        slm_plan_destroy(p);
    }
    // the autotuner looks at the default there too
    slm_tune best{};
    float ms = 0;
    REQUIRE(slm_autotune(c, st, &pr, 1, 0.8f, 1, SLM_PREC_FP32, &best, &ms) == SLM_OK);
    REQUIRE(best.items_per_sm == 0);  // the first of equals: every timing here is the same
    slm_store_destroy(st);
    slm_ctx_destroy(c);
    return 0;
}

int main(int argc, char **argv) {
    const std::map<std::string, int (*)()> checks = {
        {"tracks_that_share_matches", tracks_that_share_matches},
        {"sampson_waits_after_a_failure", sampson_waits_after_a_failure},
        {"single_pair_waits_after_a_failure", single_pair_waits_after_a_failure},
        {"plans_hold_what_is_counted", plans_hold_what_is_counted},
        {"serving_batches_of_unlike_shapes", serving_batches_of_unlike_shapes},
        {"items_asked_for", items_asked_for},
        {"detection_within_its_budget", detection_within_its_budget},
        {"idle_workspaces_give_memory_back", idle_workspaces_give_memory_back},
    };
    if (argc == 2 && checks.count(argv[1])) return checks.at(argv[1])();
    for (const auto &k : checks) std::printf("%s\n", k.first.c_str());
    return argc > 1;
}
