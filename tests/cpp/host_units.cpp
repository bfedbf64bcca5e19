// Host-side parts of the engine's headers, checked without a GPU: the largest
// batch of middle vertices whose wedge positions are 32-bit numbers; the peel's
// counters past 2^32; the device buffers of a call that ends by an exception; the
// CTAs of a batch's graphs.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <new>

#include "../../gpu_bitruss_gb300/csrc/bt_internal.h"

#define CHECK(x)                                             \
    do {                                                     \
        if (!(x)) {                                          \
            std::printf("line %d: %s\n", __LINE__, #x);      \
            return 1;                                        \
        }                                                    \
    } while (0)

static int count_batch() {
    const uint32_t rows[] = {0, 1, 511, 4190212, 4190213, 4194302, 4194303, 4194304, 0x7ffffffe, 0x7fffffff};
    for (uint32_t d : rows) {
        const uint64_t b = bt_count_batch(d);
        CHECK(b >= 1 && b <= kCountBatch);
        // no position that a warp reaches, the first past the last included, wraps
        CHECK(b * d + kCountStride <= 0xffffffffull);
        // and no smaller than it needs to be
        CHECK(b == kCountBatch || (b + 1) * (d + 1ull) + kCountStride > 0xffffffffull);
    }
    return 0;
}

// 1,000 tasks of a warp, the largest there can be, with the carry at each one's end
static int peel_counters() {
    struct {
        unsigned long long w_probes = 0, w_hits = 0, w_decs = 0;
    } totals;
    PeelWork w;
    for (uint32_t t = 0; t < 1000; t++) {
        w.probes += 0x7fffffffu;
        w.hits += 1u << 26;
        w.decs += 3u << 26;
        if (w.full()) w.carry(totals, [](unsigned long long *x, uint32_t v) { *x += v; });
        CHECK(!w.full());
    }
    CHECK(totals.w_probes + w.probes == 1000ull * 0x7fffffffu);
    CHECK(totals.w_hits + w.hits == 1000ull << 26);
    CHECK(totals.w_decs + w.decs == 3000ull << 26);
    return 0;
}

// stand-ins for the context's allocator: what is held, and one failing call
static std::vector<void *> g_held;
static int g_fail_at = -1, g_calls = 0;
bt_status ctx_alloc(bt_ctx *, void **p, uint64_t) {
    *p = nullptr;
    if (g_calls++ == g_fail_at) return BT_ERR_DEVICE_MEMORY;
    *p = new char;
    g_held.push_back(*p);
    return BT_OK;
}
void ctx_free(bt_ctx *, void *p) {
    if (!p) return;
    for (size_t i = 0; i < g_held.size(); i++)
        if (g_held[i] == p) {
            g_held.erase(g_held.begin() + (long)i);
            delete static_cast<char *>(p);
            return;
        }
    std::printf("freed twice\n");
}
static bt_status use_buffers(bool raise) {
    CtxBuffers b(nullptr);
    uint32_t *x = nullptr;
    uint2 *y = nullptr;
    BT_TRY(b.alloc(&x, 4));
    BT_TRY(b.alloc(&y, 8));
    if (!x || !y || g_held.size() != 2) return BT_ERR_STATE;
    if (raise) throw std::bad_alloc();
    return BT_OK;
}
static int call_buffers() {
    CHECK(use_buffers(false) == BT_OK && g_held.empty());
    bool caught = false;
    try {
        use_buffers(true);
    } catch (const std::bad_alloc &) {
        caught = true;
    }
    CHECK(caught && g_held.empty());
    for (int k = 0; k < 2; k++) {
        g_calls = 0;
        g_fail_at = k;
        CHECK(use_buffers(true) == BT_ERR_DEVICE_MEMORY && g_held.empty());
    }
    return 0;
}

// End of the last graph where teams of these sizes take the jobs in order.
static double makespan(const std::vector<PeelJob> &jobs, const std::vector<uint32_t> &size) {
    std::vector<double> free_at(size.size(), 0.0);
    double last = 0;
    for (size_t q = 0; q < jobs.size(); q++) {
        size_t t = 0;
        for (size_t k = 1; k < size.size(); k++)
            if (free_at[k] < free_at[t]) t = k;
        if (q < size.size()) t = q;
        free_at[t] += bt_peel_chain_us(jobs[q]) + bt_peel_walk_us(jobs[q]) / size[t];
        last = std::max(last, free_at[t]);
    }
    return last;
}
static int team_sizes() {
    const uint32_t ctas[] = {1, 2, 5, 152};
    uint32_t seed = 1;
    for (uint32_t c : ctas)
        for (uint32_t n : {1u, 2u, 3u, 40u, 700u}) {
            std::vector<PeelJob> jobs;
            for (uint32_t q = 0; q < n; q++) {
                seed = seed * 1664525u + 1013904223u;
                jobs.push_back(PeelJob{1 + (seed >> 12), seed % 3 ? (uint64_t)seed >> (seed & 15) : 0});
            }
            const std::vector<uint32_t> size = bt_plan_teams(jobs, c);
            uint32_t sum = 0;
            CHECK(!size.empty() && size.size() <= n && size.size() <= c);
            for (uint32_t s : size) {
                CHECK(s >= 1);
                sum += s;
            }
            CHECK(sum == c);
            // never longer than one after the other on all of them
            CHECK(makespan(jobs, size) <= makespan(jobs, {c}) * 1.0001);
        }
    // a hub-skewed graph of 100k edges beside ten uniform ones of 400k: by far the
    // longest, though it has the fewest edges
    std::vector<PeelJob> mixed{PeelJob{100000, 140000000}};
    for (int q = 0; q < 10; q++) mixed.push_back(PeelJob{400000, 1150});
    for (int q = 1; q <= 10; q++)
        CHECK(bt_peel_chain_us(mixed[0]) + bt_peel_walk_us(mixed[0]) > 50 * (bt_peel_chain_us(mixed[q]) + bt_peel_walk_us(mixed[q])));
    CHECK(bt_plan_teams(mixed, 152)[0] >= 100);
    // equal graphs whose chains outweigh their walks run side by side
    CHECK(bt_plan_teams(std::vector<PeelJob>(48, PeelJob{20000, 485050}), 152).size() >= 16);
    return 0;
}

int main() { return count_batch() || peel_counters() || call_buffers() || team_sizes(); }
