// Host-side parts of the engine's headers, checked without a GPU: the largest
// batch of middle vertices whose wedge positions are 32-bit numbers; the peel's
// counters past 2^32.
#include <cstdint>
#include <cstdio>

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

int main() { return count_batch() || peel_counters(); }
