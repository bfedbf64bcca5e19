// Host-side parts of the engine's headers, checked without a GPU: the largest
// batch of middle vertices whose wedge positions are 32-bit numbers.
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

int main() { return count_batch(); }
