// bt_device.cuh -- device building blocks shared by the peeling (msp) and
// h-index (hidx) kernels: the bounded grid barrier, the row hash tables and
// warp-wide sums and searches; and the search for a slot's row.
#pragma once

#include <cub/block/block_scan.cuh>

#include <cstdint>

#include "bt_internal.h"

namespace bt {

constexpr uint32_t kEmpty = 0xffffffffu;

// The row x with off[x] <= p < off[x + 1] (0 <= p < off[n]; rows may be empty).
// Neighbouring lanes ask for the same or neighbouring rows, so the ~17 loads of
// the search come from L1.
__device__ __forceinline__ uint32_t row_of_slot(const uint32_t *off, uint32_t n, uint32_t p) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(off + mid) <= p) lo = mid;
        else hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// memory-model helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// count and abort share one 8-byte word, so a waiting CTA reads both with one load.
struct __align__(8) Barrier {
    unsigned count, abort, error, pad;
};

enum : unsigned { ERR_NONE = 0, ERR_TIMEOUT = 1, ERR_OVERFLOW = 2 };

// One warp of each CTA of a cooperative grid arrives (its first lane) and waits
// until the arrivals reach `target` (the count only grows: the n-th barrier of
// N CTAs waits for n * N, compared modulo 2^32).  The caller synchronises the
// block on both sides; the release / acquire pair then orders everything the
// block did before against everything it does after.  The acquire is the first
// lane's, and a shuffle orders no memory: the __syncwarp before the return hands
// it on to the lanes that load what the others wrote without a block barrier first.
// Waiting on the arrival count itself instead of on a generation word that
// the last CTA writes saves a round trip, and polling without sleeping saves
// the rest: 1.3 us a barrier on 152 CTAs, where count, generation word and
// nanosleep took 2.6 us.  The whole warp polls, not one lane of it: after a
// loop that a single lane ran, the lanes' code stayed apart and every shuffle
// that followed cost about 300 cycles instead of 25.
// The wait is bounded by `wait_ns` of wall time; when it expires the CTA
// records ERR_TIMEOUT, raises `abort` and returns 0, and every other waiting
// CTA returns 0 too.
__device__ __forceinline__ int barrier_wait(Barrier *b, unsigned target, unsigned long long wait_ns) {
    asm volatile(
        "{ .reg .pred p; setp.eq.u32 p, %1, 0; @p red.release.gpu.global.add.u32 [%0], 1; }" ::"l"(&b->count),
        "r"(threadIdx.x & 31)
        : "memory");
    const unsigned long long *word = reinterpret_cast<const unsigned long long *>(&b->count);
    unsigned long long t0 = 0;
    for (unsigned poll = 1;; poll++) {
        unsigned long long w = 0;  // (abort << 32) | count, loaded by the first lane
        asm volatile("{ .reg .pred p; setp.eq.u32 p, %2, 0; @p ld.acquire.gpu.global.u64 %0, [%1]; }"
                     : "+l"(w)
                     : "l"(word), "r"(threadIdx.x & 31)
                     : "memory");
        w = __shfl_sync(0xffffffffu, w, 0);
        if ((unsigned)(w >> 32)) return 0;
        if ((int)((unsigned)w - target) >= 0) {
            __syncwarp();
            return 1;
        }
        if ((poll & 3) == 0) {
            const unsigned long long t = __shfl_sync(0xffffffffu, global_ns(), 0);
            if (!t0) t0 = t;
            else if (t - t0 > wait_ns) {
                atomicCAS(&b->error, 0u, (unsigned)ERR_TIMEOUT);
                atomicExch(&b->abort, 1u);
                return 0;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// row tables: neighbour -> edge id (or value) of every row's live edges
// ---------------------------------------------------------------------------
//
// 32-byte buckets of four (neighbour, edge id) pairs; a key goes to the emptier
// of two buckets, and a lookup reads both at once: one round trip whether or
// not the key is there.  (With one bucket per key and linear probing, one lane
// in twenty needed a second round trip at the same fill, so nearly every warp
// did.)  A key that finds both full goes to the buckets after the second.  A
// row of d edges has bt_row_buckets(d) buckets: 1.5 slots per edge, always at
// least one of them free.  A bucket's number is the high half of a
// multiplicative hash times the bucket count, which need not be a power of two.
struct RowPlace {
    uint32_t h1, h2;
};

__device__ __forceinline__ RowPlace row_place(uint32_t y, uint32_t nb) {
    return RowPlace{__umulhi(y * 0x9E3779B1u, nb), __umulhi(y * 0x85EBCA6Bu + 0x165667B1u, nb)};
}

struct RowBucket {
    uint4 a, b;
};

__device__ __forceinline__ RowBucket row_bucket(const uint4 *pool, uint32_t tab, uint32_t h) {
    const uint4 *p = pool + 2 * ((size_t)tab + h);
    return RowBucket{p[0], p[1]};
}

// y's edge id in a bucket, or kEmpty.
__device__ __forceinline__ uint32_t row_match(const RowBucket &q, uint32_t y) {
    uint32_t e = kEmpty;
    if (q.a.x == y) e = q.a.y;
    if (q.a.z == y) e = q.a.w;
    if (q.b.x == y) e = q.b.y;
    if (q.b.z == y) e = q.b.w;
    return e;
}

// Edge id of y, given its two buckets (nb buckets from tab), or kEmpty.
__device__ __forceinline__ uint32_t row_resolve(const uint4 *pool, uint32_t tab, uint32_t nb, RowPlace at,
                                                const RowBucket &q1, const RowBucket &q2, uint32_t y) {
    uint32_t e = min(row_match(q1, y), row_match(q2, y));  // kEmpty is the largest value
    if (e == kEmpty && q1.b.z != kEmpty && q2.b.z != kEmpty) {
        // both full (a bucket fills in order): the key may be in those after the second
        uint32_t h = at.h2;
        for (uint32_t probe = 1; probe < nb; probe++) {
            h = h + 1 == nb ? 0 : h + 1;
            const RowBucket q = row_bucket(pool, tab, h);
            e = row_match(q, y);
            if (e != kEmpty || q.b.z == kEmpty) break;
        }
    }
    return e;
}

// The same in a table filled first bucket first (row_build<true>): a key that
// is not in its first bucket is elsewhere only if that bucket is full, so most
// lookups read one bucket.  For kernels bound by the reads, not their latency.
__device__ __forceinline__ uint32_t row_find(const uint4 *pool, uint32_t tab, uint32_t nb, uint32_t y) {
    const RowPlace at = row_place(y, nb);
    RowBucket q = row_bucket(pool, tab, at.h1);
    uint32_t e = row_match(q, y);
    uint32_t h = at.h2;
    for (uint32_t probe = 0; probe <= nb && e == kEmpty && q.b.z != kEmpty; probe++) {
        q = row_bucket(pool, tab, h);
        e = row_match(q, y);
        h = h + 1 == nb ? 0 : h + 1;
    }
    return e;
}

// Build the table of one row by one warp; value(j) is what slot j's key maps to.
// FIRST: fill a key's first bucket before its second (see row_find), else both
// evenly (see row_resolve).
template <bool FIRST = false, class Value>
__device__ __forceinline__ void row_build(uint4 *pool, uint32_t tab, uint32_t d, const uint32_t *nbr, Value value) {
    const uint32_t lane = threadIdx.x & 31, nb = bt_row_buckets(d);
    uint4 *t = pool + 2 * (size_t)tab;
    for (uint32_t k = lane; k < 2 * nb; k += 32) t[k] = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
    __syncwarp();
    uint2 *slots = reinterpret_cast<uint2 *>(t);
    for (uint32_t j = lane; j < d; j += 32) {
        const uint32_t y = nbr[j], e = value(j);
        const RowPlace at = row_place(y, nb);
        bool placed = false;
        // its two buckets, then those after the second
        for (uint32_t c = 0; c < 8 && !placed; c++) {
            const uint32_t second = FIRST ? c >> 2 : c & 1;
            uint2 *slot = slots + 4 * (size_t)(second ? at.h2 : at.h1) + (FIRST ? c & 3 : c >> 1);
            const uint32_t prev = atomicCAS(&slot->x, kEmpty, y);
            if (prev == kEmpty || prev == y) {
                slot->y = e;
                placed = true;
            }
        }
        uint32_t h = at.h2;
        for (uint32_t probe = 1; probe < nb && !placed; probe++) {
            h = h + 1 == nb ? 0 : h + 1;
            for (uint32_t c = 0; c < 4 && !placed; c++) {
                uint2 *slot = slots + 4 * (size_t)h + c;
                const uint32_t prev = atomicCAS(&slot->x, kEmpty, y);
                if (prev == kEmpty || prev == y) {
                    slot->y = e;
                    placed = true;
                }
            }
        }
    }
}

// y's place in a row's table (index into the pool as (key, value) pairs), or
// ~0 when it is not there.
__device__ __forceinline__ size_t row_entry(const uint4 *pool, uint32_t tab, uint32_t nb, uint32_t y) {
    const uint2 *slots = reinterpret_cast<const uint2 *>(pool + 2 * (size_t)tab);
    const RowPlace at = row_place(y, nb);
    for (uint32_t c = 0; c < 8; c++) {
        const size_t i = 4 * (size_t)(c & 1 ? at.h2 : at.h1) + (c >> 1);
        if (slots[i].x == y) return 4 * (size_t)tab + i;
    }
    uint32_t h = at.h2;
    for (uint32_t probe = 1; probe < nb; probe++) {
        h = h + 1 == nb ? 0 : h + 1;
        for (uint32_t c = 0; c < 4; c++) {
            const size_t i = 4 * (size_t)h + c;
            if (slots[i].x == y) return 4 * (size_t)tab + i;
        }
    }
    return ~(size_t)0;
}

// Per vertex, one 16-byte load: row start, live degree, first bucket of its
// row table, and the row's position total (sum of its neighbours' degrees).
struct __align__(16) VRec {
    uint32_t off, deg, tab, hop;
};

__device__ __forceinline__ VRec load_vrec(const VRec *p) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(p));
    return VRec{q.x, q.y, q.z, q.w};
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += t;
    }
    return v;
}

// Last slot s in [0, d) with pre[s] <= f (pre ascending, pre[0] <= f),
// by one warp with a 32-way search: log32(d) coalesced steps.
__device__ inline uint32_t warp_find_slot(const uint32_t *pre, uint32_t d, uint32_t f) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = d;
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t idx = lo + lane * step;
        const bool ok = idx < hi && pre[idx] <= f;
        const uint32_t bal = __ballot_sync(0xffffffffu, ok);
        const uint32_t k = 31 - __clz(bal);
        lo = lo + k * step;
        hi = min(lo + step, hi);
    }
    const bool ok = lo + lane < hi && pre[lo + lane] <= f;
    const uint32_t bal = __ballot_sync(0xffffffffu, ok);
    return lo + 31 - __clz(bal);
}

}  // namespace bt
