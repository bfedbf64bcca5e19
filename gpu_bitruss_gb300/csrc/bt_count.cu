// bt_count.cu -- vertex-priority butterfly counting (bfc) and per-edge
// butterfly support (ebfc).
//
// Same arithmetic as the reference's bfc_kernel / ebfc_kernel
// (src/bfc/bfc_vpp.cu:33-107, 126-221) and CPU ebfc (src/bfc/cpu_bfc.cpp:24-122):
// a butterfly is counted once, at its vertex u of highest priority
// p(x) = (degree, id), as a pair of wedges u-v-w, u-x-w with p(v), p(w),
// p(x) < p(u).  With c(u,w) wedges from u to w the count gains C(c,2) and
// each wedge edge (u,v), (v,w) gains c-1 support.
//
// GB300 layout: vertices are relabelled by priority rank and rows sorted by
// rank, so the lower-priority neighbours of u are a row suffix found by one
// binary search (no per-element priority test, no reads of the skipped
// prefix).
//
// What bounds it: one random counter update and one random read per wedge, and
// for supports one update per wedge edge.  With counters in HBM / L2 (one
// array per resident CTA) the 2M-edge Chung-Lu graph's 1.6e8 wedges made 5.8e8
// L2 requests in 6.6 ms, and most vertices, which have a handful of wedges,
// still took a whole CTA through four block barriers.  Now:
//  * Counters are in shared memory: rank w counts at w - (r + 1) for the
//    kDense ranks after the start vertex r.  Ranks follow degree, so these are
//    where almost all wedges end; the rest use a counter array in HBM, one per
//    CTA, which graphs of up to kDense vertices do not need at all.
//  * A start vertex with at most kLightWedges wedges is one warp's, with a
//    small hash in shared memory; with at most 32, the warp matches them in
//    registers.  A larger one is taken by the whole CTA afterwards.
//  * The 32 warps of a CTA take ranks n / 32 apart, so a CTA meets a large
//    vertex once in a chunk, the largest first.
//  * Middle vertices are resolved one per lane (the binary search is a chain
//    of loads), 32 by a warp or 1,024 by the CTA, and their suffixes laid end to
//    end and dealt out in equal stretches, so lanes and warps stay busy whatever
//    the rows' lengths.
//  * Supports are summed per row slot: the slots of a suffix are neighbours, so
//    32 updates are 4 sectors, where the edge ids' are 32.  k_support adds a
//    slot's sum to its edge.
//  * ANY_ORDER (no supports): rows are not sorted, whole rows are walked and ends
//    that do not rank below the start vertex left out; large vertices take a pass
//    for each kDense ranks instead of counters in HBM (bt_noalloc.cu has the
//    figures).
// Supports of a 2M-edge Chung-Lu graph: 6.6 -> 2.6 ms; of a 4M-edge hub-skewed
// graph (4e7 wedges, most rows of 10) 7.0 -> 1.1 ms; of a 500k-edge graph of mean
// degree 8 2.0 -> 0.5 ms.
#include <algorithm>

#include "bt_device.cuh"
#include "bt_internal.h"

namespace {

using bt::warp_inclusive;
constexpr int kCountThreads = 1024;
constexpr uint32_t kCountWarps = kCountThreads / 32;
constexpr uint32_t kDense = 52224;         // counters in shared memory (204 KiB)
constexpr uint32_t kBatch = kCountBatch;   // middle vertices a CTA lays end to end at once
static_assert(kCountBatch == kCountThreads && kCountStride == kCountThreads * 4, "one per thread; four positions each");
// Longest row a single warp may have to walk by itself.  Supports (and counts) in
// ms with warps on their own and in batches of the CTA: hub-skewed graphs of 1 to
// 4M edges with rows of up to 51 0.50 and 0.77 (0.20 and 0.34), 212 1.45 and 1.72
// (0.51 and 0.72), 463 1.74 and 1.76 (0.65 and 0.74), 1,042 4.55 and 3.67 (2.35 and
// 1.86); uniform ones of 2 to 4M, whose rows are all about as long, 137 0.99 and 0.99
// (0.34 and 0.43), 300 2.75 and 2.16 (0.87 and 0.92), 556 8.1 and 6.2 (2.42 and 2.67);
// the Chung-Lu graph (rows of up to 10k) 5.7 and 2.6.
constexpr uint32_t kShortRow = 512;
constexpr uint32_t kSlots = 512;           // hash slots of one warp
constexpr uint32_t kLightWedges = 320;     // wedges a warp's hash takes
constexpr uint32_t kLightMids = 64;        // middle vertices a warp looks at

// first index i in row[0..len) with row[i] > key (rows ascending)
__device__ __forceinline__ uint32_t upper_bound_u32(const uint32_t *row, uint32_t len, uint32_t key) {
    uint32_t lo = 0, hi = len;
    while (lo < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (__ldg(row + mid) <= key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

struct CountArgs {
    uint32_t n, span;    // vertices; vertices of the largest graph of an arena (else n)
    uint32_t dense;      // counters in shared memory
    uint32_t batch;      // middle vertices at once: their suffixes' lengths are added in 32 bits
    uint32_t chunks;     // ceil(n / warps per CTA)
    uint32_t least;      // middle slots from which a start vertex can close a butterfly
    uint32_t short_u, short_l;  // the other side's rows are short: for a start vertex in U, in L
    const uint32_t *off, *deg, *nbr, *is_u;
    const uint2 *rows;   // ANY_ORDER: off and deg side by side (then null)
    uint32_t slots;      // ANY_ORDER: entries of nbr
    const uint32_t *seg_base;  // per rank: first rank of its graph (NULL: one graph)
    uint32_t *cnt;       // gridDim.x * span counters of ranks past the dense ones (zero on entry and exit)
    uint32_t *touched;   // gridDim.x * span
    void *acc;           // per slot: support sum (PER_EDGE), uint32 or uint64 (WIDE)
    unsigned long long *count;  // butterfly total
    uint32_t *next_chunk;       // work counter
    uint32_t *layout_error;     // set if a wedge leaves its graph's ranks
};

struct __align__(16) CountSmem {
    // a batch of middle vertices with a suffix: its first slot, the prefix of
    // the lengths, the support of (r, s), the slot of s in r's row
    uint32_t p0[kBatch], pre[kBatch + 1], sum[kBatch], at[kBatch];
    uint32_t big[kCountWarps];     // start vertices left to the CTA (rank + 1)
    uint2 row[kCountWarps];        // their rows
    uint32_t wlen[kCountWarps], wcnt[kCountWarps];
    uint32_t chunk, touched;
    unsigned long long red[kCountWarps];
};

template <bool WIDE>
__device__ __forceinline__ void acc_add(void *acc, uint32_t slot, unsigned long long v) {
    if constexpr (WIDE) atomicAdd(static_cast<unsigned long long *>(acc) + slot, v);
    else atomicAdd(static_cast<uint32_t *>(acc) + slot, (uint32_t)v);
}

// r's first slot and its degree.  ANY_ORDER: the tables may be another call's by
// now (bt_noalloc.cu); a row that leaves nbr is taken as empty.  (Comparing each
// row's end with the next one's start takes a 300k-edge count from 252 to 260 us,
// these compares to 255; only a large start vertex's own row is compared so.)
template <bool ANY_ORDER>
__device__ __forceinline__ uint2 row_of(const CountArgs &a, uint32_t r) {
    if (!ANY_ORDER) return make_uint2(__ldg(a.off + r), __ldg(a.deg + r));
    const uint2 row = __ldg(a.rows + r);
    const bool fits = row.x <= a.slots & row.y <= a.slots - row.x & row.y < a.n;
    return make_uint2(row.x, fits ? row.y : 0);
}

// 32 middle vertices of r, one per lane: where the suffix of ranks above r
// starts in each one's row, and its length (0 past the end of r's row).
// ANY_ORDER: rows are not sorted; the whole row of a middle vertex above r is
// taken, and the visitor leaves out the ranks up to r.
struct Mid {
    uint32_t p0, len;
};
template <bool ANY_ORDER>
__device__ __forceinline__ Mid load_mid(const CountArgs &a, uint32_t rb, uint32_t rl, uint32_t i, uint32_t r) {
    Mid m{0, 0};
    if (i < rl) {
        const uint32_t s = __ldg(a.nbr + rb + i);
        if (ANY_ORDER && s >= a.n) return m;
        const uint2 row = row_of<ANY_ORDER>(a, s);
        const uint32_t sb = row.x, sl = row.y;
        const uint32_t j0 = ANY_ORDER ? (s > r ? 0 : sl) : upper_bound_u32(a.nbr + sb, sl, r);
        m.p0 = sb + j0;
        m.len = sl - j0;
    }
    return m;
}

// Visit every wedge end of the warp's 32 middle vertices, their suffixes laid
// end to end, by the whole warp each time: f(active, w, slot of w in s's row,
// lane of s).
template <class F>
__device__ __forceinline__ void visit_wedges(const uint32_t *nbr, Mid m, F f) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t pre = warp_inclusive(m.len);
    const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
    pre -= m.len;
    for (uint32_t fb = 0; fb < total; fb += 32) {
        const uint32_t g = fb + lane;
        uint32_t k = 0;  // the last lane with pre <= g
#pragma unroll
        for (uint32_t o = 16; o; o >>= 1) {
            const uint32_t t = __shfl_sync(0xffffffffu, pre, k + o);
            if (t <= g) k += o;
        }
        const uint32_t p = __shfl_sync(0xffffffffu, m.p0, k) + (g - __shfl_sync(0xffffffffu, pre, k));
        f(g < total, g < total ? __ldg(nbr + p) : 0u, p, k);
    }
}

__device__ __forceinline__ uint32_t light_hash(uint32_t w) { return (w * 0x9E3779B1u) >> 23; }  // kSlots slots
static_assert(kSlots == 512, "light_hash yields 9 bits");

// Slot of key w + 1 in the warp's hash (keys[0, kSlots), 0 = free); inserts it.
__device__ __forceinline__ uint32_t light_slot(uint32_t *keys, uint32_t w) {
    uint32_t h = light_hash(w);
    for (;;) {  // at most kLightWedges keys: a free slot is always met
        const uint32_t prev = atomicCAS(keys + h, 0u, w + 1);
        if (prev == 0 || prev == w + 1) return h;
        h = (h + 1) & (kSlots - 1);
    }
}

// All of one small start vertex by one warp (at most kLightWedges wedges);
// returns the lane's share of the butterflies.  table is zero on entry and exit.
template <bool PER_EDGE, bool WIDE, bool ANY_ORDER>
__device__ __forceinline__ unsigned long long light_vertex(const CountArgs &a, uint32_t *table, uint32_t r,
                                                           uint32_t first,
                                                           const Mid (&m)[kLightMids / 32], uint32_t total) {
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long local = 0;
    uint32_t *keys = table, *cnts = table + kSlots;
    if (total <= 32) {
        // every wedge end in a register of its own lane
        uint32_t w = 0, p = 0, k = 0, at = 0;
        bool have = false;
#pragma unroll
        for (uint32_t q = 0; q < kLightMids / 32; q++) {
            visit_wedges(a.nbr, m[q], [&](bool on, uint32_t vw, uint32_t vp, uint32_t vk) {
                // this round's ends go to the lanes after those taken
                const uint32_t cnt = __popc(__ballot_sync(0xffffffffu, on));
                const uint32_t src = (lane - at) & 31;
                const uint32_t sw = __shfl_sync(0xffffffffu, vw, src), sp = __shfl_sync(0xffffffffu, vp, src);
                const uint32_t sk = __shfl_sync(0xffffffffu, vk, src);
                if (lane >= at && lane - at < cnt) {
                    w = sw;
                    p = sp;
                    k = q * 32 + sk;
                    have = true;
                }
                at += cnt;
            });
        }
        if (ANY_ORDER) have = have && w > r;
        const uint32_t same = __match_any_sync(0xffffffffu, have ? w : 0xffffffffu);
        const uint32_t c = __popc(same);
        if (have && c > 1) {
            if ((same & ((1u << lane) - 1)) == 0) local = (unsigned long long)c * (c - 1) / 2;
            if (PER_EDGE) {
                acc_add<WIDE>(a.acc, p, c - 1);
                acc_add<WIDE>(a.acc, first + k, c - 1);
            }
        }
        return local;
    }
#pragma unroll
    for (uint32_t q = 0; q < kLightMids / 32; q++)
        visit_wedges(a.nbr, m[q], [&](bool on, uint32_t w, uint32_t, uint32_t) {
            if (on && (!ANY_ORDER || w > r)) local += atomicAdd(cnts + light_slot(keys, w), 1u);
        });
    __syncwarp();
    if (PER_EDGE) {
#pragma unroll
        for (uint32_t q = 0; q < kLightMids / 32; q++)
            visit_wedges(a.nbr, m[q], [&](bool on, uint32_t w, uint32_t p, uint32_t k) {
                if (!on) return;
                const uint32_t c = cnts[light_slot(keys, w)];
                if (c > 1) {
                    acc_add<WIDE>(a.acc, p, c - 1);
                    acc_add<WIDE>(a.acc, first + q * 32 + k, c - 1);
                }
            });
        __syncwarp();
    }
    uint4 *t4 = reinterpret_cast<uint4 *>(table);
    for (uint32_t k = lane; k < 2 * kSlots / 4; k += 32) t4[k] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    return local;
}

// The middle vertices r's row slots [i0, i0 + batch) into sm, those with a
// suffix only; returns how many.  Starts and ends synchronised.
template <bool ANY_ORDER>
__device__ __forceinline__ uint32_t load_batch(const CountArgs &a, CountSmem &sm, uint32_t rb, uint32_t rl,
                                               uint32_t i0, uint32_t r) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t i = i0 + threadIdx.x;
    const Mid m = load_mid<ANY_ORDER>(a, rb, threadIdx.x < a.batch ? rl : 0, i, r);
    const uint32_t has = __ballot_sync(0xffffffffu, m.len != 0);
    uint32_t pre = warp_inclusive(m.len);
    if (lane == 31) {
        sm.wlen[warp] = pre;
        sm.wcnt[warp] = __popc(has);
    }
    pre -= m.len;
    __syncthreads();
    const uint32_t wl = warp_inclusive(sm.wlen[lane]), wc = warp_inclusive(sm.wcnt[lane]);
    const uint32_t bl = __shfl_sync(0xffffffffu, wl, warp ? warp - 1 : 0), bc = __shfl_sync(0xffffffffu, wc, warp ? warp - 1 : 0);
    const uint32_t nm = __shfl_sync(0xffffffffu, wc, 31);
    if (m.len) {
        const uint32_t k = (warp ? bc : 0) + __popc(has & ((1u << lane) - 1));
        sm.p0[k] = m.p0;
        sm.pre[k] = (warp ? bl : 0) + pre;
        sm.sum[k] = 0;
        sm.at[k] = rb + i;
    }
    if (threadIdx.x == 31) sm.pre[nm] = wl;  // the first warp's last lane: the total
    __syncthreads();
    return nm;
}
static_assert(kCountWarps == 32, "a warp scans the warps' totals");

// Visit every wedge end of the batch's nm middle vertices, laid end to end and
// dealt to the warps in stretches of 128 (four loads in flight per lane):
// f(active, w, slot of w in s's row, s's place in the batch, whether that is
// the same for the whole warp).
template <class F>
__device__ __forceinline__ void visit_batch(const uint32_t *nbr, const CountSmem &sm, uint32_t nm, F f) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t total = sm.pre[nm];
    for (uint32_t fb = warp * 128; fb < total; fb += kCountStride) {
        // the middle vertex of position fb
        uint32_t k0 = 0, hi = nm;
        while (hi - k0 > 1) {
            const uint32_t md = (k0 + hi) >> 1;
            if (sm.pre[md] <= fb) k0 = md;
            else hi = md;
        }
        uint32_t p[4], k[4], w[4], uni = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
            const uint32_t g0 = fb + q * 32, g = g0 + lane;
            if (g0 >= total) break;  // the whole warp
            uint32_t m = 0;
            if (sm.pre[k0 + 1] >= g0 + 32) {
                uni |= 1u << q;
            } else {
                // every one listed has a wedge, so 32 positions are within 32 of them
                const uint32_t pre = sm.pre[min(k0 + lane, nm)];
#pragma unroll
                for (uint32_t o = 16; o; o >>= 1) {
                    const uint32_t t = __shfl_sync(0xffffffffu, pre, m + o);
                    if (t <= g && k0 + m + o < nm) m += o;
                }
            }
            k[q] = k0 + m;
            p[q] = sm.p0[k[q]] + (g - sm.pre[k[q]]);
            if (g < total) w[q] = __ldg(nbr + p[q]);
            k0 = __shfl_sync(0xffffffffu, k[q], 31);
            if (sm.pre[k0 + 1] <= g0 + 32 && k0 + 1 < nm) k0++;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
            if (fb + q * 32 >= total) break;
            f(fb + q * 32 + lane < total, w[q], p[q], k[q], (uni >> q & 1) != 0);
        }
    }
}

// All of one large start vertex by the CTA; `dense` is zero on entry and exit.
// Ends synchronised.
template <bool PER_EDGE, bool WIDE, bool ANY_ORDER>
__device__ __forceinline__ unsigned long long big_vertex(const CountArgs &a, CountSmem &sm, uint32_t *dense,
                                                         uint32_t r, uint2 row, uint32_t skip) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t base = a.seg_base ? a.seg_base[r] : 0u;
    const uint32_t rb = row.x, rl = row.y;
    const uint32_t start = ANY_ORDER ? 0 : upper_bound_u32(a.nbr + rb, rl, r);
    uint32_t *cnt = a.cnt + (size_t)blockIdx.x * a.span;
    uint32_t *touched = a.touched + (size_t)blockIdx.x * a.span;
    // the ranks counted: the first ones of the graph after r and after `skip` more
    const uint32_t first = r + 1 + skip, most = base + a.span - first;
    const uint32_t near = most < a.dense ? most : a.dense;
    unsigned long long local = 0;
    if (threadIdx.x == 0) sm.touched = 0;
    __syncthreads();
    // pass 1: wedge counts c(r, w) (bfc_vpp.cu:163-187)
    auto count_wedge = [&](uint32_t w) {
        const uint32_t d = w - first;
        if (d < near) {
            atomicAdd(dense + d, 1u);
        } else if (ANY_ORDER) {
            if (w > r && w < a.n && d - near < 0x80000000u) sm.touched = 1;  // ranks past these: another pass
        } else if (a.span > a.dense && w - base < a.span) {
            const uint32_t old = atomicAdd(cnt + (w - base), 1u);
            local += old;
            if (old == 0) touched[atomicAdd(&sm.touched, 1u)] = w - base;
        } else {  // not in r's graph: the arena layout is broken
            *a.layout_error = 1;
        }
    };
    // pass 2: supports (bfc_vpp.cu:191-219); what a wedge end adds to its edges
    auto wedge_share = [&](bool on, uint32_t w) {
        uint32_t c = 0;
        if (on) {
            const uint32_t d = w - first;
            if (d < near) c = dense[d];
            else if (a.span > a.dense && w - base < a.span)
                c = __ldcg(cnt + (w - base));  // written by L2 atomics: bypass L1
        }
        return c > 1 ? c - 1 : 0u;
    };
    if (!ANY_ORDER && rl - start > kBatch && (a.is_u[r] ? a.short_u : a.short_l)) {
        // many short suffixes: every warp on its own, 32 of them at a time
        for (uint32_t i0 = start + warp * 32; i0 < rl; i0 += kBatch)
            visit_wedges(a.nbr, load_mid<ANY_ORDER>(a, rb, rl, i0 + lane, r), [&](bool on, uint32_t w, uint32_t, uint32_t) {
                if (on) count_wedge(w);
            });
        __syncthreads();
        if (PER_EDGE) {
            uint32_t *sum = sm.sum + warp * 32;
            for (uint32_t i0 = start + warp * 32; i0 < rl; i0 += kBatch) {
                sum[lane] = 0;
                __syncwarp();
                visit_wedges(a.nbr, load_mid<ANY_ORDER>(a, rb, rl, i0 + lane, r), [&](bool on, uint32_t w, uint32_t p, uint32_t k) {
                    const uint32_t add = wedge_share(on, w);
                    if (!add) return;
                    acc_add<WIDE>(a.acc, p, add);
                    if (WIDE) acc_add<WIDE>(a.acc, rb + i0 + k, add);
                    else atomicAdd(sum + k, add);
                });
                __syncwarp();
                const uint32_t t = sum[lane];
                if (t) acc_add<WIDE>(a.acc, rb + i0 + lane, t);
                __syncwarp();
            }
            __syncthreads();
        }
    } else {
        uint32_t nm = 0;
        uint64_t seen = 0;
        for (uint32_t i0 = start; i0 < rl; i0 += a.batch) {
            nm = load_batch<ANY_ORDER>(a, sm, rb, rl, i0, r);
            if (ANY_ORDER && (seen += sm.pre[nm]) > a.slots) break;  // no graph's: its rows share no slots
            visit_batch(a.nbr, sm, nm, [&](bool on, uint32_t w, uint32_t, uint32_t, bool) {
                if (on) count_wedge(w);
            });
            __syncthreads();
        }
        // a single batch is still loaded
        for (uint32_t i0 = start; PER_EDGE && i0 < rl; i0 += a.batch) {
            if (rl - start > a.batch) nm = load_batch<ANY_ORDER>(a, sm, rb, rl, i0, r);
            visit_batch(a.nbr, sm, nm, [&](bool on, uint32_t w, uint32_t p, uint32_t k, bool uniform) {
                const uint32_t add = wedge_share(on, w);
                if (add) acc_add<WIDE>(a.acc, p, add);
                if (WIDE) {
                    if (add) acc_add<WIDE>(a.acc, sm.at[k], add);
                } else if (uniform) {
                    const uint32_t t = __reduce_add_sync(0xffffffffu, add);
                    if (lane == 0 && t) atomicAdd(&sm.sum[k], t);
                } else if (add) {
                    atomicAdd(&sm.sum[k], add);
                }
            });
            __syncthreads();
            if (!WIDE && threadIdx.x < nm) {
                const uint32_t t = sm.sum[threadIdx.x];
                if (t) acc_add<WIDE>(a.acc, sm.at[threadIdx.x], t);
            }
            __syncthreads();
        }
    }
    // sum C(c, 2) of the shared counters while they are cleared
    uint4 *d4 = reinterpret_cast<uint4 *>(dense);
    for (uint32_t k = threadIdx.x; k < (near + 3) / 4; k += kCountThreads) {
        const uint4 q = d4[k];
        if (q.x | q.y | q.z | q.w) {
            const uint32_t c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (uint32_t t = 0; t < 4; t++)
                if (c[t]) local += (unsigned long long)c[t] * (c[t] - 1) / 2;
            d4[k] = make_uint4(0, 0, 0, 0);
        }
    }
    if constexpr (!ANY_ORDER) {
        const uint32_t nt = sm.touched;
        for (uint32_t k = threadIdx.x; k < nt; k += kCountThreads) cnt[touched[k]] = 0;
    }
    __syncthreads();
    return local;
}

template <bool PER_EDGE, bool WIDE, bool ANY_ORDER>
__global__ void __launch_bounds__(kCountThreads, 1) k_count(const __grid_constant__ CountArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CountSmem &sm = *reinterpret_cast<CountSmem *>(smem_raw);
    uint32_t *dense = reinterpret_cast<uint32_t *>(smem_raw + sizeof(CountSmem));  // also the warps' hashes
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t words = a.dense > kCountWarps * 2 * kSlots ? a.dense : kCountWarps * 2 * kSlots;
    uint4 *d4 = reinterpret_cast<uint4 *>(dense);
    for (uint32_t k = threadIdx.x; k < words / 4; k += kCountThreads) d4[k] = make_uint4(0, 0, 0, 0);
    if (__syncthreads_or(ANY_ORDER && *a.layout_error)) return;  // nothing to count here: see bt_count_any_order
    uint32_t *table = dense + warp * 2 * kSlots;
    unsigned long long local = 0;
    for (uint32_t c = blockIdx.x; c < a.chunks;) {
        // warp w: rank w * chunks + c
        const uint32_t r = warp * a.chunks + c;
        uint32_t big = 0;
        if (r < a.n) {
            uint2 row = row_of<ANY_ORDER>(a, r);
            const uint32_t rb = row.x, rl = row.y;
            // the suffix of r's own row after r, found 32 ways at a time
            uint32_t lo = 0, hi = ANY_ORDER ? 0 : rl;
            while (hi > lo) {
                const uint32_t step = (hi - lo + 31) / 32, i = lo + lane * step;
                const uint32_t le = __popc(__ballot_sync(0xffffffffu, i < hi && __ldg(a.nbr + rb + i) <= r));
                if (step == 1) {
                    lo += le;
                    break;
                }
                if (le == 0) break;
                hi = min(hi, lo + le * step);
                lo += (le - 1) * step + 1;
            }
            const uint32_t mids = rl - lo;
            if (mids > kLightMids) {
                big = r + 1;
            } else if (mids >= a.least) {
                Mid m[kLightMids / 32];
                uint32_t sum = 0;
#pragma unroll
                for (uint32_t q = 0; q < kLightMids / 32; q++) {
                    m[q] = load_mid<ANY_ORDER>(a, rb, rl, lo + q * 32 + lane, r);
                    sum += min(m[q].len, kLightWedges + 1);
                }
                const uint32_t total = __reduce_add_sync(0xffffffffu, sum);
                if (total > kLightWedges) big = r + 1;
                else if (total) local += light_vertex<PER_EDGE, WIDE, ANY_ORDER>(a, table, r, rb + lo, m, total);
            }
            // (a row that does not end where the next one starts is of no graph)
            if (ANY_ORDER && big && rb + rl != (r + 1 < a.n ? a.rows[r + 1].x : a.slots)) row.y = 0;
            if (lane == 0) sm.row[warp] = row;  // one answer for all threads
        }
        if (lane == 0) sm.big[warp] = big;
        if (threadIdx.x == 0) sm.chunk = gridDim.x + atomicAdd(a.next_chunk, 1u);
        __syncthreads();
        c = sm.chunk;
        for (uint32_t w = 0; w < kCountWarps; w++) {
            if (!sm.big[w]) continue;
            const uint32_t v = sm.big[w] - 1;
            bool more;
            uint32_t skip = 0;
            do {  // no counters but the shared ones: further passes over the ranks past them
                local += big_vertex<PER_EDGE, WIDE, ANY_ORDER>(a, sm, dense, v, sm.row[w], skip);
                more = ANY_ORDER && sm.touched != 0;
                if (ANY_ORDER) __syncthreads();
                skip += a.dense;
            } while (more);
        }
        __syncthreads();
    }
    for (int o = 16; o; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (lane == 0) sm.red[warp] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (uint32_t k = 0; k < kCountWarps; k++) t += sm.red[k];
        if (t) atomicAdd(a.count, t);
    }
}

// Every slot's sum to its edge, and the largest support: an edge's last
// addition returns (with its own share) the edge's support.
template <bool WIDE>
__global__ void __launch_bounds__(256) k_support(uint64_t slots, const void *acc, const uint32_t *eid,
                                                 unsigned long long *sup, unsigned long long *largest) {
    unsigned long long most = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < slots; i += (uint64_t)gridDim.x * blockDim.x) {
        unsigned long long v;
        if constexpr (WIDE) v = static_cast<const unsigned long long *>(acc)[i];
        else v = static_cast<const uint32_t *>(acc)[i];
        if (v) {
            const unsigned long long t = atomicAdd(sup + eid[i], v) + v;
            most = t > most ? t : most;
        }
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, most, o);
        most = t > most ? t : most;
    }
    if ((threadIdx.x & 31) == 0 && most) atomicMax(largest, most);
}

uint32_t dense_of(uint64_t span) { return (uint32_t)(span < kDense ? (span + 3) & ~3ull : kDense); }

size_t count_smem(uint32_t dense) {
    return sizeof(CountSmem) + 4ull * std::max<uint32_t>(dense, kCountWarps * 2 * kSlots);
}

const void *count_kernel(bool per_edge, bool wide) {
    if (!per_edge) return (const void *)k_count<false, false, false>;
    return wide ? (const void *)k_count<true, true, false> : (const void *)k_count<true, false, false>;
}

}  // namespace

// CTAs of the counting kernel that hold counters in device memory
int dev_count_ctas(bt_ctx *ctx) { return ctx->sm_count; }

// Supports are summed in 64 bits where rows repeat a neighbour: with k parallel
// edges r-s and k parallel edges s-w, each slot of r-s gets k (k^2 - 1) (2^32 from
// k = 1,626 on).  Elsewhere each butterfly of an edge has an opposite edge of its
// own, so no support and no slot's sum reaches m < 2^31.
static bool wide_sums(const DevGraph &g) { return g.repeats; }

// One middle slot alone closes a butterfly only if its row repeats an end.
static uint32_t least_mids(const DevGraph &g) { return g.repeats ? 1 : 2; }

uint64_t bt_count_bytes(uint64_t m, uint64_t span, uint64_t ctas, bool wide) {
    return (wide ? 16 : 8) * m + (span > kDense ? 8 * span * ctas : 0) + 1024;
}

bt_status dev_ebfc(bt_ctx *ctx, bool per_edge, uint64_t *count) {
    DevGraph &g = ctx->g;
    cudaStream_t st = ctx->stream;
    const bool wide = wide_sums(g);
    const uint64_t span = g.cnt_span ? g.cnt_span : 1;
    const uint32_t dense = dense_of(span);
    const void *kfn = count_kernel(per_edge, wide);
    const size_t smem = count_smem(dense);
    const uint32_t chunks = (g.n + kCountWarps - 1) / kCountWarps;
    // the limit belongs to the kernel, not to the call: the same value from every
    // thread, or one with a smaller graph lowers it before another's launch
    BT_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)count_smem(kDense)));
    // one CTA per SM (its counters fill the SM's shared memory)
    const uint64_t nctas = std::max<uint64_t>(1, std::min<uint64_t>(ctx->sm_count, chunks));
    // scratch: [0, 64) count, support max, work counter, layout error; then the
    // counters of ranks past the dense ones and their touched lists (zero
    // between calls: the kernel clears what it used), then the slot sums
    const uint64_t far = span > dense ? span * nctas : 0;
    const uint64_t bytes = 256 + 8 * far + (per_edge ? (wide ? 16 : 8) * g.m : 0);
    void *scr = nullptr;
    const uint64_t had = ctx->scratch_bytes;
    BT_TRY(ctx_scratch(ctx, bytes, &scr));
    unsigned long long *head = (unsigned long long *)scr;
    uint32_t *cnt = (uint32_t *)((char *)scr + 256);
    void *acc = cnt + 2 * far;
    if (ctx->scratch_bytes != had) ctx->zero_counters = 0;
    if (ctx->zero_counters < far) BT_CUDA(cudaMemsetAsync(cnt, 0, 4 * far, st));
    ctx->zero_counters = 0;  // until the kernel has ended well
    BT_CUDA(cudaMemsetAsync(head, 0, 64, st));
    if (per_edge && g.m) {
        BT_CUDA(cudaMemsetAsync(acc, 0, (wide ? 16 : 8) * g.m, st));
        BT_CUDA(cudaMemsetAsync(ctx->sup, 0, 8 * g.m, st));
    }
    CountArgs a;
    a.n = g.n;
    a.span = (uint32_t)span;
    a.dense = dense;
    a.chunks = chunks;
    a.batch = bt_count_batch(g.max_deg);
    a.seg_base = g.seg_base;
    a.least = least_mids(g);
    a.short_u = g.max_deg_l <= kShortRow;
    a.short_l = g.max_deg_u <= kShortRow;
    a.is_u = g.is_u;
    a.off = g.off;
    a.deg = g.deg0;
    a.nbr = g.nbr0;
    a.cnt = cnt;
    a.touched = cnt + far;
    a.acc = acc;
    a.count = head;
    a.next_chunk = (uint32_t *)(head + 2);
    a.layout_error = (uint32_t *)(head + 3);
    cudaEventRecord(ctx->ev[6], st);
    if (g.n) {
        void *params[] = {&a};
        BT_CUDA(cudaLaunchKernel(kfn, dim3((unsigned)nctas), dim3(kCountThreads), params, smem, st));
        bt_note_launches(1);
        if (per_edge && g.m) {
            const unsigned grid = (unsigned)std::min<uint64_t>((2 * g.m + 255) / 256, (uint64_t)ctx->sm_count * 8);
            if (wide) k_support<true><<<grid, 256, 0, st>>>(2 * g.m, acc, g.eid0, (unsigned long long *)ctx->sup, head + 1);
            else k_support<false><<<grid, 256, 0, st>>>(2 * g.m, acc, g.eid0, (unsigned long long *)ctx->sup, head + 1);
            bt_note_launches(1);
            BT_CUDA(cudaGetLastError());
        }
    }
    cudaEventRecord(ctx->ev[7], st);
    // one wait for the kernels, the results and the callers' end time: a staged
    // copy and a second wait cost a 20k-edge count 9 of its 51 us
    const uint64_t *h = ctx->host_words;
    BT_CUDA(cudaMemcpyAsync(ctx->host_words, head, 32, cudaMemcpyDeviceToHost, st));
    cudaEventRecord(ctx->ev[1], st);
    BT_CUDA(cudaStreamSynchronize(st));
    if ((uint32_t)h[3]) return bt_fail(BT_ERR_INVALID, "butterfly count: a wedge left its graph in the arena layout");
    ctx->zero_counters = far;
    float ms = -1;
    if (cudaEventElapsedTime(&ms, ctx->ev[6], ctx->ev[7]) == cudaSuccess) ctx->phase_ms[PH_EBFC] = ms;
    *count = h[0];
    if (per_edge) {
        ctx->last_sup_max = h[1];
        ctx->last_result = 1;
    }
    ctx->last_count = h[0];
    return BT_OK;
}

static const void *any_order_kernel() { return (const void *)k_count<false, false, true>; }

bt_status bt_count_any_order_setup() {
    BT_CUDA(cudaFuncSetAttribute(any_order_kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)count_smem(kDense)));
    return BT_OK;
}

bt_status bt_count_any_order(uint32_t n, uint32_t slots, const uint2 *rows, const uint32_t *nbr,
                             unsigned long long *count, uint32_t *next_chunk, uint32_t *skip, int sms, cudaStream_t st) {
    CountArgs a{};
    a.n = a.span = n;
    a.dense = dense_of(n);
    a.chunks = (n + kCountWarps - 1) / kCountWarps;
    a.batch = bt_count_batch(n - 1);  // degrees are below n
    a.least = 2;  // no row repeats a neighbour
    a.rows = rows;
    a.nbr = nbr;
    a.slots = slots;
    a.count = count;
    a.next_chunk = next_chunk;
    a.layout_error = skip;
    void *params[] = {&a};
    BT_CUDA(cudaLaunchKernel(any_order_kernel(), dim3(std::min<uint32_t>((uint32_t)sms, a.chunks)), dim3(kCountThreads),
                             params, count_smem(a.dense), st));
    bt_note_launches(1);
    return BT_OK;
}
