// bt_hidx.cu -- h-index bitruss iteration (the reference's "hidx").
//
// Same iteration as the reference (src/bitruss/bitruss_hidx.cu:51-168,
// 179-256; CPU src/bitruss/cpu_bitruss.cpp:152-266): starting from the
// butterfly supports, every round sets
//   h(uv) = h-index of { min(prev[ux], prev[wx], prev[wv]) : butterflies
//                        (u,v,w,x) of uv whose three other edges have prev > 0 }
// (0 when prev[uv] == 0), synchronously for all edges, until a round changes
// nothing.  The fixpoint is each edge's bitruss number.
//
// GB300 design: the reference gathers every min value of an edge into a
// per-block buffer of support_max entries and quicksorts it with one thread
// (bitruss_hidx.cu:111-157, with a 32-entry explicit stack).  Here no value
// list is stored: the h-index only needs counts.  Since h never rises above
// prev[uv], and rarely falls far in a round, one walk over the butterflies
// counts the values >= prev[uv] and bins those in the kBins below it; when
// there are at least prev[uv] of the former the edge is unchanged (the walk
// stops there), else the answer is the largest bin start with that many values
// at or above it.  An edge that falls further is walked again with wider bins
// over the rest, narrowed to one bin at a time.
//
// What bounds it: the butterflies visited, 4 per butterfly of the graph in a
// full round.  The values therefore lie where the walk reads: beside each row
// slot and in the row tables (neighbour -> value), so a position costs one
// coalesced read of (neighbour, value) and one table read, and mids and
// positions with values below the window cost no table read at all.  A round
// writes the changed values into both.  Small edges are a warp's, larger ones a
// CTA's, whose warps take equal parts of the positions.  With a CTA per edge,
// the anchor staged in shared memory and three values gathered per butterfly,
// the 44 rounds of a 50k-edge Chung-Lu graph took 156 ms, now 36; 28 rounds of a
// 50k-edge hub-skewed graph 628 ms, now 114.
//
// Active edges: a round only recomputes the edges that can change.  Values
// only fall, and h_k(e) = min(h_{k-1}(e), hindex(butterfly values of round
// k-1)), where a butterfly's value is the minimum of its three other edges.
// An edge keeps h = h_{k-1}(e) as long as at least h butterflies have a
// value >= h, so it can only change if some butterfly edge f fell, in round
// k-1, from a value >= h to one below h.  A butterfly of uv = (u, v) has edges
// ux, wv and wx with x a neighbour of u and w a neighbour of v, so f has an
// end in N[u] or N[v].  After each round every vertex z holds the lowest new
// value (lo) and the highest old value (hi) of the changed edges with an end
// in N[z]; edge (u, v) with value h is recomputed iff lo < h <= hi at u or at
// v.  The test never skips an edge that could change, so values, and the
// number of rounds, are those of the full synchronous iteration.
//
// Starting values.  The reference starts from the butterfly supports.  The
// iteration is monotone: started from any values s with b <= s <= supports,
// where b are the bitruss numbers (the largest fixpoint below the supports),
// every round keeps the values at or above b and they converge to the
// largest fixpoint below s, which is b.  So the result does not depend on
// the start, only the number of rounds does.  Graphs of up to 2^20 edges
// start from the supports (the reference's rounds); larger graphs start from
// the exact peel's values (bt_msp_exact, the bitruss numbers themselves),
// and the rounds then verify that those values are the fixpoint: one round
// that changes nothing.  BT_HIDX_START=support or =peel picks the start.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "bt_device.cuh"
#include "bt_internal.h"

namespace {

using bt::kEmpty;
using bt::load_vrec;
using bt::VRec;
constexpr uint32_t kBins = 256;
// Eight blocks of 256 per SM, at 32 registers: four took 38 ms where these take
// 36 (50k-edge Chung-Lu graph; 367 and 299 at 200k edges), blocks of 512 and
// 1,024 for the larger edges 45 and 56.
constexpr int kLightThreads = 256, kHeavyThreads = 256;
// An edge with at most this many row positions is one warp's: 128 rounds of 32
// (1,024 and 16,384 were 1-5% slower on four graphs).
constexpr float kLightPositions = 4096.0f;

// N32: every value is below 2^32 - 1 and no row repeats a neighbour; values lie
// beside the slots and in the tables.  Else 64-bit values, read through the edge
// ids in both places (the slots of parallel edges may share an edge id, and
// set_value finds one slot per pair of ends).
template <bool N32>
using Val = typename std::conditional<N32, uint32_t, unsigned long long>::type;

// Counts of a round, by round number mod 2.
struct RoundCtl {
    uint32_t light, heavy;            // edges recomputed: list[0, light) and the last `heavy` of list
    uint32_t next_light, next_heavy;  // work counters
    uint32_t changed;
};
struct HidxState {
    RoundCtl ctl[2];
    uint32_t marked_len, pool_used, overflow;
    unsigned long long recomputed;    // after round 1
};

struct HidxArgs {
    HidxState *s;
    uint32_t n;
    uint64_t m;
    const uint2 *ends;
    VRec *vrec;
    const uint32_t *nbr, *eid;
    uint4 *pool;      // row tables: neighbour -> value (N32) or edge id
    uint32_t *vs;     // N32: value of each slot's edge
    void *val;        // values of the last round, by edge id
    void *nval;       // this round's value of list[k], by k
    uint32_t *list;
};

template <bool N32>
__device__ __forceinline__ Val<N32> slot_value(const HidxArgs &a, uint32_t p) {
    if constexpr (N32) return a.vs[p];
    else return static_cast<const unsigned long long *>(a.val)[a.eid[p]];
}
template <bool N32>
__device__ __forceinline__ Val<N32> entry_value(const HidxArgs &a, uint32_t x) {
    if constexpr (N32) return x;
    else return static_cast<const unsigned long long *>(a.val)[x];
}

// One edge's walk: the pivot is the endpoint whose row has fewer positions.
struct EdgeWalk {
    uint32_t piv, anc, po, pd, ao, ad, at;
    float positions;
};
__device__ __forceinline__ EdgeWalk edge_walk(const HidxArgs &a, uint32_t e) {
    const uint2 uv = __ldg(a.ends + e);
    const VRec ru = load_vrec(a.vrec + uv.x), rv = load_vrec(a.vrec + uv.y);
    const bool pv = rv.hop <= ru.hop;
    const VRec &p = pv ? rv : ru, &q = pv ? ru : rv;
    return EdgeWalk{pv ? uv.y : uv.x, pv ? uv.x : uv.y, p.off, p.deg, q.off, q.deg, q.tab,
                    fminf((float)p.hop, (float)p.deg * (float)q.deg)};
}

// The values in [lo, hi) go to bins of `width`, those >= hi are counted.
template <bool N32>
struct Window {
    Val<N32> lo, hi, width;
};

// Walk task `task` (a block of 32 of the pivot's mids, or part task mod 2^lg of
// its positions) by one warp.
template <bool N32>
__device__ __forceinline__ void walk_task(const HidxArgs &a, const EdgeWalk &ew, uint32_t task, uint32_t lg,
                                          const Window<N32> &w, uint32_t *hist, uint32_t &above) {
    const uint32_t lane = threadIdx.x & 31;
    const Val<N32> least = w.lo ? w.lo : 1;  // values below the window say nothing, nor does 0
    const uint32_t k = (task >> lg) * 32 + lane, part = task & ((1u << lg) - 1);
    uint32_t row = 0, tab = 0, nb = 0, len = 0;
    Val<N32> vm = 0;
    if (k < ew.pd) {
        const uint32_t mid = __ldg(a.nbr + ew.po + k);
        vm = slot_value<N32>(a, ew.po + k);
        if (mid != ew.anc && vm >= least) {
            const VRec rm = load_vrec(a.vrec + mid);
            const bool rev = ew.ad < rm.deg;  // the shorter row is walked, the other's table looked up
            row = rev ? ew.ao : rm.off;
            tab = rev ? rm.tab : ew.at;
            nb = bt_row_buckets(rev ? rm.deg : ew.ad);
            len = rev ? ew.ad : rm.deg;
        }
    }
    uint32_t pre = bt::warp_inclusive(len);
    const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
    pre -= len;
    uint32_t f0 = 0, f1 = total;
    if (lg) {
        const uint32_t q = total >> lg, rem = total & ((1u << lg) - 1);
        f0 = q * part + (rem * part >> lg);
        f1 = q * (part + 1) + (rem * (part + 1) >> lg);
    }
    for (uint32_t fb = f0; fb < f1; fb += 32) {
        const uint32_t f = fb + lane;
        uint32_t m = 0;  // the last lane with pre <= f and a position of its own
#pragma unroll
        for (uint32_t o = 16; o; o >>= 1) {
            const uint32_t t = __shfl_sync(0xffffffffu, pre, m + o);
            if (t <= f) m += o;
        }
        const uint32_t p = __shfl_sync(0xffffffffu, row, m) + (f - __shfl_sync(0xffffffffu, pre, m));
        const uint32_t mtab = __shfl_sync(0xffffffffu, tab, m), mnb = __shfl_sync(0xffffffffu, nb, m);
        const Val<N32> mv = __shfl_sync(0xffffffffu, vm, m);
        if (f >= f1) continue;
        const uint32_t y = __ldg(a.nbr + p);
        Val<N32> v = slot_value<N32>(a, p);
        if (y == ew.piv || v < least) continue;
        const uint32_t x = bt::row_find(a.pool, mtab, mnb, y);
        if (x == kEmpty) continue;
        v = min(min(v, mv), entry_value<N32>(a, x));
        if (v >= w.hi) above++;
        else if (v >= least) atomicAdd(hist + (w.width == 1 ? (uint32_t)(v - w.lo) : (uint32_t)((v - w.lo) / w.width)), 1u);
    }
}

// The largest bin whose start x has at least x values at or above it (`above`
// of them past the window), by one warp, which clears the bins; false: none.
template <bool N32>
__device__ __forceinline__ bool pick_bin(uint32_t *hist, const Window<N32> &w, unsigned long long above, Val<N32> &x) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t bins = (uint32_t)(((unsigned long long)(w.hi - w.lo) + w.width - 1) / w.width);
    bool found = false;
    for (uint32_t top = (bins + 31) & ~31u; top; top -= 32) {
        const uint32_t b = top - 1 - lane;
        const uint32_t c = b < bins ? hist[b] : 0;
        if (b < bins) hist[b] = 0;
        if (found) continue;
        const uint32_t inc = bt::warp_inclusive(c);
        const unsigned long long start = (unsigned long long)w.lo + (unsigned long long)b * w.width;
        const uint32_t ok = __ballot_sync(0xffffffffu, b < bins && above + inc >= start);
        if (ok) {
            found = true;
            const uint32_t q = top - __ffs(ok);  // the lowest such lane has the largest start
            x = w.lo + (Val<N32>)q * w.width;
        }
        above += __shfl_sync(0xffffffffu, inc, 31);
    }
    __syncwarp();
    return found;
}

// After a window: true when h is known, else `w` is the next window.
template <bool N32>
__device__ __forceinline__ bool next_window(bool found, Val<N32> x, Window<N32> &w, Val<N32> &h) {
    if (found) {
        const Val<N32> end = w.hi - x > w.width ? x + w.width : w.hi;
        if (end - x == 1) {
            h = x;
            return true;
        }
        w.lo = x;
        w.hi = end;
    } else {  // below the window (at 0 every count is enough)
        w.hi = w.lo;
        w.lo = 0;
    }
    w.width = (w.hi - w.lo + kBins - 1) / kBins;
    return false;
}

template <bool N32>
__device__ __forceinline__ Window<N32> first_window(Val<N32> H) {
    return Window<N32>{H > kBins ? H - (Val<N32>)kBins : (Val<N32>)0, H, 1};
}

// Edges of few positions: one warp each.
template <bool N32>
__global__ void __launch_bounds__(kLightThreads, 8) k_hidx_light(HidxArgs a, uint32_t parity) {
    __shared__ uint32_t s_hist[kLightThreads / 32][kBins];
    const uint32_t lane = threadIdx.x & 31;
    uint32_t *hist = s_hist[threadIdx.x >> 5];
    for (uint32_t k = lane; k < kBins; k += 32) hist[k] = 0;
    __syncwarp();
    RoundCtl &ctl = a.s->ctl[parity];
    const uint32_t count = ctl.light;
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(&ctl.next_light, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= count) break;
        const uint32_t e = a.list[i];
        const Val<N32> H = static_cast<const Val<N32> *>(a.val)[e];
        const EdgeWalk ew = edge_walk(a, e);
        const uint32_t blocks = (ew.pd + 31) / 32;
        Window<N32> w = first_window<N32>(H);
        Val<N32> h = H;
        for (bool first = true;; first = false) {
            uint32_t above = 0, sum = 0;
            for (uint32_t t = 0; t < blocks; t++) {
                walk_task<N32>(a, ew, t, 0, w, hist, above);
                if (first && (sum = __reduce_add_sync(0xffffffffu, above)) >= H) break;
            }
            __syncwarp();
            sum = __reduce_add_sync(0xffffffffu, above);
            Val<N32> x = 0;
            const bool found = pick_bin<N32>(hist, w, sum, x);
            if (first && sum >= H) break;  // unchanged
            if (next_window<N32>(found, x, w, h)) break;
        }
        if (lane == 0) {
            static_cast<Val<N32> *>(a.nval)[i] = h;
            if (h != H) ctl.changed = 1;
        }
    }
}

// Edges of many positions: one CTA each.
template <bool N32>
__global__ void __launch_bounds__(kHeavyThreads, 8) k_hidx_heavy(HidxArgs a, uint32_t parity, bool first_round) {
    __shared__ uint32_t hist[kBins];
    __shared__ unsigned long long s_above;
    __shared__ uint32_t s_i, s_done;
    __shared__ Window<N32> s_w;
    __shared__ Val<N32> s_h;
    constexpr uint32_t kWarps = kHeavyThreads / 32;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t k = threadIdx.x; k < kBins; k += kHeavyThreads) hist[k] = 0;
    RoundCtl &ctl = a.s->ctl[parity];
    const uint32_t count = ctl.heavy;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // this kernel is the round's first: the next round's counts start at zero
        a.s->ctl[parity ^ 1] = RoundCtl{0, 0, 0, 0, 0};
        a.s->marked_len = 0;
        if (!first_round) a.s->recomputed += (unsigned long long)ctl.light + count;
    }
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s_i = atomicAdd(&ctl.next_heavy, 1u);
            s_above = 0;
            s_done = 0;
        }
        __syncthreads();
        const uint32_t i = s_i;
        if (i >= count) break;
        const uint64_t at = a.m - 1 - i;
        const uint32_t e = a.list[at];
        const Val<N32> H = static_cast<const Val<N32> *>(a.val)[e];
        const EdgeWalk ew = edge_walk(a, e);
        // two tasks per warp at least
        const uint32_t blocks = (ew.pd + 31) / 32;
        const uint32_t lg = blocks >= 2 * kWarps ? 0 : 32 - __clz((2 * kWarps - 1) / blocks);
        Window<N32> w = first_window<N32>(H);
        Val<N32> h = H;
        for (bool first = true;; first = false) {
            for (uint32_t t = warp; t < (blocks << lg); t += kWarps) {
                uint32_t above = 0;
                walk_task<N32>(a, ew, t, lg, w, hist, above);
                above = __reduce_add_sync(0xffffffffu, above);
                unsigned long long so_far = 0;
                if (lane == 0) so_far = atomicAdd(&s_above, (unsigned long long)above) + above;
                // H values >= H: the edge keeps H whatever the rest
                if (first && __shfl_sync(0xffffffffu, so_far, 0) >= H) break;
            }
            __syncthreads();
            if (warp == 0) {
                const unsigned long long above = s_above;
                Val<N32> x = 0;
                const bool found = pick_bin<N32>(hist, w, above, x);
                const bool done = (first && above >= H) || next_window<N32>(found, x, w, h);
                if (lane == 0) {
                    s_done = done;
                    s_w = w;
                    s_h = h;
                    s_above = 0;
                }
            }
            __syncthreads();
            if (s_done) break;
            w = s_w;
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            static_cast<Val<N32> *>(a.nval)[at] = s_h;
            if (s_h != H) ctl.changed = 1;
        }
    }
}

// Vertex records, row tables and slot values (as in the peel's set-up: a block
// lays out its tables, then its warps build them).
template <bool N32>
__global__ void __launch_bounds__(256) k_hidx_rows(HidxArgs a, const uint32_t *off, const uint32_t *deg) {
    __shared__ uint32_t base, s_tab[256];
    __shared__ typename cub::BlockScan<uint32_t, 256>::TempStorage scan;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t step = gridDim.x;
    for (uint64_t x0 = blockIdx.x; x0 < a.n; x0 += step * 256) {
        const uint64_t x = x0 + step * threadIdx.x;
        const uint32_t d = x < a.n ? deg[x] : 0;
        uint32_t excl, tot;
        cub::BlockScan<uint32_t, 256>(scan).ExclusiveSum(d ? bt_row_buckets(d) : 0, excl, tot);
        if (threadIdx.x == 0) base = atomicAdd(&a.s->pool_used, tot);
        __syncthreads();
        s_tab[threadIdx.x] = base + excl;
        __syncthreads();
        for (uint32_t k = threadIdx.x >> 5; k < 256 && x0 + step * k < a.n; k += 8) {
            const uint32_t y = (uint32_t)(x0 + step * k), dy = deg[y], oy = off[y];
            unsigned long long hop = 0;
            for (uint32_t j = lane; j < dy; j += 32) {
                hop += __ldg(deg + a.nbr[oy + j]);
                if constexpr (N32) a.vs[oy + j] = static_cast<const uint32_t *>(a.val)[a.eid[oy + j]];
            }
            hop = bt::warp_sum(hop);
            if (lane == 0) a.vrec[y] = VRec{oy, dy, s_tab[k], hop > 0xffffffffull ? 0xffffffffu : (uint32_t)hop};
            __syncwarp();
            if (dy)
                bt::row_build<true>(a.pool, s_tab[k], dy, a.nbr + oy, [&](uint32_t j) {
                    if constexpr (N32) return a.vs[oy + j];
                    else return a.eid[oy + j];
                });
        }
        __syncthreads();
    }
}

// A changed value in x's row: beside its slot and in the row's table.
__device__ __forceinline__ void set_value(const HidxArgs &a, uint32_t x, uint32_t y, uint32_t v) {
    const VRec r = load_vrec(a.vrec + x);
    uint32_t lo = 0, hi = r.deg;
    while (lo < hi) {
        const uint32_t md = (lo + hi) >> 1;
        if (__ldg(a.nbr + r.off + md) < y) lo = md + 1;
        else hi = md;
    }
    if (lo < r.deg) a.vs[r.off + lo] = v;
    const size_t at = bt::row_entry(a.pool, r.tab, bt_row_buckets(r.deg), y);
    if (at != ~(size_t)0) reinterpret_cast<uint2 *>(a.pool)[at].y = v;
}

// Apply a round: every recomputed edge whose value changed takes the new value;
// its endpoints record the lowest new and the highest old value of their
// changed edges and are listed once (stamp r).
template <bool N32>
__global__ void k_hidx_apply(HidxArgs a, uint32_t parity, uint32_t r, uint32_t *mark, uint32_t *marked,
                             unsigned long long *vlo, unsigned long long *vhi) {
    const uint64_t light = a.s->ctl[parity].light, len = light + a.s->ctl[parity].heavy;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < len;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = k < light ? k : a.m - 1 - (k - light);
        const uint32_t e = a.list[i];
        Val<N32> *val = static_cast<Val<N32> *>(a.val);
        const Val<N32> b = static_cast<const Val<N32> *>(a.nval)[i], old = val[e];
        if (b == old) continue;
        val[e] = b;
        const uint2 uv = a.ends[e];
        if constexpr (N32) {
            set_value(a, uv.x, uv.y, b);
            set_value(a, uv.y, uv.x, b);
        }
        atomicMin(&vlo[uv.x], (unsigned long long)b);
        atomicMax(&vhi[uv.x], (unsigned long long)old);
        atomicMin(&vlo[uv.y], (unsigned long long)b);
        atomicMax(&vhi[uv.y], (unsigned long long)old);
        if (atomicExch(&mark[uv.x], r) != r) marked[atomicAdd(&a.s->marked_len, 1u)] = uv.x;
        if (atomicExch(&mark[uv.y], r) != r) marked[atomicAdd(&a.s->marked_len, 1u)] = uv.y;
    }
}

// Spread each listed vertex's (lo, hi) to itself and its neighbours (one
// warp per listed vertex).
__global__ void k_hidx_near(HidxArgs a, const uint32_t *marked, const unsigned long long *vlo,
                            const unsigned long long *vhi, unsigned long long *nlo, unsigned long long *nhi) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t len = a.s->marked_len;
    for (uint32_t i = warp; i < len; i += nw) {
        const uint32_t z = marked[i];
        const unsigned long long lo = vlo[z], hi = vhi[z];
        const VRec rz = load_vrec(a.vrec + z);
        if (lane == 0) {
            atomicMin(&nlo[z], lo);
            atomicMax(&nhi[z], hi);
        }
        for (uint32_t j = lane; j < rz.deg; j += 32) {
            const uint32_t y = a.nbr[rz.off + j];
            atomicMin(&nlo[y], lo);
            atomicMax(&nhi[y], hi);
        }
    }
}

// List the edges the next round recomputes -- value h > 0 with lo < h <= hi at
// one of its ends, or every edge with h > 0 (`all`) -- small ones from the
// front, large ones from the back.
template <bool N32>
__global__ void __launch_bounds__(256) k_hidx_list(HidxArgs a, uint32_t parity, bool all,
                                                   const unsigned long long *nlo, const unsigned long long *nhi) {
    const uint32_t lane = threadIdx.x & 31;
    RoundCtl &ctl = a.s->ctl[parity];
    for (uint64_t e0 = blockIdx.x * 256ull; e0 < a.m; e0 += gridDim.x * 256ull) {
        const uint64_t e = e0 + threadIdx.x;
        bool f = false, large = false;
        if (e < a.m) {
            const unsigned long long h = static_cast<const Val<N32> *>(a.val)[e];
            if (h > 0) {
                const uint2 uv = a.ends[e];
                f = all || (nlo[uv.x] < h && h <= nhi[uv.x]) || (nlo[uv.y] < h && h <= nhi[uv.y]);
                if (f) large = edge_walk(a, (uint32_t)e).positions > kLightPositions;
            }
        }
        const uint32_t bl = __ballot_sync(0xffffffffu, f && !large), bh = __ballot_sync(0xffffffffu, f && large);
        uint32_t at = 0;
        if (lane == 0 && bl) at = atomicAdd(&ctl.light, (uint32_t)__popc(bl));
        if (lane == 1 && bh) at = atomicAdd(&ctl.heavy, (uint32_t)__popc(bh));
        const uint32_t al = __shfl_sync(0xffffffffu, at, 0), ah = __shfl_sync(0xffffffffu, at, 1);
        const uint32_t below = (1u << lane) - 1;
        if (f && !large) a.list[al + __popc(bl & below)] = (uint32_t)e;
        if (f && large) a.list[a.m - 1 - (ah + __popc(bh & below))] = (uint32_t)e;
    }
}

// Starting values: supports, or a uint32 result (the exact peel).
template <bool N32>
__global__ void k_hidx_start(uint64_t m, const unsigned long long *sup, const uint32_t *result, Val<N32> *v) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m;
         e += (uint64_t)gridDim.x * blockDim.x)
        v[e] = sup ? (Val<N32>)sup[e] : (Val<N32>)result[e];
}

template <bool N32>
__global__ void k_hidx_result(HidxArgs a, uint32_t *out) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < a.m;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const Val<N32> v = static_cast<const Val<N32> *>(a.val)[e];
        if (v > 0xffffffffull) atomicExch(&a.s->overflow, 1u);
        out[e] = (uint32_t)v;
    }
}

}  // namespace

// Start of the iteration: true = the exact peel's values, false = supports.
static bool hidx_from_peel(uint64_t m) {
    const char *v = getenv("BT_HIDX_START");
    if (v && !strcmp(v, "peel")) return true;
    if (v && !strcmp(v, "support")) return false;
    return m > (1ull << 20);
}

template <bool N32>
static bt_status run_hidx(bt_ctx *ctx, bool from_peel, uint32_t *rounds) {
    DevGraph &g = ctx->g;
    cudaStream_t st = ctx->stream;
    const uint64_t m = g.m, n = g.n;
    const uint64_t mm = m ? m : 1, nn = n ? n : 1;
    cudaEvent_t e0 = ctx->ev[2], e1 = ctx->ev[3];
    cudaEventRecord(e0, st);
    HidxArgs a{};
    uint32_t *mark = nullptr, *marked = nullptr;
    unsigned long long *vlo = nullptr, *vhi = nullptr, *nlo = nullptr, *nhi = nullptr;
    auto release = [&]() {
        for (void *p : {(void *)a.s, (void *)a.vrec, (void *)a.pool, (void *)a.vs, a.val, a.nval, (void *)a.list,
                        (void *)mark, (void *)marked, (void *)vlo, (void *)vhi, (void *)nlo, (void *)nhi})
            ctx_free(ctx, p);
    };
    bt_status rc;
    if ((rc = ctx_alloc(ctx, (void **)&a.s, sizeof(HidxState))) != BT_OK ||
        (rc = ctx_alloc_t(ctx, &a.vrec, nn)) != BT_OK ||
        (rc = ctx_alloc(ctx, (void **)&a.pool, 32 * (g.tab_buckets ? g.tab_buckets : 1))) != BT_OK ||
        (N32 && (rc = ctx_alloc_t(ctx, &a.vs, 2 * mm)) != BT_OK) ||
        (rc = ctx_alloc(ctx, &a.val, sizeof(Val<N32>) * mm)) != BT_OK ||
        (rc = ctx_alloc(ctx, &a.nval, sizeof(Val<N32>) * mm)) != BT_OK ||
        (rc = ctx_alloc_t(ctx, &a.list, mm)) != BT_OK || (rc = ctx_alloc_t(ctx, &mark, nn)) != BT_OK ||
        (rc = ctx_alloc_t(ctx, &marked, nn)) != BT_OK || (rc = ctx_alloc_t(ctx, &vlo, nn)) != BT_OK ||
        (rc = ctx_alloc_t(ctx, &vhi, nn)) != BT_OK || (rc = ctx_alloc_t(ctx, &nlo, nn)) != BT_OK ||
        (rc = ctx_alloc_t(ctx, &nhi, nn)) != BT_OK) {
        release();
        return rc;
    }
#define C(x)                                                                  \
    do {                                                                      \
        cudaError_t _e = (x);                                                 \
        if (_e != cudaSuccess) { release(); return bt_cuda_fail(_e, #x, __FILE__, __LINE__); } \
    } while (0)
    a.n = g.n;
    a.m = m;
    a.ends = g.ends;
    a.nbr = g.nbr0;
    a.eid = g.eid0;
    C(cudaMemsetAsync(a.s, 0, sizeof(HidxState), st));
    C(cudaMemsetAsync(mark, 0, 4 * nn, st));
    const unsigned blk = 256, cap = (unsigned)ctx->sm_count * 8;
    const unsigned egrid = (unsigned)std::min<uint64_t>((mm + blk - 1) / blk, cap);
    int light_per_sm = 0, heavy_per_sm = 0;
    C(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&light_per_sm, k_hidx_light<N32>, kLightThreads, 0));
    C(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&heavy_per_sm, k_hidx_heavy<N32>, kHeavyThreads, 0));
    const unsigned light_grid = (unsigned)(ctx->sm_count * std::max(light_per_sm, 1));
    const unsigned heavy_grid = (unsigned)(ctx->sm_count * std::max(heavy_per_sm, 1));
    if (m) {
        k_hidx_start<N32><<<egrid, blk, 0, st>>>(m, from_peel ? nullptr : (const unsigned long long *)ctx->sup,
                                                ctx->result, (Val<N32> *)a.val);
        k_hidx_rows<N32><<<(unsigned)std::min<uint64_t>((n * 32 + blk - 1) / blk, cap), blk, 0, st>>>(a, g.off, g.deg0);
        k_hidx_list<N32><<<egrid, blk, 0, st>>>(a, 1, true, nullptr, nullptr);  // round 1
        bt_note_launches(3);
        C(cudaGetLastError());
    }
    uint32_t r = 0;
    for (;;) {
        r++;
        const uint32_t parity = r & 1;
        uint32_t changed = 0;
        if (m) {
            // the round, its values applied, the next round's edges listed
            // (nothing to apply or list when nothing changed)
            C(cudaMemsetAsync(vlo, 0xff, 8 * nn, st));
            C(cudaMemsetAsync(vhi, 0, 8 * nn, st));
            C(cudaMemsetAsync(nlo, 0xff, 8 * nn, st));
            C(cudaMemsetAsync(nhi, 0, 8 * nn, st));
            k_hidx_heavy<N32><<<heavy_grid, kHeavyThreads, 0, st>>>(a, parity, r == 1);
            k_hidx_light<N32><<<light_grid, kLightThreads, 0, st>>>(a, parity);
            k_hidx_apply<N32><<<egrid, blk, 0, st>>>(a, parity, r, mark, marked, vlo, vhi);
            k_hidx_near<<<cap, blk, 0, st>>>(a, marked, vlo, vhi, nlo, nhi);
            k_hidx_list<N32><<<egrid, blk, 0, st>>>(a, parity ^ 1, false, nlo, nhi);
            bt_note_launches(5);
            C(cudaGetLastError());
            C(cudaMemcpyAsync(&changed, &a.s->ctl[parity].changed, 4, cudaMemcpyDeviceToHost, st));
            C(cudaStreamSynchronize(st));
        }
        if (!changed) break;
    }
    HidxState h{};
    if (m) {
        k_hidx_result<N32><<<egrid, blk, 0, st>>>(a, ctx->result); bt_note_launches(1);
        C(cudaGetLastError());
    }
    C(cudaMemcpyAsync(&h, a.s, sizeof(h), cudaMemcpyDeviceToHost, st));
    cudaEventRecord(e1, st);
    C(cudaStreamSynchronize(st));
#undef C
    float ms = -1;
    cudaEventElapsedTime(&ms, e0, e1);
    ctx->phase_ms[PH_HIDX] = ms;
    release();
    if (h.overflow) return bt_fail(BT_ERR_OVERFLOW, "hidx: a bitruss number exceeds uint32");
    ctx->stats[4] = r;
    ctx->work[10] = m + h.recomputed;  // edge recomputations over all rounds; the first is of every edge
    ctx->work[11] = from_peel ? 1 : 0;
    ctx->last_result = 2;
    if (rounds) *rounds = r;
    return BT_OK;
}

bt_status dev_hidx(bt_ctx *ctx, uint32_t *rounds) {
    const bool from_peel = hidx_from_peel(ctx->g.m);
    if (from_peel) {
        uint32_t lv = 0;
        BT_TRY(dev_msp(ctx, true, &lv));  // ctx->result = the exact peel's values
    } else {
        uint64_t dummy = 0;
        BT_TRY(dev_ebfc(ctx, true, &dummy));
    }
    // no value exceeds the largest support (BT_MSP_WIDE=1: as in the peel)
    const char *wide = getenv("BT_MSP_WIDE");
    if (ctx->last_sup_max < 0xffffffffull && !ctx->g.repeats && !(wide && *wide == '1')) return run_hidx<true>(ctx, from_peel, rounds);
    return run_hidx<false>(ctx, from_peel, rounds);
}
