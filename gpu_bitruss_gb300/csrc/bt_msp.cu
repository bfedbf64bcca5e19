// bt_msp.cu -- multi-stage bitruss peeling (GBiD, the reference's "msp").
//
// Semantics (bit-exact with the reference, src/bitruss/bitruss_msp.cu:440-583
// and src/bitruss/cpu_bitruss.cpp:563-624):
//  * edges with support 0 are processed first (count_es_zero, :38-65);
//  * level L: the frontier is every unprocessed edge with support == L
//    (scan_sub_kernel, :77-93); levels with an empty frontier change nothing
//    and are skipped here;
//  * a sub-round peels the whole frontier: for each frontier edge uv and each
//    butterfly (u,v,w,x) whose three other edges wv, wx, ux are unprocessed,
//    the peel rule (peel_one/two/three_edge, :126-184) decides which of them
//    lose one support; a decrement that takes an edge from L+1 to L puts it
//    in the next frontier and supports are clamped at L (update_edge_support,
//    :110-123);
//  * the frontier is then marked processed and the next frontier becomes the
//    frontier of a new sub-round at the same level (:516-534);
//  * the result is each edge's support when it was processed, i.e. the level
//    at which it joined a frontier.
// The order of decrements inside a sub-round does not change the result, so
// the GPU may apply them in any order and aggregate them.
//
// GB300 design: one cooperative persistent kernel runs the whole level /
// sub-round loop on the device (the reference pays 3 host syncs and ~9m bytes
// of copies per sub-round, :527-533).  One graph has the whole grid; the graphs
// of a batched arena are peeled side by side, each by a team of CTAs with its
// own barrier, lists and levels ("grid" below is the team's).
//
// What bounds it: the chain.  A decomposition is tens of thousands of
// sub-rounds that depend on one another, most of them of 10^3 to 10^5 row
// positions, so a sub-round's time is the number of dependent L2 round trips
// (430 cycles each) and barriers on its longest path, not bandwidth.  Measured
// per sub-round, against staging the anchor row in shared memory and walking
// equal shares of probe positions by whole CTAs: Chung-Lu graphs of 10k / 200k
// / 1M edges 6.6 / 8.1 / 10.8 us (19.4 / 21.8 / 28.7 before), the 20M-edge one
// 46 us (87), hub-skewed graphs of 200k / 2M edges 12.4 / 32 us (28.5 / 49).
// What follows from that:
//  * Edge state is one stamp per edge: enter[e] = the index of the sub-round
//    whose frontier e joined (0: not yet).  In sub-round r an edge is in the
//    frontier iff enter == r and processed iff 0 < enter < r, so "mark the
//    frontier processed, promote the next frontier" costs nothing: the thread
//    that pushes an edge to the next frontier stamps it r+1 and records its
//    result (L).  A sub-round therefore needs one grid barrier.
//  * Every row has a hash table (neighbour -> edge id) over its live edges,
//    rebuilt at each row compaction, so a (mid, anchor) pair is intersected
//    from its shorter row with one table read per position and nothing has to
//    be staged first.
//  * A frontier of up to 32 edges is planned inside the barrier: its entries
//    are loaded with the control words, whoever pushed them having written
//    their endpoints beside them.  Up to 512 edges every CTA plans the whole
//    frontier; more than that are cut into chunks that CTAs take from a
//    counter.
//  * A task is a warp on a block of 32 pivot slots (mids), one per lane, or on
//    an equal part of the block's positions; the positions of the block's live
//    mids lie end to end and are taken 32 at a time, so lanes stay full
//    whatever the rows' lengths.  Tasks are dealt to the CTAs round robin and
//    taken by their warps one by one.  No block barriers.
//  * Only one warp per CTA reads what all of them need (control words, the
//    frontier): the same word read by every warp of the grid at once is served
//    one request at a time and costs more than the rest of the plan.
//  * Frontier discovery uses two support buckets: "near" holds the live
//    edges with support < hi, "far" the rest.  A level scans only the near
//    list; when it runs dry the far list is split again.  A decrement that
//    crosses hi appends the edge to near.  The next level is known before the
//    scan: every support that is written or scanned above the level takes part
//    in a running minimum (see Control::cand), so a level costs one scan and
//    one barrier.
//  * Processed edges are dropped from the rows (device-side compaction)
//    whenever the live edges have halved (the reference's trigger, :537-549,
//    without its floor at a tenth of the edges); compaction only changes
//    work, not results.
// 512 threads a CTA: with 1,024 (64 registers) the lone sub-rounds took 20%
// longer and only hub rows of 500k edges and more gained (3%).
// Grid barriers are bounded by a time limit; an expired wait sets an error and
// the kernel returns.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <condition_variable>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "bt_device.cuh"
#include "bt_internal.h"

namespace {

using bt::kEmpty;
using bt::load_vrec;
using bt::VRec;
using bt::warp_inclusive;
using bt::warp_sum;
constexpr int kThreads = 512;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kEdges = kMspLocalPlan;  // frontier edges a CTA plans at once

// What every CTA reads after a barrier, in one warp-wide load (barrier()).
//
// A CTA that leaves a barrier first goes on while others have yet to load these
// words.  So no word that a CTA uses after barrier b may be written between b
// and the barrier after it.  For each word, who writes it, and the barrier
// (S: a level's scan, P: a sub-round, F1 / F2: the two of a far split) after
// which it is used:
//  * len[r % 3]: appended to by sub-round r - 1 only, used after its P; zeroed in
//    sub-round r + 1.
//  * scan_len[k % 3]: appended to by the scan of level number k only, used after
//    that S (and after the barriers of a row compaction behind it); zeroed at the
//    scan of number k + 2.  It is not len: a CTA that finds len at 0 after a P goes
//    straight to the scan, as a slower one must, which reads the same len.
//  * cand[k % 3]: lowered at the S of level number k and at its P's, used when that
//    level has run out: after its last P, or S if it was empty; reset at the
//    scan of number k + 2.
//  * near_ctr[nsel]: appended to by sub-rounds, used at a scan, after the last P,
//    F2 or S.  near_ctr[nsel ^ 1]: appended to between F1 and F2 or by a scan that
//    compacts, used after that F2 or S as the new near_ctr[nsel]; the one left is
//    zeroed behind the same barrier and next appended to behind another (near_dead
//    is 0 there, so a scan that follows at once does not compact).
//  * far_len, far2_len, far_min, delta: far2_len is appended to and far_min
//    lowered before F2 and F1, and used after them; all four are set behind
//    F2 and next used after the S that follows at the earliest.
struct Control {
    unsigned long long delta;      // width of the near bucket
    unsigned long long far_min;
    // cand[k % 3]: a lower bound of the supports that are live above level
    // number k, collected while that level is scanned and peeled
    unsigned long long cand[3];
    uint32_t len[3];               // lengths of the frontiers that sub-rounds find, by index mod 3
    uint32_t scan_len[3];          // of those that levels' scans find, by level number mod 3
    uint32_t near_ctr[2];          // near bucket lengths (selector kept by every CTA)
    uint32_t far_len, far2_len;
};
constexpr uint32_t kControlWords = sizeof(Control) / 4;
static_assert(kControlWords <= 32, "the control words are loaded by one warp");

// The state of one graph's peel (zero but for far_len when the kernel starts; the
// team that takes it sets the rest).
struct MspState {
    __align__(128) Control ctl;
    // the first entries of the two frontier lists as (edge, U end, V end, 0):
    // what a short frontier's plan needs, written by whoever appends
    uint4 head[2][32];
    uint32_t task_ctr[3];          // chunk counters by sub-round index mod 3
};

// A graph of the arena: its ranks [v0, v1) and edges [e0, e0 + m).
struct Job {
    uint32_t v0, v1, e0, m;
};

// CTAs [cta0, cta0 + size) that peel one graph after another.
struct __align__(128) TeamState {
    bt::Barrier bar;
    uint32_t job, cta0, size;
};

// Of the whole launch.
struct MspShared {
    uint32_t queue;                // jobs given out past the teams' first ones
    uint32_t pool_used;            // row table buckets given out
    uint32_t done, overflow, error;
    unsigned long long last_level; // the largest last level with a non-empty frontier
    unsigned long long ph_ns[2];   // the first team's time in: level transitions, sub-rounds
    unsigned long long prof[8];    // SM cycles summed over CTAs, by step (PF_*)
    // statistics
    unsigned long long subrounds, compressions, tasks, levels_seen, rebuilds;
    // work counters (algorithmic bytes): row positions walked, anchor slots of
    // the peeled edges, butterflies found, decrements
    unsigned long long w_probes, w_anchor, w_hits, w_decs;
};

// A CTA's place in its team, and the graph the team is on.
struct Team {
    uint32_t rank, size;
    bt::Barrier *bar;
    MspState *s;
    Job job;
    __device__ __forceinline__ uint32_t thread() const { return rank * kThreads + threadIdx.x; }
    __device__ __forceinline__ uint32_t threads() const { return size * kThreads; }
};

// Optional per-sub-round trace (BT_MSP_TRACE=<path>): what bounds a sub-round.
struct TraceRow {
    unsigned long long t_ns;        // sub-round duration seen by CTA 0 (plan to barrier exit)
    unsigned long long max_task_ns; // longest CTA
    unsigned long long walked;      // row positions walked
    uint32_t frontier, tasks;
};

struct MspArgs {
    MspShared *sh;
    TeamState *teams;
    MspState *states;               // per job
    const Job *jobs;                // longest first
    uint32_t njobs, nteams;
    const uint32_t *team_of;        // per CTA
    uint32_t n, exact;
    uint32_t chunks_per_cta, local_plan;  // schedule, with inv_task (results do not depend on it)
    // row compaction trigger: compact when the live edges fall to cfrac of
    // the live edges at the last compaction, while those were at least
    // cfloor * m (compaction changes work, never results)
    float cfrac, cfloor;
    float inv_task;                 // 1 / positions of a task
    uint64_t m;
    unsigned long long wait_ns;
    uint32_t late_ns;               // see linger()
    const uint2 *ends;
    VRec *vrec;
    uint32_t *nbr, *eid;            // live rows (compacted in place)
    uint4 *pool;                    // row tables (bt::row_resolve)
    unsigned long long *sup;        // working supports (64-bit)
    uint32_t *sup32;                // working supports when every support fits 32 bits (else null)
    uint32_t *enter;                // sub-round index at which the edge joined a frontier
    uint32_t *result;               // bitruss number per edge
    uint32_t *list0, *list1;        // frontier lists by sub-round index mod 2
    uint32_t *near_a, *near_b, *far_a, *far_b;
    TraceRow *trace;                // optional, trace_cap rows
    uint32_t trace_cap;
};

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t next3(uint32_t i) { return i == 2 ? 0 : i + 1; }

__device__ __forceinline__ bool is_done(uint32_t en, uint32_t r) { return en != 0 && en < r; }

__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) {
    for (int o = 16; o; o >>= 1) {
        unsigned long long t = __shfl_xor_sync(0xffffffffu, v, o);
        v = t < v ? t : v;
    }
    return v;
}

// The peel rule for one butterfly seen from frontier edge uv; returns a 3-bit
// mask of the edges to decrement: bit0 wv, bit1 wx, bit2 ux.  An edge that is
// in the frontier itself (c..) is never decremented, and the frontier edges of
// the butterfly share the work by their ids:
//  * none besides uv: all three lose one (peel_three_edge, bitruss_msp.cu:178-184);
//  * one besides uv: the smaller of the two decrements (peel_two_edge, :148-175);
//  * two besides uv (peel_one_edge, :126-145): exact: the smallest of the three
//    decrements the survivor.  Reference: with the survivor wv, wx or ux, uv
//    decrements it only if uv < ux < wx, uv < ux < wv or uv < wv < wx.
// So uv decrements when its id is below every other frontier edge's, and the
// reference's rule asks for the order of the other two as well.  Written
// without branches: lanes of a warp disagree about the case.
__device__ __forceinline__ uint32_t peel_rule(uint32_t uv, uint32_t wv, uint32_t wx, uint32_t ux, bool cwv,
                                              bool cwx, bool cux, uint32_t exact) {
    const uint32_t live = (cwv ? 0u : 1u) | (cwx ? 0u : 2u) | (cux ? 0u : 4u);
    const bool first = (!cwv | (uv < wv)) & (!cwx | (uv < wx)) & (!cux | (uv < ux));
    const bool chain = (live == 2 & (ux < wv)) | (live == 1 & (ux < wx)) | (live == 4 & (wv < wx));
    const bool one = live == 1 | live == 2 | live == 4;
    return first & (!one | (exact != 0) | chain) ? live : 0u;
}

// The kernel is compiled twice: N32 = every working support is below 2^32 - 1
// (4-byte supports, levels and atomics), else 64-bit supports.
template <bool N32>
using SupWord = typename std::conditional<N32, uint32_t, unsigned long long>::type;

// One sub-round's view of the state.
template <bool N32>
struct Round {
    uint32_t r;                     // sub-round index
    SupWord<N32> L, hi;             // level and near-bucket bound
    uint32_t *next, *next_len;      // next frontier
    uint4 *next_head;
    uint32_t *near_list, *near_len;
};

template <bool N32>
__device__ __forceinline__ SupWord<N32> sup_of(const MspArgs &a, uint32_t e) {
    if constexpr (N32) return __ldcg(a.sup32 + e);
    else return __ldcg(a.sup + e);
}

// Subtract k from sup[e].  The decrement that takes it from above L to L or
// below puts e in the next frontier (stamp r+1, result L): the reference's
// clamp at L (update_edge_support, bitruss_msp.cu:110-123) then only matters
// for the value it is processed with, which is L.  A decrement crossing hi
// appends e to the near bucket.
// A decrement is split in two so that a thread can have several in flight:
// dec_issue sends the atomic and returns the old support (nothing waits for
// it until the value is used), dec_settle acts on the crossings it shows.
template <bool N32>
__device__ __forceinline__ SupWord<N32> dec_issue(const MspArgs &a, uint32_t e, uint32_t k) {
    // supports never fall below 0: a decrement reaches an edge only while it is
    // above the level, and each butterfly decrements an edge at most once
    if constexpr (N32) return atomicSub(a.sup32 + e, k);
    else return atomicAdd(a.sup + e, (unsigned long long)(-(long long)k));
}

// Append n of the edges e[0..2] (those in `mask`) to a frontier list.
__device__ __forceinline__ void list_append(const MspArgs &a, uint32_t *list, uint32_t *len, uint4 *head,
                                            uint32_t e0, uint32_t e1, uint32_t e2, uint32_t mask, uint32_t stamp,
                                         uint32_t value) {
    const uint32_t e[3] = {e0, e1, e2};
    uint2 ends[3];
#pragma unroll
    for (uint32_t q = 0; q < 3; q++)
        if (mask >> q & 1) ends[q] = __ldg(a.ends + e[q]);  // beside the counter's round trip
    uint32_t at = atomicAdd(len, (uint32_t)__popc(mask));
#pragma unroll
    for (uint32_t q = 0; q < 3; q++)
        if (mask >> q & 1) {
            list[at] = e[q];
            if (at < 32) head[at] = make_uint4(e[q], ends[q].x, ends[q].y, 0);
            at++;
            a.enter[e[q]] = stamp;
            a.result[e[q]] = value;
        }
}

// Settle up to three decrements, of k[q] on e[q] with old support old[q] (0:
// none).  low: the thread's running minimum of the supports left above the
// level.
template <bool N32>
__device__ __forceinline__ void dec_settle(const MspArgs &a, const Round<N32> &rd, const uint32_t (&e)[3],
                                           uint32_t k2, const SupWord<N32> (&old)[3], SupWord<N32> &low) {
    uint32_t push = 0, near = 0;
#pragma unroll
    for (uint32_t q = 0; q < 3; q++) {
        const SupWord<N32> nw = old[q] - (q == 2 ? k2 : 1u);
        if (old[q] > rd.L) {
            if (nw > rd.L) low = nw < low ? nw : low;
            else push |= 1u << q;
            if (old[q] >= rd.hi && nw < rd.hi) near |= 1u << q;
        }
    }
    if (push) list_append(a, rd.next, rd.next_len, rd.next_head, e[0], e[1], e[2], push, rd.r + 1, (uint32_t)rd.L);
    if (near) {
        uint32_t at = atomicAdd(rd.near_len, (uint32_t)__popc(near));
#pragma unroll
        for (uint32_t q = 0; q < 3; q++)
            if (near >> q & 1) rd.near_list[at++] = e[q];
    }
}

// ---------------------------------------------------------------------------
// shared memory
// ---------------------------------------------------------------------------

// Frontier edges as this CTA has planned them.
struct Smem {
    uint32_t e_uv[kEdges], e_piv[kEdges], e_anc[kEdges];
    uint32_t e_po[kEdges], e_pd[kEdges];   // pivot row: start, degree
    uint32_t e_ao[kEdges], e_ad[kEdges], e_at[kEdges];  // anchor row: start, degree, table
    uint32_t e_info[kEdges];               // log2 of the tasks that share a block of mids; kPivIsV
    uint32_t e_pre[kEdges + 1];            // exclusive prefix of the task counts
    uint32_t dec[kThreads];                // per warp and mid: pending pivot-side decrements
    uint32_t wsum[kWarps];
    unsigned long long low;                // running minimum of the supports above the level
    uint32_t chunk, total, next_task;
    Control now;                           // the control words as of the last barrier
    unsigned long long tasks, anchor;      // counters of this CTA
    unsigned long long prof_t, prof[8];    // see PF_*
};

constexpr uint32_t kPivIsV = 0x80000000u;  // the pivot is the edge's V end

// Steps of the time accounting (indices of the published counters).
enum { PF_PROBE = 3, PF_BARRIER = 6, PF_OTHER = 7 };

// Time accounting and bookkeeping are done by a CTA's last thread: the first
// warp plans and has the first task, so it is on the longest path.
__device__ __forceinline__ bool is_clerk() { return threadIdx.x == kThreads - 1; }

__device__ __forceinline__ void prof_mark(Smem &sm, int k) {
    if (is_clerk()) {
        const unsigned long long t = clock64();
        sm.prof[k] += t - sm.prof_t;
        sm.prof_t = t;
    }
}

// The control words and the head of a frontier list (lane i: entry i), by the
// first warp (the caller synchronises the block).
// One request per CTA: the same word read by all 2,432 warps of the grid at
// once is served one request at a time by its L2 slice (about a microsecond).
__device__ __forceinline__ uint4 load_control(const MspState *s, Smem &sm, uint32_t list) {
    const uint4 head = __ldcg(&s->head[list][threadIdx.x]);
    if (threadIdx.x < kControlWords)
        reinterpret_cast<uint32_t *>(&sm.now)[threadIdx.x] =
            __ldcg(reinterpret_cast<const uint32_t *>(&s->ctl) + threadIdx.x);
    return head;
}

// ---------------------------------------------------------------------------
// peel
// ---------------------------------------------------------------------------

// Plan frontier edge e as entry i: orientation and tasks; returns their number.
//  * The pivot is the endpoint whose row's position total is smaller; both
//    orientations visit the same butterflies.
//  * A task is a warp on a block of 32 of the pivot's mids, or, where their
//    rows hold more positions than a task should (1 / inv_task), on an equal
//    part of them: a power of two of parts, at most about `budget` tasks for
//    the edge, beyond which the warps of the grid have enough to do.
__device__ __forceinline__ uint32_t plan_edge(const MspArgs &a, Smem &sm, uint32_t i, uint32_t e, uint2 uv,
                                              float budget, uint32_t &anchor) {
    const VRec ru = load_vrec(a.vrec + uv.x), rv = load_vrec(a.vrec + uv.y);
    const bool pv = rv.hop <= ru.hop;
    const VRec &p = pv ? rv : ru, &q = pv ? ru : rv;
    const uint32_t blocks = (p.deg + 31) >> 5;
    // positions of a block: every mid has at most the anchor's degree
    const float est = fminf((float)p.hop, (float)p.deg * (float)q.deg);
    const float parts = __fdividef(fminf(est * a.inv_task, budget), (float)blocks);
    const int lg = parts > 1.0f ? min(16, (__float_as_int(parts) >> 23) - 126) : 0;  // ceil(log2), or one more
    sm.e_uv[i] = e;
    sm.e_piv[i] = pv ? uv.y : uv.x;
    sm.e_anc[i] = pv ? uv.x : uv.y;
    sm.e_po[i] = p.off;
    sm.e_pd[i] = p.deg;
    sm.e_ao[i] = q.off;
    sm.e_ad[i] = q.deg;
    sm.e_at[i] = q.tab;
    sm.e_info[i] = (uint32_t)lg | (pv ? kPivIsV : 0u);
    anchor = q.deg;
    return blocks << lg;
}

// Plan up to 32 edges (lane i: entry h of frontier edge i) by one warp; the
// caller synchronises the block.
__device__ __forceinline__ void plan_warp(const MspArgs &a, Smem &sm, uint32_t cnt, uint4 h, uint32_t warps,
                                          bool count_anchor) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t t = 0, anchor = 0;
    if (lane < cnt)
        t = plan_edge(a, sm, lane, h.x, make_uint2(h.y, h.z), __fdividef(4.0f * (float)warps, (float)cnt) + 1.0f,
                      anchor);
    const uint32_t inc = warp_inclusive(t);
    if (lane < cnt) sm.e_pre[lane] = inc - t;
    if (lane == 31) {
        sm.total = inc;
        sm.next_task = kWarps;
    }
    if (count_anchor) {
        anchor = __reduce_add_sync(0xffffffffu, anchor);
        if (lane == 0) sm.anchor += anchor;
    }
}

// Plan curr[0, cnt) (cnt <= kEdges) for `warps` warps.  Ends synchronised.
__device__ __forceinline__ void plan_block(const MspArgs &a, Smem &sm, const uint32_t *curr, uint32_t cnt,
                                           uint32_t warps, bool count_anchor) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = threadIdx.x;
    uint32_t t = 0, anchor = 0;
    if (i < cnt) {
        const uint32_t e = __ldcg(curr + i);
        t = plan_edge(a, sm, i, e, __ldg(a.ends + e), __fdividef(4.0f * (float)warps, (float)cnt) + 1.0f, anchor);
    }
    const uint32_t inc = warp_inclusive(t);
    if (lane == 31) sm.wsum[warp] = inc;
    anchor = __reduce_add_sync(0xffffffffu, anchor);
    if (lane == 0 && count_anchor) atomicAdd(&sm.anchor, (unsigned long long)anchor);
    __syncthreads();
    const uint32_t w = warp_inclusive(lane < kWarps ? sm.wsum[lane] : 0);
    const uint32_t before = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0);
    if (i < cnt) sm.e_pre[i] = (warp ? before : 0) + inc - t;
    if (i == kThreads - 1) {
        sm.total = (warp ? before : 0) + inc;
        sm.next_task = kWarps;
    }
    __syncthreads();
}

// BT_MSP_LATE_NS: an eighth of the CTAs, other ones each time, stay about that
// long between a barrier and what they read behind it.  Whatever the others do
// meanwhile, the results are the same.
__device__ __forceinline__ void linger(const MspArgs &a, uint32_t epoch) {
    if (a.late_ns && ((blockIdx.x * 0x9E3779B1u ^ epoch * 0x85EBCA6Bu) * 0xC2B2AE35u >> 29) == 0) __nanosleep(a.late_ns);
}

// Barrier of the team.  Publishes the CTA's running minimum to cand[k3], refreshes
// sm.now, and with `plan` plans the next frontier (`len`, a word of sm.now, is its length,
// `list` its list) when it is a short one: its entries come with the control words.
__device__ __forceinline__ bool barrier(const MspArgs &a, const Team &t, Smem &sm, uint32_t &epoch, uint32_t k3,
                                        const uint32_t &len, uint32_t list, bool plan) {
    __syncthreads();
    prof_mark(sm, PF_OTHER);
    int ok = 1;
    if (threadIdx.x < 32) {
        const unsigned long long low = sm.low;
        __syncwarp();
        if (threadIdx.x == 0) {
            // (sm.now is of the last barrier: cand only falls meanwhile)
            if (low < sm.now.cand[k3]) atomicMin(&t.s->ctl.cand[k3], low);
            sm.low = ~0ull;
        }
        __syncwarp();
        epoch += t.size;
        ok = bt::barrier_wait(t.bar, epoch, a.wait_ns);
        if (!ok) a.sh->error = bt::ERR_TIMEOUT;
        linger(a, epoch);
        const uint4 head = load_control(t.s, sm, list);
        __syncwarp();
        const uint32_t cnt = len;
        if (plan && cnt - 1 < 32 && cnt <= a.local_plan)
            plan_warp(a, sm, cnt, head, t.size * kWarps, t.rank == 0);
    }
    ok = __syncthreads_and(ok);
    prof_mark(sm, PF_BARRIER);
    return ok != 0;
}

// Every thread's running minimum into the CTA's (before a barrier).
template <bool N32>
__device__ __forceinline__ void fold_low(Smem &sm, SupWord<N32> low) {
    if constexpr (N32) low = __reduce_min_sync(0xffffffffu, low);
    else low = warp_min(low);
    if ((threadIdx.x & 31) == 0 && low != (SupWord<N32>)~0ull) atomicMin(&sm.low, (unsigned long long)low);
}

constexpr uint32_t kRev = 0x40000000u;     // the anchor's row is walked, the mid's table looked up
constexpr uint32_t kPmCurr = 0x80000000u;  // edge (pivot, mid) is in the frontier
constexpr uint32_t kNbMask = 0x3fffffffu;

// Run this CTA's tasks (first + step * j for j = 0, 1, ..., below `tasks`) of
// the planned edges and rule on every butterfly found.  Its warps take them
// one by one; no block barriers.
template <bool N32>
__device__ __forceinline__ void run_tasks(const MspArgs &a, Smem &sm, uint32_t cnt, uint32_t tasks, uint32_t first,
                                          uint32_t step, const Round<N32> &rd, PeelWork &wk, SupWord<N32> &low) {
    const uint32_t lane = threadIdx.x & 31, r = rd.r;
    uint32_t *dec = sm.dec + (threadIdx.x & ~31u);
    for (uint32_t task = first + step * (threadIdx.x >> 5); task < tasks;) {
        const uint32_t i = bt::warp_find_slot(sm.e_pre, cnt, task);
        const uint32_t lg = sm.e_info[i] & 31, piv = sm.e_piv[i], ad = sm.e_ad[i];
        const uint32_t local = task - sm.e_pre[i], part = local & ((1u << lg) - 1);
        // one mid per lane: shorter side, table and length of the (mid, anchor) pair
        const uint32_t k = (local >> lg) * 32 + lane;
        uint32_t row = 0, tab = 0, nb = 0, e_pm = 0, len = 0;
        if (k < sm.e_pd[i]) {
            const uint32_t pos = sm.e_po[i] + k;
            const uint32_t mid = a.nbr[pos];
            e_pm = a.eid[pos];
            const uint32_t en = a.enter[e_pm];
            const VRec rm = load_vrec(a.vrec + mid);
            if (mid != sm.e_anc[i] && !is_done(en, r)) {
                const bool rev = ad < rm.deg;
                row = rev ? sm.e_ao[i] : rm.off;
                tab = rev ? rm.tab : sm.e_at[i];
                nb = bt_row_buckets(rev ? rm.deg : ad) | (rev ? kRev : 0u) | (en == r ? kPmCurr : 0u);
                len = rev ? ad : rm.deg;
            }
        }
        uint32_t pre = warp_inclusive(len);
        const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
        pre -= len;
        // this part's positions: [total * part / 2^lg, total * (part + 1) / 2^lg)
        uint32_t f0 = 0, f1 = total;
        if (lg) {
            const uint32_t q = total >> lg, rem = total & ((1u << lg) - 1);
            f0 = q * part + (rem * part >> lg);
            f1 = q * (part + 1) + (rem * (part + 1) >> lg);
        }
        if (lane == 0) wk.probes += f1 - f0;
        // decrements in flight: each is settled a round later, beside that
        // round's loads, the last ones beside the pivot-side decrement
        uint32_t pe[3] = {0, 0, e_pm};
        SupWord<N32> old[3] = {0, 0, 0};
        for (uint32_t fb = f0; fb < f1; fb += 32) {
            const uint32_t f = fb + lane;
            // the mid of position f: the last lane with pre <= f and a position of its own
            uint32_t m = 0;
#pragma unroll
            for (uint32_t o = 16; o; o >>= 1) {
                const uint32_t t = __shfl_sync(0xffffffffu, pre, m + o);
                if (t <= f) m += o;
            }
            const uint32_t mrow = __shfl_sync(0xffffffffu, row, m), mtab = __shfl_sync(0xffffffffu, tab, m);
            const uint32_t mnb = __shfl_sync(0xffffffffu, nb, m), mpre = __shfl_sync(0xffffffffu, pre, m);
            const uint32_t mpm = __shfl_sync(0xffffffffu, e_pm, m);
            uint32_t y = piv, e1 = 0;
            if (f < f1) {
                y = a.nbr[mrow + (f - mpre)];
                e1 = a.eid[mrow + (f - mpre)];
            }
            dec_settle<N32>(a, rd, pe, 0, old, low);
            old[0] = old[1] = 0;
            if (y == piv) continue;
            const bt::RowPlace at = bt::row_place(y, mnb & kNbMask);
            const bt::RowBucket q1 = bt::row_bucket(a.pool, mtab, at.h1);
            const bt::RowBucket q2 = bt::row_bucket(a.pool, mtab, at.h2);
            const uint32_t en1 = a.enter[e1];
            const uint32_t e2 = bt::row_resolve(a.pool, mtab, mnb & kNbMask, at, q1, q2, y);
            if (e2 == kEmpty) continue;
            wk.hits++;  // a butterfly visited (the reference's intersection hit)
            const uint32_t en2 = a.enter[e2];
            if (is_done(en1, r) || is_done(en2, r)) continue;
            const bool rev = mnb & kRev, isv = sm.e_info[i] & kPivIsV;
            const uint32_t e_my = rev ? e2 : e1, e_ay = rev ? e1 : e2;
            const bool c1 = en1 == r, c2 = en2 == r, c_pm = mnb & kPmCurr;
            const bool c_my = rev ? c2 : c1, c_ay = rev ? c1 : c2;
            // name the edges as the reference does: w on u's side, x on v's
            const uint32_t d = peel_rule(sm.e_uv[i], isv ? mpm : e_ay, e_my, isv ? e_ay : mpm, isv ? c_pm : c_ay,
                                         c_my, isv ? c_ay : c_pm, a.exact);
            wk.decs += __popc(d);
            const bool d_wv = d & 1, d_wx = d & 2, d_ux = d & 4;
            const bool d_ay = isv ? d_ux : d_wv;
            pe[0] = e1;
            pe[1] = e2;
            if (rev ? d_ay : d_wx) old[0] = dec_issue<N32>(a, e1, 1);
            if (rev ? d_wx : d_ay) old[1] = dec_issue<N32>(a, e2, 1);
            if (isv ? d_wv : d_ux) atomicAdd(dec + m, 1u);
        }
        // the next task, and the pivot-side decrements: one edge per mid
        uint32_t j = 0;
        if (lane == 0) j = atomicAdd(&sm.next_task, 1u);
        __syncwarp();
        const uint32_t n_pm = dec[lane];
        if (n_pm) {
            dec[lane] = 0;
            old[2] = dec_issue<N32>(a, e_pm, n_pm);
        }
        dec_settle<N32>(a, rd, pe, n_pm, old, low);
        if (wk.full()) wk.carry(*a.sh, [](unsigned long long *t, uint32_t v) { atomicAdd(t, (unsigned long long)v); });
        __syncwarp();
        task = first + step * __shfl_sync(0xffffffffu, j, 0);
    }
}

// Peel the frontier curr[0, len): one sub-round without its barrier (which
// has planned it already when it is short).
template <bool N32>
__device__ __forceinline__ void peel(const MspArgs &a, const Team &t, Smem &sm, const uint32_t *curr, uint32_t len, uint32_t *ctr,
                                     const Round<N32> &rd, PeelWork &wk, SupWord<N32> &low) {
    const uint32_t rank = t.rank, size = t.size;
    // a frontier that every CTA plans whole, its tasks dealt to all CTAs, or
    // chunks of it that a CTA plans and runs alone: its first is its own
    // rank, the rest come from the counter
    const bool whole = len <= a.local_plan;
    uint32_t chunk = len;
    if (!whole) {
        chunk = len / (size * a.chunks_per_cta) + 1;
        chunk = chunk < 8 ? 8 : chunk > kEdges ? kEdges : chunk;
    }
    for (uint32_t c = whole ? 0 : rank; c * chunk < len;) {
        const uint32_t first = c * chunk, cnt = len - first < chunk ? len - first : chunk;
        if (!whole && threadIdx.x == 0) sm.chunk = size + atomicAdd(ctr, 1u);
        if (!whole || cnt > 32) plan_block(a, sm, curr + first, cnt, whole ? size * kWarps : kWarps, !whole || rank == 0);
        const uint32_t tasks = sm.total;
        if (is_clerk() && (!whole || rank == 0)) sm.tasks += tasks;
        run_tasks<N32>(a, sm, cnt, tasks, whole ? rank : 0, whole ? size : 1, rd, wk, low);
        if (whole) break;
        __syncthreads();
        c = sm.chunk;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// level transition helpers
// ---------------------------------------------------------------------------

// Minimum support over the live entries of `list` (team-wide atomicMin).
template <bool N32>
__device__ __forceinline__ void list_min(const MspArgs &a, const Team &t, const uint32_t *list, uint32_t len, unsigned long long *out) {
    unsigned long long v = ~0ull;
    const uint32_t gtid = t.thread(), gsz = t.threads();
    for (uint32_t i = gtid; i < len; i += gsz) {
        const uint32_t e = __ldcg(list + i);
        const uint32_t en = __ldcg(a.enter + e);
        const unsigned long long s = sup_of<N32>(a, e);
        if (en == 0) v = s < v ? s : v;
    }
    v = warp_min(v);
    if ((threadIdx.x & 31) == 0 && v != ~0ull) atomicMin(out, v);
}

// Drop processed edges (enter in (0, r)) from every row; one warp per vertex,
// in place.
__device__ __forceinline__ void compress_rows(const MspArgs &a, const Team &t, uint32_t r) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nw = t.threads() >> 5;
    for (uint32_t x = t.job.v0 + (t.thread() >> 5); x < t.job.v1; x += nw) {
        const uint32_t b = a.vrec[x].off, d = a.vrec[x].deg;
        uint32_t w = 0;
        for (uint32_t j0 = 0; j0 < d; j0 += 32) {
            const uint32_t j = j0 + lane;
            uint32_t y = 0, e = 0;
            bool keep = false;
            if (j < d) {
                y = a.nbr[b + j];
                e = a.eid[b + j];
                keep = !is_done(__ldcg(a.enter + e), r);
            }
            const uint32_t bal = __ballot_sync(0xffffffffu, keep);
            __syncwarp();
            if (keep) {
                const uint32_t pos = w + __popc(bal & ((1u << lane) - 1));
                a.nbr[b + pos] = y;
                a.eid[b + pos] = e;
            }
            w += __popc(bal);
            __syncwarp();
        }
        if (lane == 0) a.vrec[x].deg = w;
    }
}

// Position total (from the degrees `deg` gives) and table of row x, by one warp.
template <class Deg>
__device__ __forceinline__ void prepare_row(const MspArgs &a, uint32_t x, uint32_t off, uint32_t d, uint32_t tab,
                                            Deg deg) {
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long hop = 0;
    for (uint32_t j = lane; j < d; j += 32) hop += deg(a.nbr[off + j]);
    hop = warp_sum(hop);
    if (lane == 0) a.vrec[x].hop = hop > 0xffffffffull ? 0xffffffffu : (uint32_t)hop;
    bt::row_build(a.pool, tab, d, a.nbr + off, [&](uint32_t j) { return a.eid[off + j]; });
}

__device__ __forceinline__ void prepare_rows(const MspArgs &a, const Team &t) {
    const uint32_t nw = t.threads() >> 5;
    for (uint32_t x = t.job.v0 + (t.thread() >> 5); x < t.job.v1; x += nw) {
        const VRec v = load_vrec(a.vrec + x);
        if (v.deg) prepare_row(a, x, v.off, v.deg, v.tab, [&](uint32_t y) { return __ldcg(&a.vrec[y].deg); });
    }
}

// ---------------------------------------------------------------------------
// the persistent kernel
// ---------------------------------------------------------------------------

template <bool N32>
__global__ void __launch_bounds__(kThreads, 1) k_msp(const __grid_constant__ MspArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
    if (threadIdx.x == 0) {
        sm.low = ~0ull;
        sm.tasks = sm.anchor = 0;
        for (int k = 0; k < 8; k++) sm.prof[k] = 0;
    }
    if (is_clerk()) sm.prof_t = clock64();
    sm.dec[threadIdx.x] = 0;
    __syncthreads();
    Team t;
    const uint32_t team_index = a.team_of[blockIdx.x];
    TeamState *team = a.teams + team_index;
    t.size = team->size;
    t.rank = blockIdx.x - team->cta0;
    t.bar = &team->bar;
    const uint32_t gtid = t.thread(), gsz = t.threads();
    const bool clerk = t.rank == 0 && is_clerk();
    PeelWork wk;
    uint32_t epoch = 0;               // barrier arrivals so far (the same in every CTA of the team)
    // of the team's clerk
    const unsigned long long t_start = bt::global_ns(), c_start = clock64();
    unsigned long long t_mark = c_start, ph0 = 0, ph1 = 0;  // SM cycles
    unsigned long long subrounds = 0, levels = 0, rebuilds = 0, compressions = 0;

    for (bool first = true;; first = false) {
        // ---------------------------------------------------- the next graph
        if (t.rank == 0 && threadIdx.x == 0) {
            const uint32_t q = first ? team_index : a.nteams + atomicAdd(&a.sh->queue, 1u);
            if (q < a.njobs) {
                Control &c = a.states[q].ctl;
                c.delta = 1;
                c.far_min = c.cand[0] = c.cand[1] = c.cand[2] = ~0ull;
            }
            team->job = q;
        }
        __syncthreads();
        int ok = 1;
        if (threadIdx.x < 32) {
            epoch += t.size;
            ok = bt::barrier_wait(t.bar, epoch, a.wait_ns);
            if (!ok) a.sh->error = bt::ERR_TIMEOUT;
            linger(a, epoch);
            const uint32_t q = __ldcg(&team->job);
            if (threadIdx.x == 0) sm.chunk = q;
            if (q < a.njobs) load_control(a.states + q, sm, 0);
        }
        if (!__syncthreads_and(ok)) return;
        const uint32_t q = sm.chunk;
        if (q >= a.njobs) break;
        MspState *s = t.s = a.states + q;
        t.job = a.jobs[q];
        // the same in every CTA of the team
        uint32_t r = 2, r3 = 2;       // sub-round index (1 marks the zero-support edges), modulo 3
        uint32_t k3 = 0;              // level number modulo 3 (slot of cand)
        unsigned long long L = 0;     // current level
        uint32_t nsel = 0;            // near bucket: near0, length near_ctr[nsel]
        const uint32_t e0 = t.job.e0; // the lists of a graph lie at its edges' place
        uint32_t *near0 = a.near_a + e0, *near1 = a.near_b + e0, *far0 = a.far_a + e0, *far1 = a.far_b + e0;
        uint32_t near_dead = 0;       // its entries processed since it was last compacted
        unsigned long long hi = 0;    // bound of the near bucket
        unsigned long long live = sm.now.far_len, live_at_compress = t.job.m;
        for (;;) {
            // ------------------------------------------------ level transition
            uint32_t curr_len = sm.now.len[r3];
            if (curr_len == 0) {
                bool squeeze = false, dry = false;
                for (;;) {
                    L = sm.now.cand[k3];
                    if (L >= hi) {
                        // near is dry: split the far bucket
                        const uint32_t far_len = sm.now.far_len;
                        list_min<N32>(a, t, far0, far_len, &s->ctl.far_min);
                        if (!barrier(a, t, sm, epoch, k3, sm.now.len[r3], r & 1, false)) return;
                        L = sm.now.far_min;
                        if (L == ~0ull) {  // nothing left
                            dry = true;
                            break;
                        }
                        // all of it at once when a scan of it takes one entry per thread
                        hi = live <= gsz ? ~0ull : L + sm.now.delta;
                        for (uint32_t i = gtid; i < far_len; i += gsz) {
                            const uint32_t e = __ldcg(far0 + i);
                            if (__ldcg(a.enter + e) != 0) continue;
                            if (sup_of<N32>(a, e) < hi) near1[atomicAdd(&s->ctl.near_ctr[nsel ^ 1], 1u)] = e;
                            else far1[atomicAdd(&s->ctl.far2_len, 1u)] = e;
                        }
                        if (!barrier(a, t, sm, epoch, k3, sm.now.len[r3], r & 1, false)) return;
                        {   // every CTA swaps its copies of the bucket pointers
                            uint32_t *t = near0; near0 = near1; near1 = t;
                            t = far0; far0 = far1; far1 = t;
                        }
                        nsel ^= 1;
                        near_dead = 0;
                        if (clerk) {
                            s->ctl.near_ctr[nsel ^ 1] = 0;
                            s->ctl.far_len = sm.now.far2_len;
                            s->ctl.far2_len = 0;
                            s->ctl.far_min = ~0ull;
                            rebuilds++;
                            const uint32_t near_len = sm.now.near_ctr[nsel];
                            if (near_len > 4 * gsz && sm.now.delta > 1) s->ctl.delta = sm.now.delta >> 1;
                            else if (near_len < gsz / 4) s->ctl.delta = sm.now.delta << 1;
                        }
                    }
                    // frontier of sub-round r = near edges with support == L, and
                    // the lowest support above it; entries processed meanwhile are
                    // dropped from the list once they are half of it
                    k3 = next3(k3);
                    if (clerk) {
                        s->ctl.cand[next3(k3)] = ~0ull;
                        s->ctl.scan_len[next3(k3)] = 0;
                    }
                    const uint32_t near_len = sm.now.near_ctr[nsel];
                    const bool compact = near_len > gsz && near_dead > near_len / 2;
                    uint32_t *front = ((r & 1 ? a.list1 : a.list0) + e0);
                    SupWord<N32> low = (SupWord<N32>)~0ull;
                    for (uint32_t i = gtid; i < near_len; i += gsz) {
                        const uint32_t e = __ldcg(near0 + i);
                        const uint32_t en = __ldcg(a.enter + e);
                        const SupWord<N32> v = sup_of<N32>(a, e);
                        if (en != 0) continue;
                        if (v == L) {
                            list_append(a, front, &s->ctl.scan_len[k3], s->head[r & 1], e, 0, 0, 1, r, (uint32_t)L);
                        } else {
                            if (v < low) low = v;
                            if (compact) near1[atomicAdd(&s->ctl.near_ctr[nsel ^ 1], 1u)] = e;
                        }
                    }
                    fold_low<N32>(sm, low);
                    squeeze = (double)live <= (double)a.cfrac * (double)live_at_compress &&
                              (double)live_at_compress >= (double)a.cfloor * (double)t.job.m;
                    // (a compaction changes the rows that a plan is made from: it comes after it)
                    if (!barrier(a, t, sm, epoch, k3, sm.now.scan_len[k3], r & 1, !squeeze)) return;
                    curr_len = sm.now.scan_len[k3];
                    if (compact) {
                        uint32_t *t = near0; near0 = near1; near1 = t;
                        nsel ^= 1;
                        near_dead = 0;
                        if (clerk) s->ctl.near_ctr[nsel ^ 1] = 0;
                    }
                    // no edge at L: the minimum was of an edge that has since left;
                    // what this scan collected is exact
                    if (curr_len != 0) break;
                }
                if (dry) break;
                if (clerk) {
                    atomicMax(&a.sh->last_level, L);
                    levels++;
                    if (L > 0xffffffffull) a.sh->overflow = 1;
                }
                if (squeeze) {
                    live_at_compress = live;
                    if (clerk) compressions++;
                    compress_rows(a, t, r);
                    if (!barrier(a, t, sm, epoch, k3, sm.now.scan_len[k3], r & 1, false)) return;
                    prepare_rows(a, t);
                    if (!barrier(a, t, sm, epoch, k3, sm.now.scan_len[k3], r & 1, true)) return;
                }
                if (clerk) {
                    const unsigned long long t = clock64();
                    ph0 += t - t_mark;
                    t_mark = t;
                }
            }
            // ------------------------------------------------ sub-round r
            Round<N32> rd;
            rd.r = r;
            rd.L = (SupWord<N32>)L;
            // a bound above every support works like any other
            rd.hi = N32 && hi > 0xffffffffull ? (SupWord<N32>)0xffffffffull : (SupWord<N32>)hi;
            rd.next = ((r & 1 ? a.list0 : a.list1) + e0);
            rd.next_len = &s->ctl.len[next3(r3)];
            rd.next_head = s->head[(r + 1) & 1];
            rd.near_list = near0;
            rd.near_len = &s->ctl.near_ctr[nsel];
            if (clerk) {
                // slots used two sub-rounds from now; every CTA is past their last use
                s->ctl.len[next3(next3(r3))] = 0;
                s->task_ctr[next3(next3(r3))] = 0;
                subrounds++;
            }
            live -= curr_len;
            near_dead += curr_len;
            const unsigned long long task_t0 = a.trace ? bt::global_ns() : 0;
            const unsigned long long tasks0 = sm.tasks;
            const uint32_t probes0 = wk.probes;
            SupWord<N32> low = (SupWord<N32>)~0ull;
            peel<N32>(a, t, sm, ((r & 1 ? a.list1 : a.list0) + e0), curr_len, &s->task_ctr[r3], rd, wk, low);
            prof_mark(sm, PF_PROBE);
            fold_low<N32>(sm, low);
            if (a.trace && r < a.trace_cap) {
                // (less than 2^31 a warp; bit 31 may have been carried meanwhile)
                const unsigned long long walked = warp_sum((wk.probes - probes0) & 0x7fffffffu);
                if ((threadIdx.x & 31) == 0) {
                    atomicMax(&a.trace[r].max_task_ns, bt::global_ns() - task_t0);
                    atomicAdd(&a.trace[r].walked, walked);
                }
                if (threadIdx.x == 0) atomicAdd(&a.trace[r].tasks, (uint32_t)(sm.tasks - tasks0));
            }
            if (!barrier(a, t, sm, epoch, k3, sm.now.len[next3(r3)], (r + 1) & 1, true)) return;
            if (clerk) {
                const unsigned long long t = clock64();
                if (a.trace && r < a.trace_cap) {
                    a.trace[r].t_ns = bt::global_ns() - task_t0;
                    a.trace[r].frontier = curr_len;
                }
                ph1 += t - t_mark;
                t_mark = t;
            }
            r++;
            r3 = next3(r3);
        }
        if (clerk) atomicAdd(&a.sh->done, 1u);
    }
    // flush the counters
    if (clerk) {
        if (blockIdx.x == 0) {
            const double ns = (double)(bt::global_ns() - t_start) / (double)(clock64() - c_start);
            a.sh->ph_ns[0] = (unsigned long long)((double)ph0 * ns);
            a.sh->ph_ns[1] = (unsigned long long)((double)ph1 * ns);
        }
        atomicAdd(&a.sh->subrounds, subrounds);
        atomicAdd(&a.sh->levels_seen, levels);
        atomicAdd(&a.sh->rebuilds, rebuilds);
        atomicAdd(&a.sh->compressions, compressions);
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < 8; q++) atomicAdd(&a.sh->prof[q], sm.prof[q]);
        atomicAdd(&a.sh->tasks, sm.tasks);
        atomicAdd(&a.sh->w_anchor, sm.anchor);
    }
    const unsigned long long probes = warp_sum(wk.probes), hits = warp_sum(wk.hits), decs = warp_sum(wk.decs);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&a.sh->w_probes, probes);
        atomicAdd(&a.sh->w_hits, hits);
        atomicAdd(&a.sh->w_decs, decs);
    }
}

// ---------------------------------------------------------------------------
// set-up kernels
// ---------------------------------------------------------------------------

// Every graph's supports added up (four per butterfly); gridDim.y blocks a graph.
__global__ void __launch_bounds__(256) k_job_supports(const Job *jobs, const unsigned long long *sup,
                                                      unsigned long long *sums) {
    const Job j = jobs[blockIdx.x];
    unsigned long long v = 0;
    for (uint64_t i = blockIdx.y * 256ull + threadIdx.x; i < j.m; i += gridDim.y * 256ull) v += sup[(uint64_t)j.e0 + i];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(sums + blockIdx.x, v);
}

constexpr int kInitThreads = 256;

// Edge states, vertex records and row tables (the tables' places in the pool
// are given out block by block).  by_edge: (first edge, job) of every graph, by
// first edge.
__global__ void __launch_bounds__(kInitThreads) k_msp_init(MspArgs a, const unsigned long long *sup_in,
                                                           const uint32_t *off, const uint32_t *deg,
                                                           const uint2 *by_edge) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t e0 = blockIdx.x * (uint64_t)kInitThreads; e0 < a.m; e0 += (uint64_t)gridDim.x * kInitThreads) {
        const uint64_t e = e0 + threadIdx.x;
        const unsigned long long v = e < a.m ? sup_in[e] : 0;
        if (e < a.m) {
            if (a.sup32) a.sup32[e] = (uint32_t)v;  // every support fits (checked on the host)
            else a.sup[e] = v;
            a.result[e] = 0;
            a.enter[e] = v == 0 ? 1 : 0;  // support 0: processed first (count_es_zero, bitruss_msp.cu:38-50)
        }
        // the far list of the edge's graph: one counter update per warp and graph
        uint32_t q = 0;
        if (a.njobs > 1) {
            uint32_t hi = a.njobs;
            while (hi - q > 1) {  // the last graph whose first edge is at or below e
                const uint32_t md = (q + hi) >> 1;
                if (by_edge[md].x <= e) q = md;
                else hi = md;
            }
        }
        const uint32_t peers = __match_any_sync(0xffffffffu, v != 0 ? q : kEmpty);
        uint32_t at = 0;
        const uint32_t leader = __ffs(peers) - 1;
        if (v != 0 && lane == leader)
            at = atomicAdd(&a.states[a.njobs > 1 ? by_edge[q].y : 0].ctl.far_len, (uint32_t)__popc(peers));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (v != 0)
            a.far_a[(a.njobs > 1 ? by_edge[q].x : 0) + at + __popc(peers & ((1u << lane) - 1))] = (uint32_t)e;
    }
    // vertices: a block's tables are laid out first, then its warps build them
    __shared__ uint32_t base;
    __shared__ uint32_t s_tab[kInitThreads];
    __shared__ typename cub::BlockScan<uint32_t, kInitThreads>::TempStorage scan;
    const uint64_t step = gridDim.x;  // a block's vertices lie this far apart: ranks follow degree
    for (uint64_t x0 = blockIdx.x; x0 < a.n; x0 += step * kInitThreads) {
        const uint64_t x = x0 + step * threadIdx.x;
        const uint32_t d = x < a.n ? deg[x] : 0;
        uint32_t excl, tot;
        cub::BlockScan<uint32_t, kInitThreads>(scan).ExclusiveSum(d ? bt_row_buckets(d) : 0, excl, tot);
        if (threadIdx.x == 0) base = atomicAdd(&a.sh->pool_used, tot);
        __syncthreads();
        s_tab[threadIdx.x] = base + excl;
        if (x < a.n) a.vrec[x] = VRec{off[x], d, base + excl, 0};
        __syncthreads();
        for (uint32_t k = threadIdx.x >> 5; k < kInitThreads && x0 + step * k < a.n; k += kInitThreads / 32) {
            const uint32_t y = (uint32_t)(x0 + step * k), dy = deg[y];
            if (dy) prepare_row(a, y, off[y], dy, s_tab[k], [&](uint32_t z) { return __ldg(deg + z); });
        }
        __syncthreads();
    }
}

}  // namespace

// SM slots of the peeling kernel, per device.  A cooperative peel of nblocks
// CTAs (per_sm resident per SM) holds ceil(nblocks / per_sm) slots from its
// launch until it has finished; a device has one slot per SM, so the peels
// that run together -- contexts with a share of the SMs each, such as serving
// slots -- always fit side by side and never wait at a grid barrier for CTAs
// that cannot be placed.  A peel that wants every SM waits for the others to
// finish.
namespace {
constexpr int kMaxPoolDevices = 64;
std::mutex g_pool_mu;
std::condition_variable g_pool_cv;
int g_pool_free[kMaxPoolDevices];
bool g_pool_init[kMaxPoolDevices];

struct CtaSlots {
    int dev = -1, n = 0;
    void acquire(int device, int capacity, int want) {
        std::unique_lock<std::mutex> lk(g_pool_mu);
        if (!g_pool_init[device]) {
            g_pool_free[device] = capacity;
            g_pool_init[device] = true;
        }
        g_pool_cv.wait(lk, [&] { return g_pool_free[device] >= want; });
        g_pool_free[device] -= want;
        dev = device;
        n = want;
    }
    void release() {
        if (n == 0) return;
        {
            std::lock_guard<std::mutex> lk(g_pool_mu);
            g_pool_free[dev] += n;
            n = 0;
        }
        g_pool_cv.notify_all();
    }
    ~CtaSlots() { release(); }
};
}  // namespace

static unsigned long long wait_limit_ns() {
    const char *us = getenv("BT_WAIT_LIMIT_US");
    if (us && strtoull(us, nullptr, 10) > 0) return strtoull(us, nullptr, 10) * 1000ull;
    const char *v = getenv("BT_WAIT_LIMIT_MS");
    unsigned long long ms = v ? strtoull(v, nullptr, 10) : 120000ull;
    if (ms == 0) ms = 120000ull;
    return ms * 1000000ull;
}

static uint32_t late_ns() {
    const char *v = getenv("BT_MSP_LATE_NS");
    return v ? (uint32_t)std::min<unsigned long long>(strtoull(v, nullptr, 10), 1000000ull) : 0u;
}

static bt_status run_msp(bt_ctx *ctx, bool exact, uint32_t *levels) {
    uint64_t dummy = 0;
    BT_TRY(dev_ebfc(ctx, true, &dummy));
    DevGraph &g = ctx->g;
    cudaStream_t st = ctx->stream;
    const uint64_t m = g.m, n = g.n;
    cudaEvent_t e0 = ctx->ev[2], e1 = ctx->ev[3];
    cudaEventRecord(e0, st);

    CtxBuffers buffers(ctx);
    // the graphs to peel, and (of several) their work
    std::vector<Job> jobs;
    for (const auto &sp : g.spans)
        if (sp.m) jobs.push_back(Job{sp.v0, sp.v0 + sp.n, sp.e0, sp.m});
    const uint32_t njobs = (uint32_t)jobs.size();
    std::vector<PeelJob> job_work(njobs, PeelJob{0, 0});
    MspArgs a{};
    uint2 *d_by_edge = nullptr;
    const uint64_t mm = m ? m : 1, nn = n ? n : 1;
#define A(p, bytes) BT_TRY(buffers.alloc(&(p), (bytes)))
    A(a.sh, sizeof(MspShared));
    A(a.states, sizeof(MspState) * (njobs ? njobs : 1));
    A(a.jobs, sizeof(Job) * (njobs ? njobs : 1));
    A(d_by_edge, sizeof(uint2) * (njobs ? njobs : 1));
    A(a.vrec, sizeof(VRec) * nn);
    A(a.nbr, 8 * mm);
    A(a.eid, 8 * mm);
    A(a.pool, 32 * (g.tab_buckets ? g.tab_buckets : 1));
    // 32-bit working supports when they all fit: half the footprint and
    // 4-byte atomics for the decrements
    // (BT_MSP_WIDE=1 keeps 64-bit supports: the path graphs with a support
    // above 2^32 take, testable on small graphs)
    const char *wide = getenv("BT_MSP_WIDE");
    if (ctx->last_sup_max < 0xffffffffull && !(wide && *wide == '1')) A(a.sup32, 4 * mm);
    else A(a.sup, 8 * mm);
    A(a.enter, 4 * mm);
    A(a.list0, 4 * mm);
    A(a.list1, 4 * mm);
    A(a.near_a, 4 * mm);
    A(a.near_b, 4 * mm);
    A(a.far_a, 4 * mm);
    A(a.far_b, 4 * mm);
    const char *trace_path = getenv("BT_MSP_TRACE");
    if (trace_path && *trace_path && njobs == 1) {
        a.trace_cap = 4u << 20;
        A(a.trace, sizeof(TraceRow) * a.trace_cap);
    }
    a.result = ctx->result;
    // cooperative persistent launch: its CTAs, in teams
    const size_t smem = sizeof(Smem);
    const void *kfn = a.sup32 ? (const void *)k_msp<true> : (const void *)k_msp<false>;
    BT_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    BT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, kThreads, smem));
    if (per_sm < 1) return bt_fail(BT_ERR_CUDA, "msp kernel does not fit on an SM");
    const uint32_t capacity = (uint32_t)(ctx->sm_count * per_sm);
    const uint32_t ctas = ctx->peel_ctas && ctx->peel_ctas < capacity ? ctx->peel_ctas : capacity;
    std::vector<uint2> by_edge;
    if (njobs > 1) {
        unsigned long long *d_sums = nullptr;
        std::vector<unsigned long long> sums(njobs);
        A(d_sums, 8ull * njobs);
        BT_CUDA(cudaMemsetAsync(d_sums, 0, 8ull * njobs, st));
        BT_CUDA(cudaMemcpyAsync((void *)a.jobs, jobs.data(), sizeof(Job) * njobs, cudaMemcpyHostToDevice, st));
        k_job_supports<<<dim3(njobs, std::min(64u, std::max(1u, 1024u / njobs))), 256, 0, st>>>(
            a.jobs, (const unsigned long long *)ctx->sup, d_sums);
        bt_note_launches(1);
        BT_CUDA(cudaGetLastError());
        BT_CUDA(cudaMemcpyAsync(sums.data(), d_sums, 8ull * njobs, cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaStreamSynchronize(st));
        // those that take longest on one CTA first
        std::vector<uint32_t> order(njobs);
        for (uint32_t q = 0; q < njobs; q++) {
            order[q] = q;
            job_work[q] = PeelJob{jobs[q].m, sums[q] / 4};
        }
        auto cost = [&](uint32_t q) { return bt_peel_chain_us(job_work[q]) + bt_peel_walk_us(job_work[q]); };
        std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return cost(x) > cost(y); });
        std::vector<Job> jobs_by_cost;
        std::vector<PeelJob> work_by_cost;
        for (uint32_t q : order) {
            jobs_by_cost.push_back(jobs[q]);
            work_by_cost.push_back(job_work[q]);
        }
        jobs.swap(jobs_by_cost);
        job_work.swap(work_by_cost);
    }
    for (uint32_t q = 0; q < njobs; q++) by_edge.push_back(make_uint2(jobs[q].e0, q));
    std::sort(by_edge.begin(), by_edge.end(), [](const uint2 &x, const uint2 &y) { return x.x < y.x; });
    // how many CTAs peel each
    const std::vector<uint32_t> sizes = bt_plan_teams(job_work, ctas);
    std::vector<TeamState> teams(sizes.size());
    std::vector<uint32_t> team_of;
    for (uint32_t t = 0; t < sizes.size(); t++) {
        teams[t] = TeamState{};
        teams[t].cta0 = (uint32_t)team_of.size();
        teams[t].size = sizes[t];
        team_of.insert(team_of.end(), sizes[t], t);
    }
    const uint32_t nblocks = (uint32_t)team_of.size();
    a.nteams = (uint32_t)sizes.size();
    A(a.teams, sizeof(TeamState) * teams.size());
    A(a.team_of, 4 * team_of.size());
#undef A
    BT_CUDA(cudaMemsetAsync(a.sh, 0, sizeof(MspShared), st));
    // (these are copied before the calls return: pageable memory)
    BT_CUDA(cudaMemcpyAsync(a.teams, teams.data(), sizeof(TeamState) * teams.size(), cudaMemcpyHostToDevice, st));
    BT_CUDA(cudaMemcpyAsync((void *)a.team_of, team_of.data(), 4 * team_of.size(), cudaMemcpyHostToDevice, st));
    BT_CUDA(cudaMemsetAsync(a.states, 0, sizeof(MspState) * (njobs ? njobs : 1), st));
    if (njobs) {
        BT_CUDA(cudaMemcpyAsync((void *)a.jobs, jobs.data(), sizeof(Job) * njobs, cudaMemcpyHostToDevice, st));
        BT_CUDA(cudaMemcpyAsync(d_by_edge, by_edge.data(), sizeof(uint2) * njobs, cudaMemcpyHostToDevice, st));
    }
    if (a.trace) BT_CUDA(cudaMemsetAsync(a.trace, 0, sizeof(TraceRow) * a.trace_cap, st));
    BT_CUDA(cudaMemcpyAsync(a.nbr, g.nbr0, 8 * m, cudaMemcpyDeviceToDevice, st));
    BT_CUDA(cudaMemcpyAsync(a.eid, g.eid0, 8 * m, cudaMemcpyDeviceToDevice, st));
    a.njobs = njobs;
    a.n = g.n;
    a.m = m;
    a.exact = exact ? 1u : 0u;
    a.inv_task = 32.0f / (float)(ctx->msp_schedule[0] ? ctx->msp_schedule[0] : kMspMinGrain);
    a.chunks_per_cta = ctx->msp_schedule[1] ? ctx->msp_schedule[1] : kMspTasksPerCta;
    a.local_plan = std::min(ctx->msp_schedule[2] ? ctx->msp_schedule[2] : kMspLocalPlan, kEdges);
    a.wait_ns = wait_limit_ns();
    a.late_ns = late_ns();
    // Row compaction: whenever the live edges have halved since the last
    // compaction.  The reference also stops compacting once fewer than a tenth
    // of all edges are live (bitruss_msp.cu:537), which leaves the long tail
    // of the peel walking rows full of processed edges; dropping that floor
    // cut the row positions walked on the 20M-edge Chung-Lu graph by 11%.
    // Compaction changes which rows are walked, never a result.
    // BT_MSP_COMPACT="frac,floor" sets the trigger (the reference's is 0.5,0.1).
    a.cfrac = 0.5f;
    a.cfloor = 0.0f;
    if (const char *cv = getenv("BT_MSP_COMPACT")) {
        float f = 0, fl = 0;
        if (sscanf(cv, "%f,%f", &f, &fl) == 2 && f > 0 && f < 1 && fl >= 0 && fl <= 1) {
            a.cfrac = f;
            a.cfloor = fl;
        }
    }
    a.ends = g.ends;
    const unsigned blk = kInitThreads, cap = (unsigned)ctx->sm_count * 8;
    if (m) {
        // a thread per edge, a warp per row
        const uint64_t blocks = std::max<uint64_t>((m + blk - 1) / blk, (n * 32 + blk - 1) / blk);
        k_msp_init<<<(unsigned)std::min<uint64_t>(blocks, cap), blk, 0, st>>>(
            a, (const unsigned long long *)ctx->sup, g.off, g.deg0, d_by_edge);
        bt_note_launches(1);
        BT_CUDA(cudaGetLastError());
    }
    if (ctx->device < 0 || ctx->device >= kMaxPoolDevices)
        return bt_fail(BT_ERR_INVALID, "device index out of range");
    // SM slots (see CtaSlots): concurrent peels of this process fit side by side
    CtaSlots slots;
    NvtxRange range("k_msp");
    if (m) {
        slots.acquire(ctx->device, ctx->sm_count, (int)((nblocks + per_sm - 1) / per_sm));
        void *params[] = {&a};
        cudaEventRecord(ctx->ev[4], st);
        cudaError_t le = cudaLaunchCooperativeKernel(kfn, dim3(nblocks), dim3(kThreads), params, smem, st);
        if (le == cudaSuccess) le = cudaGetLastError();
        if (le != cudaSuccess) {
            slots.release();
            return bt_cuda_fail(le, "cudaLaunchCooperativeKernel(k_msp)", __FILE__, __LINE__);
        }
        cudaEventRecord(ctx->ev[5], st);
        bt_note_launches(1);
    }
    cudaEventRecord(e1, st);
    MspShared h{};
    {
        cudaError_t ce = cudaMemcpyAsync(&h, a.sh, sizeof(MspShared), cudaMemcpyDeviceToHost, st);
        if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
        slots.release();
        if (ce != cudaSuccess) return bt_cuda_fail(ce, "msp state readback", __FILE__, __LINE__);
    }
    if (a.trace) {
        // rows 2 .. subrounds+1 are sub-rounds; written as raw TraceRow records
        const uint64_t rows = std::min<uint64_t>(h.subrounds + 2, a.trace_cap);
        std::vector<TraceRow> tr(rows);
        BT_CUDA(cudaMemcpyAsync(tr.data(), a.trace, sizeof(TraceRow) * rows, cudaMemcpyDeviceToHost, st));
        BT_CUDA(cudaStreamSynchronize(st));
        if (FILE *f = fopen(trace_path, "wb")) {
            fwrite(tr.data(), sizeof(TraceRow), rows, f);
            fclose(f);
        }
    }
    float ms = -1;
    cudaEventElapsedTime(&ms, e0, e1);
    ctx->phase_ms[PH_MSP] = ms;
    ms = -1;
    if (m) cudaEventElapsedTime(&ms, ctx->ev[4], ctx->ev[5]);
    ctx->phase_ms[PH_PEEL] = ms;
    if (h.error == bt::ERR_TIMEOUT)
        return bt_fail(BT_ERR_TIMEOUT, "msp: a grid barrier wait exceeded its time limit");
    if (h.overflow) return bt_fail(BT_ERR_OVERFLOW, "msp: a bitruss number exceeds uint32");
    if (h.done != njobs) return bt_fail(BT_ERR_CUDA, "msp kernel ended without finishing");
    ctx->stats[0] = h.last_level;
    ctx->stats[1] = h.subrounds;
    ctx->stats[2] = h.compressions;
    ctx->stats[3] = h.tasks;
    ctx->stats[5] = h.levels_seen;
    ctx->stats[6] = h.rebuilds;
    ctx->work[0] = h.tasks;
    ctx->work[1] = h.w_probes;
    ctx->work[2] = h.w_anchor;
    ctx->work[3] = h.w_hits;
    ctx->work[4] = h.w_decs;
    ctx->work[5] = m;
    ctx->work[6] = h.ph_ns[0];
    ctx->work[7] = h.ph_ns[1];
    ctx->work[8] = 0;
    ctx->work[9] = a.sup32 ? 4 : 8;  // bytes per working support (and per decrement)
    for (int q = 0; q < 8; q++) ctx->prof[q] = h.prof[q] / (nblocks ? nblocks : 1);
    ctx->last_result = 2;
    if (levels) *levels = (uint32_t)h.last_level;
    return BT_OK;
}

bt_status dev_msp(bt_ctx *ctx, bool exact, uint32_t *levels) {
    try {
        return run_msp(ctx, exact, levels);
    } catch (const std::bad_alloc &) {
        return bt_fail(BT_ERR_HOST_MEMORY, "host allocation failed");
    }
}
