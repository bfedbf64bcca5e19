// bt_internal.h -- shared definitions of the GB300 bitruss engine.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/bitruss.h"

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------

// Record a message for bt_last_error() on this host thread and return `s`.
bt_status bt_fail(bt_status s, const std::string &msg);
bt_status bt_cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define BT_CUDA(call)                                                        \
    do {                                                                     \
        cudaError_t _e = (call);                                             \
        if (_e != cudaSuccess) return bt_cuda_fail(_e, #call, __FILE__, __LINE__); \
    } while (0)

#define BT_TRY(call)                                                         \
    do {                                                                     \
        bt_status _s = (call);                                               \
        if (_s != BT_OK) return _s;                                          \
    } while (0)

// Count of this library's own kernel launches (every launch site adds its
// launches; read by bt_kernel_launches).
void bt_note_launches(uint64_t k);

// NVTX range over a scope: each public call shows up as a named range on a
// profiler's timeline (no cost without a tool attached).
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// ---------------------------------------------------------------------------
// host graph: the reference's Graph fields (src/graph/graph.h:43-51)
// ---------------------------------------------------------------------------

struct bt_graph {
    uint32_t u_num = 0, l_num = 0, u_max = 0, n = 0;
    uint64_t m = 0;
    uint64_t support_max = 0;
    std::vector<uint32_t> offsets;    // n+1
    std::vector<uint32_t> neighbors;  // 2m
    std::vector<uint32_t> degrees;    // n
    std::vector<uint32_t> edges;      // 2m
    std::vector<uint32_t> edge_ids;   // 2m
    std::vector<uint32_t> edge_support_raw;  // m, as stored in a .bin (int32 bits)
    std::vector<uint32_t> bitruss_raw;       // m, as stored in a .bin
    // a row may hold a neighbour twice (duplicate lines are kept): some row does
    // not ascend strictly
    bool repeats = false;
    // batched arena only: graph index of every vertex (empty for one graph)
    // and the vertex count of the largest graph
    std::vector<uint32_t> segment;
    uint32_t seg_max_n = 0;
    std::vector<uint32_t> seg_n, seg_m;  // vertices and edges of every graph
};

// ---------------------------------------------------------------------------
// device graph: vertices relabelled by priority rank, rows sorted by rank
// ---------------------------------------------------------------------------
//
// Rank 0 is the vertex of highest priority p(x) = (degree, id) -- the order of
// the reference's vertex-priority counting (src/bfc/cpu_bfc.cpp:59-60).  A
// vertex's row lists its neighbours' ranks in ascending order, so "neighbours
// of lower priority than r" is the suffix of the row after r.  Edge ids stay
// the reference's ids (the msp tie rule compares them).
struct DevGraph {
    uint32_t n = 0, u_num = 0;
    uint64_t m = 0;
    uint32_t max_deg = 0;
    uint32_t max_deg_u = 0, max_deg_l = 0;  // largest degree of either side
    bool repeats = false;       // a row may hold a neighbour twice
    uint32_t *off = nullptr;    // n+1 row starts
    uint32_t *deg0 = nullptr;   // n   degree
    uint32_t *nbr0 = nullptr;   // 2m  neighbour rank, ascending per row
    uint32_t *eid0 = nullptr;   // 2m  reference edge id of each slot
    uint2 *ends = nullptr;      // m   (rank of U end, rank of V end) per edge id
    uint32_t *is_u = nullptr;   // n   1 if the rank's vertex is on the U side
    uint64_t tab_buckets = 0;  // row table buckets of the peel (32 bytes each)
    // batched arena: ranks are grouped by graph; seg_base[r] = first rank of
    // r's graph (NULL for one graph); cnt_span = vertices of the largest graph
    uint32_t *seg_base = nullptr;
    // every graph's ranks [v0, v0 + n) and edges [e0, e0 + m) (one entry for one graph)
    struct Span {
        uint32_t v0, n, e0, m;
    };
    std::vector<Span> spans;
    uint32_t cnt_span = 0;
};

// 32-byte buckets of the peel's hash table of a row of d edges: 1.5 slots per
// edge, at least one of them free.
__host__ __device__ inline uint32_t bt_row_buckets(uint32_t d) { return (d + (d >> 1) + 4) >> 2; }

// ---------------------------------------------------------------------------
// device context
// ---------------------------------------------------------------------------

struct bt_ctx {
    int device = 0;
    int sm_count = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    uint64_t budget = 0;       // 0 = unlimited
    uint64_t used = 0;
    uint64_t peak = 0;         // high-water mark of `used`
    std::vector<std::pair<void *, uint64_t>> allocs;

    DevGraph g;
    bool has_graph = false;
    uint32_t u_max = 0, l_num = 0;

    // results of the last call (by reference edge id)
    uint64_t *sup = nullptr;     // m uint64 supports (ebfc)
    uint32_t *result = nullptr;  // m uint32 bitruss (hidx / msp)
    int last_result = 0;         // 0 none, 1 supports, 2 bitruss
    uint64_t last_count = 0, last_sup_max = 0;

    // scratch reused across calls
    void *scratch = nullptr;
    uint64_t scratch_bytes = 0;
    uint64_t zero_counters = 0;  // leading counters of the scratch known to be zero (bt_count.cu)

    double phase_ms[8] = {-1, -1, -1, -1, -1, -1, -1, -1};
    uint64_t stats[8] = {0};
    uint64_t work[12] = {0};  // msp work counters and phase times of the last call
    uint64_t prof[8] = {0};   // msp: SM cycles per CTA by step (3 walking, 6 at barriers, 7 the rest)
    cudaEvent_t ev[8] = {};
    uint64_t *host_words = nullptr;  // 4 page-locked words: a count's results come back without a staging copy

    // msp task schedule (0 = built-in value): positions per 32 tasks, chunks per CTA, whole-plan limit
    uint32_t msp_schedule[3] = {0, 0, 0};
    uint64_t arena_edges = 1ull << 28;  // batched calls: edges per arena, at most
    uint32_t peel_ctas = 0;             // CTAs of the peeling kernel (0 = one per SM)
};

// Counters of one thread of the peel (a warp's positions are its first lane's).
// They pass 2^32: the 10M-edge hub graph walks 1.4e12 positions, 4.5e9 a warp on an
// eighth of the SMs.  In 64 bits they cost the kernel 16 bytes of spills, so
// each keeps 31 and a task's end carries what is above to the totals.  A task
// adds less than 2^31 to each.
struct PeelWork {
    uint32_t probes = 0, hits = 0, decs = 0;
    __host__ __device__ bool full() const { return (probes | hits | decs) >> 31; }
    // totals: the sums in 64 bits, which add(address, value) adds to
    template <class S, class Add>
    __host__ __device__ void carry(S &totals, Add add) {
        add(&totals.w_probes, probes & 0x80000000u);
        add(&totals.w_hits, hits & 0x80000000u);
        add(&totals.w_decs, decs & 0x80000000u);
        probes &= 0x7fffffffu;
        hits &= 0x7fffffffu;
        decs &= 0x7fffffffu;
    }
};

// Default msp task schedule (bt_ctx_set_msp_schedule with 0 picks these):
// probe positions per 32 tasks, frontier chunks per CTA, whole-plan limit.
constexpr uint32_t kMspMinGrain = 2048;
constexpr uint32_t kMspTasksPerCta = 2;
constexpr uint32_t kMspLocalPlan = 512;

enum { PH_UPLOAD = 0, PH_EBFC = 1, PH_PEEL = 2, PH_HIDX = 3, PH_TOTAL = 4, PH_MSP = 5 };

// device arena (tracked against the context's budget)
bt_status ctx_alloc(bt_ctx *ctx, void **p, uint64_t bytes);
void ctx_free(bt_ctx *ctx, void *p);
template <class T>
bt_status ctx_alloc_t(bt_ctx *ctx, T **p, uint64_t count) {
    return ctx_alloc(ctx, reinterpret_cast<void **>(p), count * sizeof(T));
}
bt_status ctx_scratch(bt_ctx *ctx, uint64_t bytes, void **p);

// Device buffers of one call, given back when it ends, also by an exception.
class CtxBuffers {
public:
    explicit CtxBuffers(bt_ctx *ctx) : ctx_(ctx) {}
    ~CtxBuffers() {
        for (void *p : held_) ctx_free(ctx_, p);
    }
    CtxBuffers(const CtxBuffers &) = delete;
    CtxBuffers &operator=(const CtxBuffers &) = delete;
    template <class T>
    bt_status alloc(T **p, uint64_t bytes) {
        held_.push_back(nullptr);  // may throw: before there is anything to lose
        void *q = nullptr;
        const bt_status s = ctx_alloc(ctx_, &q, bytes);
        held_.back() = q;
        *p = static_cast<T *>(q);
        return s;
    }

private:
    bt_ctx *ctx_;
    std::vector<void *> held_;
};
void ctx_release_graph(bt_ctx *ctx);

// Middle vertices whose wedges the counting kernel lays end to end at once, at
// most, and the positions its warps go on by.
constexpr uint32_t kCountBatch = 1024, kCountStride = 4096;

// As many of them as can be laid end to end where no row is longer: positions are
// 32-bit numbers, also the one a warp reaches past the last.  (With repeated
// lines the rows of a batch may all be the longest.)
inline uint32_t bt_count_batch(uint32_t longest_row) {
    const uint64_t fit = (0xffffffffull - kCountStride) / (longest_row + 1ull);
    return fit < 1 ? 1 : fit < kCountBatch ? (uint32_t)fit : kCountBatch;
}

// most bytes the counting kernel's scratch takes (bt_count.cu)
uint64_t bt_count_bytes(uint64_t m, uint64_t span, uint64_t ctas, bool wide);

// Butterflies of one graph given by ranks, its rows in any order and without a
// neighbour twice, on one CTA per SM with counters in shared memory only; every
// buffer is the caller's and nothing is allocated.  rows holds each rank's first
// slot and degree (below n, n < 2^31), the rows one after the other; nbr has `slots`
// entries.  Where the tables are not those of a graph the count
// is wrong, but nothing outside them is read.
// *next_chunk is zero on entry; nothing is counted if *skip is not (bt_count.cu).
// The set-up is made once per device and context.
bt_status bt_count_any_order_setup();
bt_status bt_count_any_order(uint32_t n, uint32_t slots, const uint2 *rows, const uint32_t *nbr,
                             unsigned long long *count, uint32_t *next_chunk, uint32_t *skip, int sms, cudaStream_t st);

// A graph of a batch as its peel's plan sees it, estimates of its peel (the chain
// of sub-rounds, and what CTAs share, in microseconds of one), and the sizes of the
// teams of CTAs that take the graphs in the order given (bt_plan.cpp).
struct PeelJob {
    uint64_t edges, butterflies;
};
double bt_peel_chain_us(const PeelJob &j);
double bt_peel_walk_us(const PeelJob &j);
std::vector<uint32_t> bt_plan_teams(const std::vector<PeelJob> &jobs, uint32_t ctas);

// algorithm entry points implemented in the .cu files
bt_status dev_build_graph(bt_ctx *ctx, const bt_graph *g);
bt_status dev_ebfc(bt_ctx *ctx, bool per_edge, uint64_t *count);
bt_status dev_msp(bt_ctx *ctx, bool exact, uint32_t *levels);
bt_status dev_hidx(bt_ctx *ctx, uint32_t *rounds);
