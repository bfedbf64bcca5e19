// bt_noalloc.cu -- global butterfly count that allocates no device memory.
//
// For callers that may not allocate on the device: plugin hosts that own the
// whole device heap and only hand buffers in, and latency-sensitive paths
// where a cudaMalloc / cudaFree (which can synchronise the device) is not
// acceptable.  The caller passes the graph and the output in its own device
// buffers; the wedge counters this count needs live in one file-scope device
// array, so nothing is allocated per call.
//
// Scratch: g_noalloc_scratch, kScratchWords 32-bit words (32 MiB).  Every GPU
// that loads this library holds it until the process exits.  Two ways to use it:
//  * Ranks.  The vertices are numbered by descending degree (a counting sort
//    over the degrees; which of two equal ones comes first does not matter to
//    the count, any strict order will do) and the rows copied with these numbers,
//    unsorted: 6n + 2m words.  The counting kernel then tests a neighbour's
//    priority by comparing two numbers it has in hand, keeps its counters in
//    shared memory and runs on every SM; each 52k vertices past the first cost
//    the large start vertices one more pass over their wedges.  For graphs that
//    fit, of at least kRankEdges edges: six kernels in a row take 40 us, so below
//    them the other way is as fast (16k edges: 44-53 us by ranks, 33-61 us by
//    counters; 25k: 49-55 and 44-88 us).
//  * Counters.  Each CTA uses 2n words (a wedge counter and a touched list per
//    vertex), so the count runs on min(2 per SM, kScratchWords / 2n) CTAs; every
//    priority test reads two row offsets.  Also for what the ranks' kernels find
//    on the way to be no graph in the layout (below): a flag on the device
//    chooses, no host read.
// Graphs of more than kScratchWords / 2 vertices are rejected.  The last 64
// words hold the work counters and the flag.
// Measured, by counters and by ranks: 300k edges on 69k vertices (skewed) 1,822
// and 243 us; 300k on 176k vertices 9,600 and 282 us; 1M on 140k 9,918 and 1,037
// us; 1M on 641k 117,028 and 1,142 us.  By counters the bound is the few CTAs
// that the scratch has room for (60 at 69k vertices, 6 at 641k) and two offset
// loads per wedge; by ranks it is the wedges' shared-memory atomics.
//
// All calls share the array: calls that overlap on the GPU (on different
// streams or threads, without ordering between them) race on it and give
// wrong counts, but touch nothing outside the array and the callers' buffers:
// an index that comes from the array is compared with its range before it is
// used, loops end whatever the array holds, and a block takes a branch that has
// block barriers behind it on one answer for all its threads.  The array keeps
// the last call's contents; each call clears the parts that must start at zero
// (its counters and the work counter).
//
// The first call on a device looks up the array's device address with
// cudaGetSymbolAddress (the host-side name of a __device__ array is only a
// stand-in); that set-up runs once per device and context, with the device
// current, and that first call should come before any stream capture.  The
// address is cached together with the CUDA context it belongs to: after the
// caller resets the device (cudaDeviceReset) the next call sees a new context
// and looks the address up again, so it never launches on a stale pointer.
//
// The call makes `device` current only for its own work and restores the
// caller's current device before it returns, on every path.
//
// Arithmetic: the vertex-priority count of the reference's bfc_kernel
// (src/bfc/bfc_vpp.cu:33-107) on the reference CSR layout (rows sorted by
// vertex id, priority p(x) = (degree, id) tested per neighbour).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "bt_device.cuh"

namespace {

constexpr uint64_t kScratchWords = 8ull << 20;  // 32 MiB
constexpr uint64_t kCounterWords = 64;          // work counter at the end
constexpr uint64_t kRankEdges = 24'576;
constexpr int kMaxDevices = 64;
constexpr int kThreadsNA = 512;

__device__ __align__(256) uint32_t g_noalloc_scratch[kScratchWords + kCounterWords];

uint32_t *g_scratch_addr[kMaxDevices];
CUcontext g_scratch_ctx[kMaxDevices];  // context the cached address belongs to
std::mutex g_scratch_mutex;

// The caller's current device, put back when the scope ends.
struct DeviceGuard {
    int saved = -1;
    DeviceGuard() {
        if (cudaGetDevice(&saved) != cudaSuccess) saved = -1;
    }
    ~DeviceGuard() {
        if (saved >= 0) cudaSetDevice(saved);
    }
    DeviceGuard(const DeviceGuard &) = delete;
    DeviceGuard &operator=(const DeviceGuard &) = delete;
};

// The current CUDA context, through the driver entry point the runtime hands
// out (the library does not link the driver library itself).
bt_status current_context(CUcontext *out) {
    using GetCurrent = CUresult (*)(CUcontext *);
    // looked up once; a function-local static is initialised thread-safely
    static const GetCurrent fn = []() -> GetCurrent {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 4000, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
        return reinterpret_cast<GetCurrent>(p);
    }();
    if (!fn) return bt_fail(BT_ERR_CUDA, "cuCtxGetCurrent is not available from the CUDA driver");
    *out = nullptr;
    if (fn(out) != CUDA_SUCCESS || !*out) return bt_fail(BT_ERR_CUDA, "no current CUDA context");
    return BT_OK;
}

__device__ __forceinline__ bool higher(const uint32_t *off, uint32_t a, uint32_t b) {
    const uint32_t da = off[a + 1] - off[a], db = off[b + 1] - off[b];
    return da > db || (da == db && a > b);
}

// scratch: per CTA cnt[n] then touched[n]; counter[0] = next vertex.  Does
// nothing if only_if is given and zero.
__global__ void __launch_bounds__(kThreadsNA) k_bfc_noalloc(uint32_t n, const uint32_t *off, const uint32_t *nbr,
                                                            uint32_t *scratch, uint32_t *counter,
                                                            const uint32_t *only_if, unsigned long long *count) {
    __shared__ uint32_t s_r, s_nt;
    __shared__ unsigned long long s_red[kThreadsNA / 32];
    if (only_if && !__syncthreads_or(*only_if != 0)) return;
    uint32_t *cnt = scratch + (size_t)blockIdx.x * 2 * n;
    uint32_t *touched = cnt + n;
    for (uint32_t x = threadIdx.x; x < n; x += blockDim.x) cnt[x] = 0;  // left over from the last call
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned long long local = 0;
    for (;;) {
        if (threadIdx.x == 0) {
            s_r = atomicAdd(counter, 1u);
            s_nt = 0;
        }
        __syncthreads();
        const uint32_t u = s_r;
        if (u >= n) break;
        for (uint32_t i = off[u] + warp; i < off[u + 1]; i += nw) {
            const uint32_t v = nbr[i];
            if (!higher(off, u, v)) continue;
            for (uint32_t j = off[v] + lane; j < off[v + 1]; j += 32) {
                const uint32_t w = nbr[j];
                if (!higher(off, u, w)) continue;
                const uint32_t old = atomicAdd(cnt + w, 1u);
                local += old;
                if (old == 0) {
                    const uint32_t at = atomicAdd(&s_nt, 1u);
                    if (at < n) touched[at] = w;
                }
            }
        }
        __syncthreads();
        const uint32_t nt = min(s_nt, n);
        for (uint32_t k = threadIdx.x; k < nt; k += blockDim.x) {
            const uint32_t w = touched[k];
            if (w < n) cnt[w] = 0;
        }
        __syncthreads();
    }
    for (int o = 16; o; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (lane == 0) s_red[warp] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (uint32_t k = 0; k < nw; k++) t += s_red[k];
        if (t) atomicAdd(count, t);
    }
}

// ---- ranks ------------------------------------------------------------------

// Work counters and flags at the end of the scratch, zeroed by each call.
struct Words {
    uint32_t next_vertex, largest, next_chunk, irregular;
};
static_assert(sizeof(Words) <= kCounterWords * 4, "fits");

// The ranks' tables in the scratch: n words each, and the 2m slots of the rows.
struct Ranks {
    uint32_t *bins;   // per degree: its vertices, then the rank of the first (zero on entry)
    uint32_t *taken;  // per degree: ranks given out (zero on entry)
    uint32_t *slots;  // per degree: first row slot
    uint32_t *rank;
    uint2 *rows;      // per rank: first row slot, degree (2n words)
    uint32_t *nbr;
};

// Vertices per degree and the largest degree.  The later kernels' indexes rest
// on what is tested here: every degree is below n, and the rows fill [0, 2m).
__global__ void k_na_degrees(uint32_t n, uint64_t m, const uint32_t *off, Ranks t, Words *w) {
    uint32_t most = 0;
    bool bad = off[0] != 0 || off[n] != 2 * m;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
        const uint32_t d = off[x + 1] - off[x];
        if (d < n) {
            // the lanes of one degree add together: most vertices share a few
            const uint32_t same = __match_any_sync(__activemask(), d);
            if ((threadIdx.x & 31) == (uint32_t)__ffs(same) - 1) atomicAdd(t.bins + d, (uint32_t)__popc(same));
            most = d > most ? d : most;
        } else {
            bad = true;
        }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0 && most) atomicMax(&w->largest, most);
    if (bad) w->irregular = 1;
}

// Per degree, the first rank and the first row slot of its vertices, largest
// degree first; one block.
__global__ void __launch_bounds__(1024) k_na_scan(uint32_t n, Ranks t, const Words *w) {
    __shared__ unsigned long long s_warp[32];
    __shared__ uint32_t s_top;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_top = min(w->largest, n - 1);
    if (__syncthreads_or(w->irregular != 0)) return;
    const uint32_t top = s_top;
    unsigned long long run = 0;
    for (uint32_t i0 = 0; i0 <= top; i0 += 1024) {
        const uint32_t i = i0 + threadIdx.x, d = top - i;  // degrees downwards
        const uint32_t c = i <= top ? t.bins[d] : 0;
        // vertices in the low half, row slots in the high half
        const unsigned long long own = c | (unsigned long long)(i <= top ? c * d : 0) << 32;
        unsigned long long v = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long p = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= (uint32_t)o) v += p;
        }
        if (lane == 31) s_warp[warp] = v;
        __syncthreads();
        unsigned long long u = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long p = __shfl_up_sync(0xffffffffu, u, o);
            if (lane >= (uint32_t)o) u += p;
        }
        const unsigned long long before = __shfl_sync(0xffffffffu, u, warp ? warp - 1 : 0);
        const unsigned long long ex = run + (warp ? before : 0) + v - own;
        if (i <= top) {
            t.bins[d] = (uint32_t)ex;
            t.slots[d] = (uint32_t)(ex >> 32);
        }
        run += __shfl_sync(0xffffffffu, u, 31);
        __syncthreads();
    }
}

// Every vertex's rank, and its rank's row start and degree.
__global__ void k_na_rank(uint32_t n, const uint32_t *off, Ranks t, const Words *w) {
    if (w->irregular) return;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < n; x += gridDim.x * blockDim.x) {
        const uint32_t d = off[x + 1] - off[x];
        if (d >= n) continue;
        // the lanes of one degree take their ranks together
        const uint32_t on = __activemask(), same = __match_any_sync(on, d);
        const uint32_t lane = threadIdx.x & 31, lead = __ffs(same) - 1;
        uint32_t k = 0;
        if (lane == lead) k = atomicAdd(t.taken + d, (uint32_t)__popc(same));
        k = __shfl_sync(same, k, lead) + __popc(same & ((1u << lane) - 1));
        const uint32_t r = t.bins[d] + k;
        if (r >= n) continue;
        t.rank[x] = r;
        t.rows[r] = make_uint2(t.slots[d] + k * d, d);
    }
}

// The rows with ranks in place of vertices; one thread per slot (a warp per row
// waits for the longest: 100 us of the 300k-edge graph's 314, now 15).  Rows that
// do not ascend strictly may hold a neighbour twice: then the order of equal
// degrees matters to the count, and the other way keeps it by vertex id.
__global__ void k_na_rows(uint32_t n, const uint32_t *off, const uint32_t *nbr, uint64_t slots, Ranks t, Words *w) {
    if (w->irregular) return;
    bool bad = false;
    for (uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; p < slots; p += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t y = nbr[p], before = p ? nbr[p - 1] : 0;
        const uint32_t x = bt::row_of_slot(off, n, (uint32_t)p), j = (uint32_t)p - off[x];
        if (y >= n || (j && before >= y)) bad = true;
        const uint32_t r = t.rank[x];
        const uint64_t dst = r < n ? (uint64_t)t.rows[r].x + j : slots;
        if (dst < slots) t.nbr[dst] = y < n ? t.rank[y] : 0;
    }
    if (bad) w->irregular = 1;
}

// Device address of the scratch array on the current device: looked up once
// per device and context (`device` is current: cudaSetDevice has created or
// bound its primary context).
bt_status scratch_address(int device, uint32_t **out) {
    if (device < 0 || device >= kMaxDevices) return bt_fail(BT_ERR_INVALID, "device index out of range");
    CUcontext cur = nullptr;
    BT_TRY(current_context(&cur));
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_ctx[device] != cur) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return bt_cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
        // load every kernel a later call may launch, so that a captured call loads none
        cudaFuncAttributes fa;
        for (const void *k : {(const void *)k_bfc_noalloc, (const void *)k_na_degrees, (const void *)k_na_scan,
                              (const void *)k_na_rank, (const void *)k_na_rows})
            BT_CUDA(cudaFuncGetAttributes(&fa, k));
        BT_TRY(bt_count_any_order_setup());
        g_scratch_addr[device] = static_cast<uint32_t *>(p);
        g_scratch_ctx[device] = cur;
    }
    *out = g_scratch_addr[device];
    return BT_OK;
}

}  // namespace

extern "C" bt_status bt_bfc_noalloc(int device, const uint32_t *d_offsets, const uint32_t *d_neighbors,
                                    uint32_t n, uint64_t m, unsigned long long *d_count, void *stream) {
    if (!d_offsets || !d_count || (m && !d_neighbors)) return bt_fail(BT_ERR_INVALID, "null argument");
    if ((uint64_t)n > kScratchWords / 2)
        return bt_fail(BT_ERR_INVALID, "bt_bfc_noalloc: " + std::to_string(n) +
                                           " vertices exceed the scratch limit of " +
                                           std::to_string(kScratchWords / 2) + " vertices");
    if (m > 0x7fffffffull) return bt_fail(BT_ERR_INVALID, "edge count exceeds the 32-bit CSR offsets");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
        return bt_fail(BT_ERR_NO_DEVICE, "gpu device id " + std::to_string(device) + " is not available");
    DeviceGuard restore;  // the caller's current device comes back on every return
    BT_CUDA(cudaSetDevice(device));
    uint32_t *scratch = nullptr;
    BT_TRY(scratch_address(device, &scratch));
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t *counter = scratch + kScratchWords;
    BT_CUDA(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), st));
    if (n == 0) return BT_OK;
    BT_CUDA(cudaMemsetAsync(counter, 0, kCounterWords * sizeof(uint32_t), st));
    int sms = 0;
    BT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    Words *words = reinterpret_cast<Words *>(counter);
    const bool by_rank = m >= kRankEdges && 6ull * n + 2 * m <= kScratchWords;
    if (by_rank) {
        uint32_t *p = scratch;
        const Ranks t{p, p + n, p + 2ull * n, p + 3ull * n, reinterpret_cast<uint2 *>(p + 4ull * n), p + 6ull * n};
        BT_CUDA(cudaMemsetAsync(t.bins, 0, 8ull * n, st));  // and taken
        const unsigned most = (unsigned)sms * 8, per_vertex = std::min(most, (n + 255) / 256);
        const unsigned per_slot = (unsigned)std::min<uint64_t>(most, (2 * m + 255) / 256);
        k_na_degrees<<<per_vertex, 256, 0, st>>>(n, m, d_offsets, t, words);
        k_na_scan<<<1, 1024, 0, st>>>(n, t, words);
        k_na_rank<<<per_vertex, 256, 0, st>>>(n, d_offsets, t, words);
        k_na_rows<<<per_slot, 256, 0, st>>>(n, d_offsets, d_neighbors, 2 * m, t, words);
        bt_note_launches(4);
        BT_CUDA(cudaGetLastError());
        BT_TRY(bt_count_any_order(n, (uint32_t)(2 * m), t.rows, t.nbr, d_count, &words->next_chunk, &words->irregular, sms, st));
    }
    uint64_t ctas = (uint64_t)sms * 2;
    const uint64_t fit = kScratchWords / (2ull * n);
    if (ctas > fit) ctas = fit;
    if (ctas > n) ctas = n;
    k_bfc_noalloc<<<(unsigned)ctas, kThreadsNA, 0, st>>>(n, d_offsets, d_neighbors, scratch, &words->next_vertex,
                                                        by_rank ? &words->irregular : nullptr, d_count);
    bt_note_launches(1);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}
