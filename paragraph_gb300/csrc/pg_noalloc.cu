// pg_noalloc.cu -- G(n,p) edge generation that allocates no device memory.
//
// Some callers cannot allocate device memory when they call this library -- for instance a host
// program that must not call cudaMalloc while other work on the device is being timed or captured,
// or a runtime that hands out pre-sized buffers and forbids allocation inside its callbacks.  For
// them this file provides one entry point that generates an Erdos-Renyi epoch's edge list into
// buffers the caller already owns.  Its only scratch (per-task edge counts, their exclusive scan
// and the scan's block sums, each in its own region) lives in a fixed file-scope __device__ array,
// so no cudaMalloc, cudaFree or allocating library routine is ever called.
//
// The edges are the ones pg_er_epoch appends for the same (seed, epoch, n_existing, delta, p):
// the same Philox streams, the same 2^16-id chunks, the same library log, the same
// (source, target) order.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>

#include "../../include/paragraph_gb300.h"
#include "pg_engine.cuh"

namespace pg {
namespace {

constexpr int64_t kNoAllocMaxTasks = PG_NOALLOC_MAX_TASKS;
constexpr int64_t kNoAllocBlocks = (kNoAllocMaxTasks + 1023) / 1024 + 2;

// Three regions: per-task counts [kNoAllocMaxTasks], their exclusive scan [kNoAllocMaxTasks + 1]
// (entry [tasks] = total) and the scan's block sums.  Every GPU that loads the library holds this
// array (about 4 MiB) until the process exits.
constexpr int64_t kNoAllocWords = 2 * kNoAllocMaxTasks + 1 + kNoAllocBlocks;
static __device__ __align__(256) int64_t g_noalloc_scratch[kNoAllocWords];

// Device address of the array, looked up once per device; several host threads may call.
std::atomic<int64_t*> g_scratch_addr[64] = {};

// Every task by a group of G lanes, twice: the counting pass leaves each task's number of edges, the
// writing pass (out_src set) walks again from the scanned offsets.  Walking is cheaper than keeping:
// no room is needed for edges whose number is not yet known.  A call's time is that of a few dependent
// launches; a lane walking a task alone took one gap after another (18.5 us for each pass over
// 1,017 x 2 tasks of up to 6.5 edges, now 6.9; the call 87 us, now 53).
template <int G>
__global__ void __launch_bounds__(256) k_na_walk(uint64_t seed, uint32_t ep, int64_t n, int64_t tasks, int64_t chunks,
                                                 ErSkip K, int64_t* cnt, const int64_t* off, int32_t* out_src,
                                                 int32_t* out_dst, int64_t capacity) {
    if (out_src && off[tasks] > capacity) return;  // reported by the host: nothing is written
    constexpr int per = 32 / G;  // tasks per warp and round
    const int gl = lane_id() & (G - 1);
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t0 = warp * per; t0 < tasks; t0 += nwarps * per) {
        const int64_t t = t0 + lane_id() / G;
        const bool live = t < tasks;
        const int64_t i = (live ? t : 0) / chunks, c = (live ? t : 0) % chunks;
        const int64_t lo = c * kErChunk;
        const int len = (int)(lo + kErChunk < n ? kErChunk : n - lo);
        int64_t k = out_src && live ? off[t] : 0;
        bool act = live;
        int pos = -1;
        for (uint32_t b = 0; __any_sync(0xffffffffu, act); b += G) {
            int q0, q1;
            const int got = er_round<G>(seed, ep, i, c, K, b, act, len, pos, q0, q1);
            if (out_src && act) {
                const int64_t e = k + 2 * gl;
                if (q0 < len) {
                    out_src[e] = (int32_t)(n + i);
                    out_dst[e] = (int32_t)(lo + q0);
                }
                if (q1 < len) {
                    out_src[e + 1] = (int32_t)(n + i);
                    out_dst[e + 1] = (int32_t)(lo + q1);
                }
            }
            k += got;
            if (got < 2 * G) act = false;
        }
        if (!out_src && live && gl == 0) cnt[t] = k;
    }
}

void launch_walk(int G, uint64_t seed, uint32_t ep, int64_t n, int64_t tasks, int64_t chunks, const ErSkip& K,
                 int64_t* cnt, const int64_t* off, int32_t* src, int32_t* dst, int64_t capacity, cudaStream_t st) {
    int64_t g = (tasks * G + 255) / 256;
    if (g > 4096) g = 4096;
    const unsigned grid = (unsigned)g;
    switch (G) {
        case 1: k_na_walk<1><<<grid, 256, 0, st>>>(seed, ep, n, tasks, chunks, K, cnt, off, src, dst, capacity); break;
        case 2: k_na_walk<2><<<grid, 256, 0, st>>>(seed, ep, n, tasks, chunks, K, cnt, off, src, dst, capacity); break;
        case 4: k_na_walk<4><<<grid, 256, 0, st>>>(seed, ep, n, tasks, chunks, K, cnt, off, src, dst, capacity); break;
        case 8: k_na_walk<8><<<grid, 256, 0, st>>>(seed, ep, n, tasks, chunks, K, cnt, off, src, dst, capacity); break;
        case 16: k_na_walk<16><<<grid, 256, 0, st>>>(seed, ep, n, tasks, chunks, K, cnt, off, src, dst, capacity); break;
        default: k_na_walk<32><<<grid, 256, 0, st>>>(seed, ep, n, tasks, chunks, K, cnt, off, src, dst, capacity); break;
    }
}

// Device address of the scratch array for the current device (set up once per device).
pg_status scratch_for_current_device(int64_t** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return PG_ERR_CUDA;
    int64_t* a = g_scratch_addr[dev].load(std::memory_order_acquire);
    if (!a) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return PG_ERR_CUDA;
        a = static_cast<int64_t*>(p);
        g_scratch_addr[dev].store(a, std::memory_order_release);  // every thread stores the same value
    }
    *out = a;
    return PG_OK;
}

}  // namespace
}  // namespace pg

extern "C" pg_status pg_er_generate_noalloc(uint64_t seed, int64_t epoch, int64_t n_existing,
                                            int64_t delta, double p, int32_t* d_src,
                                            int32_t* d_dst, int64_t capacity, int64_t* num_edges,
                                            void* stream) {
    using namespace pg;
    if (!num_edges) return PG_ERR_ARG;
    *num_edges = 0;
    if (n_existing <= 0 || n_existing > (int64_t)INT32_MAX / 2 || delta <= 0 || std::isnan(p) ||
        capacity < 0 || (capacity > 0 && (!d_src || !d_dst)))
        return PG_ERR_ARG;
    if (n_existing + delta > (int64_t)INT32_MAX) return PG_ERR_ARG;
    const int64_t chunks = (n_existing + kErChunk - 1) / kErChunk;
    if (delta > kNoAllocMaxTasks / chunks) return PG_ERR_CAPACITY;  // scratch holds one count per task
    const int64_t tasks = delta * chunks;
    if (!(p > 0.0)) return PG_OK;  // no edges
    const ErSkip K = er_skip_constants(p);
    int64_t* scratch = nullptr;
    pg_status s = scratch_for_current_device(&scratch);
    if (s != PG_OK) return s;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int64_t* cnt = scratch;                          // [tasks]
    int64_t* off = scratch + kNoAllocMaxTasks;        // [tasks + 1], exclusive scan of cnt
    int64_t* blocksum = off + kNoAllocMaxTasks + 1;   // [scan blocks + 1]
    const uint32_t ep = (uint32_t)epoch;
    const int G = er_lanes(n_existing, p);
    launch_walk(G, seed, ep, n_existing, tasks, chunks, K, cnt, nullptr, nullptr, nullptr, 0, st);
    launch_scan_i64(cnt, off, tasks, blocksum, st);
    // the writing pass looks at the total itself, so that it need not wait for the host to have seen it
    if (capacity > 0)
        launch_walk(G, seed, ep, n_existing, tasks, chunks, K, cnt, off, d_src, d_dst, capacity, st);
    if (cudaGetLastError() != cudaSuccess) return PG_ERR_CUDA;  // *num_edges stays 0
    int64_t total = 0;
    if (cudaMemcpyAsync(&total, off + tasks, sizeof(int64_t), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return PG_ERR_CUDA;
    *num_edges = total;
    return total > capacity ? PG_ERR_CAPACITY : PG_OK;  // over capacity: nothing written
}
