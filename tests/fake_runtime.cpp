// A CUDA runtime of host memory for tests of the library's host code (test_host_state_cpu.py): linked with
// the library's own objects in place of cudart.  Device and page-locked memory come from calloc and are
// counted against a total that a test sets, an allocation can be made to fail, a stream runs what it is
// given at once, and a capture keeps what it is given for the graph's launches.  Kernels do nothing, except
// that an epoch's kernels keep its counts: every agent cites one paper, itself.
#include <cxxabi.h>
#include <math.h>
#include <string.h>

#include <cmath>
#include <cstdlib>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace pg {
struct ErSkip;  // device code only
}
#include "../paragraph_gb300/csrc/pg_engine.cuh"
#include "../paragraph_gb300/csrc/pg_lik.cuh"

using pg::Arena;

namespace {
struct Block {
    size_t bytes;
    int kind;  // 0 device, 1 page-locked, 2 pool
};
size_t g_total = 64ull << 30;  // device memory
size_t g_used = 0;             // device allocations, and what the pool has reserved
size_t g_pool_used = 0, g_pool_reserved = 0;
uint64_t g_pool_keep = 0;
int64_t g_fail_in = -1;        // device allocations from now until they fail; < 0: they do not
int64_t g_mallocs = 0, g_queries = 0;
int64_t g_ball = 1;            // elements of every agent's ball
int64_t g_faults = 0;          // kernels that would have read through a null pointer
int g_sms = 152;
std::map<uintptr_t, Block> g_blocks;
std::map<const void*, std::string> g_kernels;
std::vector<std::function<void()>>* g_capture = nullptr;
struct Launch {
    std::string name;
    long long grid, block;
    int attrs;
};
std::vector<Launch> g_launches;

void submit(std::function<void()> f) {
    if (g_capture)
        g_capture->push_back(std::move(f));
    else
        f();
}

bool fails() {
    ++g_mallocs;
    if (g_fail_in > 0) return g_fail_in--, false;
    return g_fail_in == 0;
}

void* take(size_t bytes, int kind) {
    void* p = calloc(bytes ? bytes : 1, 1);
    g_blocks[(uintptr_t)p] = Block{bytes, kind};
    return p;
}

void drop(void* p) {
    if (!p) return;
    auto it = g_blocks.find((uintptr_t)p);
    if (it == g_blocks.end()) abort();
    if (it->second.kind == 0) g_used -= it->second.bytes;
    if (it->second.kind == 2) g_pool_used -= it->second.bytes;
    g_blocks.erase(it);
    free(p);
}

// ---- the kernels of an epoch that keep its counts
void epoch_begin(const Arena& A, int64_t epoch, int64_t delta) {
    int64_t at = 0;
    A.st->epoch = epoch;
    for (int r = 0; r < A.R; ++r) {
        pg::Replica& rp = A.rep[r];
        rp.delta = delta >= 0 ? (r == 0 ? delta : 0)
                              : (rp.growth_rate > 0.0 ? (int64_t)std::ceil((double)rp.n * rp.growth_rate) : rp.fixed_new);
        rp.abase = at;
        at += rp.delta;
    }
    A.st->agents = at;
}
void copy_out(const Arena& A, int64_t agents) {
    if (!A.out_src) return;
    if ((int64_t)A.st->out_count + agents > A.out_cap) {
        A.st->out_short += (unsigned long long)agents;
        return;
    }
    for (int r = 0; r < A.R; ++r) {
        const pg::Replica& rp = A.rep[r];
        A.out_counts[A.st->cum_epochs * A.R + r] = rp.delta;
        for (int64_t i = 0; i < rp.delta; ++i) {
            A.out_src[A.st->out_count + rp.abase + i] = (int32_t)(rp.n + i);
            A.out_dst[A.st->out_count + rp.abase + i] = (int32_t)(rp.n + i);
        }
    }
}
void epoch_end(const Arena& A, int64_t agents) {
    if (agents != A.st->agents) A.st->error |= pg::kErrArg;  // launched for another number of agents
    for (int r = 0; r < A.R; ++r) {
        A.rep[r].m += A.rep[r].delta;
        A.rep[r].n += A.rep[r].delta;
    }
    A.st->edges = A.st->agents;
    A.st->cum_epochs += 1;
    A.st->cum_edges += (unsigned long long)A.st->agents;
    A.st->cum_new_nodes += (unsigned long long)A.st->agents;
    if (A.out_src && (int64_t)A.st->out_count + A.st->agents <= A.out_cap) A.st->out_count += (unsigned long long)A.st->agents;
}
void copy_segments(const pg::CopySeg* s, int num, pg::EpochState* st) {
    if (!s) {
        ++g_faults;
        return;
    }
    for (int i = 0; i < num; ++i) {
        if (s[i].src)
            memcpy(s[i].dst, s[i].src, (size_t)s[i].bytes);
        else
            memset(s[i].dst, 0, (size_t)s[i].bytes);
    }
    st->error = 0;
}

cudaError_t launch(const void* f, dim3 grid, dim3 block, void** args, int attrs) {
    const std::string& name = g_kernels[f];
    auto is = [&](const char* k) { return name.find(std::string("pg::") + k + "(") != std::string::npos; };
    const long long threads = (long long)block.x * block.y * block.z;
    g_launches.push_back(Launch{name, (long long)grid.x * grid.y * grid.z, threads, attrs});
    if (is("k_epoch_begin")) {
        const Arena A = *(Arena*)args[0];
        const int64_t e = *(int64_t*)args[1], d = *(int64_t*)args[2];
        submit([=]() { epoch_begin(A, e, d); });
    } else if (is("k_copy_out") || is("k_epoch_end")) {
        const Arena A = *(Arena*)args[0];
        const int64_t agents = *(int64_t*)args[1];
        const bool end = is("k_epoch_end");
        submit([=]() { end ? epoch_end(A, agents) : copy_out(A, agents); });
    } else if (is("k_rc_big")) {
        const Arena& A = *(Arena*)args[0];
        if (!A.rc_big_id || !A.rc_big_meta || !A.rc_part || !A.rc_item || !A.rc_item_list || !A.rc_item_meta || !A.rc_ticket)
            ++g_faults;
    } else if (name.find("pg::k_lik_ball<false>(") != std::string::npos) {
        const pg::LikBalls B = *(pg::LikBalls*)args[1];
        const int64_t a0 = *(int64_t*)args[2], a1 = *(int64_t*)args[3];
        for (int64_t a = a0; a < a1; ++a) B.cnt[a] = g_ball;
    } else if (is("k_copy_segments")) {
        const pg::CopySeg* s = *(pg::CopySeg**)args[0];
        const int num = *(int*)args[1];
        pg::EpochState* st = *(pg::EpochState**)args[3];
        submit([=]() { copy_segments(s, num, st); });
    }
    return cudaSuccess;
}
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;
}  // namespace

extern "C" {
// ---- for the tests
void fake_reset(int64_t total_bytes, int32_t sms) {
    g_total = (size_t)total_bytes;
    g_sms = sms;
    g_fail_in = -1;
    g_mallocs = g_queries = g_faults = 0;
    g_launches.clear();
}
void fake_fail_in(int64_t n) { g_fail_in = n; }
void fake_ball(int64_t elements) { g_ball = elements; }
int64_t fake_mallocs(void) { return g_mallocs; }
int64_t fake_faults(void) { return g_faults; }
int64_t fake_memory_queries(void) { return g_queries; }
int64_t fake_free_bytes(void) { return (int64_t)(g_total - g_used); }
int64_t fake_pool_idle(void) { return (int64_t)(g_pool_reserved - g_pool_used); }
int64_t fake_hold(int64_t bytes) {  // memory of another user of the device; negative: given back
    g_used += bytes;
    return (int64_t)g_used;
}
int32_t fake_launches(const char* kernel) {
    int32_t n = 0;
    for (const Launch& l : g_launches) n += l.name.find(kernel) != std::string::npos;
    return n;
}
void fake_clear_launches(void) { g_launches.clear(); }
// the largest dependent launch and the smallest plain one of the kernels named, in threads (0: none)
void fake_dependent_range(const char* kernel, int64_t* largest, int64_t* smallest) {
    *largest = *smallest = 0;
    for (const Launch& l : g_launches) {
        if (l.name.find(kernel) == std::string::npos) continue;
        const int64_t t = l.grid * l.block;
        if (l.attrs && t > *largest) *largest = t;
        if (!l.attrs && (*smallest == 0 || t < *smallest)) *smallest = t;
    }
}
void* fake_page_locked(int64_t bytes) { return take((size_t)bytes, 1); }
void fake_page_locked_free(void* p) { drop(p); }

// ---- the runtime
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    int st = 0;
    char* d = abi::__cxa_demangle(name, nullptr, nullptr, &st);
    g_kernels[host] = d ? d : name;
    free(d);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* s) {
    g_grid = grid, g_block = block, g_smem = smem, g_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
    *grid = g_grid, *block = g_block, *smem = g_smem, *(cudaStream_t*)s = g_stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void** args, size_t, cudaStream_t) {
    return launch((const void*)k, grid, block, args, 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return launch(f, c->gridDim, c->blockDim, args, (int)c->numAttrs);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void** args, size_t, cudaStream_t) {
    return launch(f, grid, block, args, 0);
}
cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorNotSupported; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? g_sms : 1;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaPeekAtLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake runtime error"; }

cudaError_t cudaMalloc(void** p, size_t n) {
    *p = nullptr;
    if (fails() || g_used + n > g_total) return cudaErrorMemoryAllocation;
    g_used += n;
    *p = take(n, 0);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    drop(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    ++g_queries;
    *f = g_total - g_used;
    *t = g_total;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = take(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    drop(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    auto it = g_blocks.upper_bound((uintptr_t)p);
    if (it == g_blocks.begin()) return cudaSuccess;
    --it;
    if ((uintptr_t)p < it->first + it->second.bytes && it->second.kind == 1) {
        a->type = cudaMemoryTypeHost;
        a->devicePointer = const_cast<void*>(p);
        a->hostPointer = const_cast<void*>(p);
    }
    return cudaSuccess;
}

// one pool, whose idle memory stays reserved until it is trimmed
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*) {
    static int h;
    *pool = (cudaMemPool_t)&h;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, enum cudaMemPoolAttr a, void* v) {
    *(uint64_t*)v = a == cudaMemPoolAttrReservedMemCurrent ? g_pool_reserved : a == cudaMemPoolAttrUsedMemCurrent ? g_pool_used : 0;
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep) {
    const size_t want = keep > g_pool_used ? keep : g_pool_used;
    if (g_pool_reserved > want) {
        g_used -= g_pool_reserved - want;
        g_pool_reserved = want;
    }
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    *p = nullptr;
    const size_t more = g_pool_used + n > g_pool_reserved ? g_pool_used + n - g_pool_reserved : 0;
    if (g_used + more > g_total) return cudaErrorMemoryAllocation;
    g_used += more;
    g_pool_reserved += more;
    g_pool_used += n;
    *p = take(n, 2);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    drop(p);
    return cudaSuccess;
}

cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind, cudaStream_t) {
    submit([=]() { memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    submit([=]() { memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemset2DAsync(void* d, size_t pitch, int v, size_t w, size_t h, cudaStream_t) {
    submit([=]() {
        for (size_t i = 0; i < h; ++i) memset((char*)d + i * pitch, v, w);
    });
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.0f;
    return cudaSuccess;
}

cudaError_t cudaStreamIsCapturing(cudaStream_t, enum cudaStreamCaptureStatus* s) {
    *s = g_capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) {
    g_capture = new std::vector<std::function<void()>>();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = (cudaGraph_t)g_capture;
    g_capture = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = (cudaGraphExec_t) new std::vector<std::function<void()>>(*(std::vector<std::function<void()>>*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete (std::vector<std::function<void()>>*)g;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    delete (std::vector<std::function<void()>>*)e;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    for (auto& f : *(std::vector<std::function<void()>>*)e) f();
    return cudaSuccess;
}
}  // extern "C"
