// Context, error plumbing, device-memory helpers, scans and BLAS-1 kernels.
#include "hn_internal.cuh"

#include <cuda.h>

#include <cstring>
#include <map>
#include <vector>

namespace hn {

namespace {
thread_local std::string g_last_error;
Context g_ctx;
}  // namespace

void set_last_error(const std::string& msg) { g_last_error = msg; }

void fail(int status, const std::string& msg) { throw Error(status, msg); }

void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        cudaGetLastError();
        fail(e == cudaErrorMemoryAllocation ? HN_ERR_OUT_OF_MEMORY : HN_ERR_CUDA,
             std::string(what) + ": " + cudaGetErrorString(e));
    }
}

void launched(const char* what) {
    g_ctx.launches.fetch_add(1, std::memory_order_relaxed);
    check_cuda(cudaGetLastError(), what);
}

Context& ctx() { return g_ctx; }

void require_init() {
    if (g_ctx.device < 0) fail(HN_ERR_NOT_INITIALIZED, "hn_init has not been called");
    int cur = -1;
    check_cuda(cudaGetDevice(&cur), "cudaGetDevice");
    if (cur != g_ctx.device) check_cuda(cudaSetDevice(g_ctx.device), "cudaSetDevice");
}

// ---------------------------------------------------------------- device memory
// Setting a model up makes about 70 short-lived allocations, and solving it 30
// more; cudaMalloc and cudaFree of those took 13 of the 14.4 ms of a
// 20,000-row set-up. Freed blocks are kept for the next request that needs at
// least 4/5 of one: at most kPoolBlock bytes each and kPoolBytes in all, the
// ones freed longest ago making room (blocks of a model that is gone would
// otherwise keep the next one's out: after a batch of 384 LPs a 20,000-row
// set-up took 5.1 ms, 2.9 now). All go back when an allocation fails for lack
// of memory, in hn_trim and in hn_shutdown. Any thread may allocate or free. A
// block is known by its allocation's id: one that was freed past the library
// and whose address the driver gave to somebody else is not taken for it.
namespace {
// The driver's id of the allocation that p lies in, unique in the process's
// life; 0 if there is none (0.1 us).
unsigned long long allocation_id(const void* p) {
    using Get = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
    static const Get get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuPointerGetAttribute", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Get>(f);
    }();
    if (!get) return 0;
    const auto at = reinterpret_cast<CUdeviceptr>(p);
    unsigned long long id = 0;
    CUresult r = get(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, at);
    if (r == CUDA_ERROR_INVALID_CONTEXT) {  // a thread's first call; the context becomes its own
        int device = 0;
        if (cudaGetDevice(&device) == cudaSuccess) cudaSetDevice(device);
        r = get(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, at);
    }
    return r == CUDA_SUCCESS ? id : 0;
}

constexpr size_t kPoolBlock = size_t(256) << 20, kPoolBytes = size_t(1) << 30;
struct PoolBlock {
    size_t bytes;
    int device;
    unsigned long long id;  // allocation_id
    uint64_t freed = 0;     // when, in frees
};
// Frees an idle block, unless it is gone already.
cudaError_t give_back(void* p, const PoolBlock& b) { return allocation_id(p) == b.id ? cudaFree(p) : cudaSuccess; }
struct Pool {
    std::mutex mu;
    std::unordered_map<void*, PoolBlock> live, idle;
    std::multimap<std::pair<int, size_t>, void*> by_size;  // the idle blocks
    std::map<uint64_t, void*> by_age;                      // and again, by PoolBlock::freed
    size_t idle_bytes = 0;
    uint64_t frees = 0;

    // takes an idle block out
    PoolBlock remove(void* p) {
        auto it = idle.find(p);
        const PoolBlock b = it->second;
        idle.erase(it);
        idle_bytes -= b.bytes;
        by_age.erase(b.freed);
        auto range = by_size.equal_range({b.device, b.bytes});
        while (range.first->second != p) ++range.first;
        by_size.erase(range.first);
        return b;
    }
    void* take(int device, size_t bytes) {
        std::lock_guard<std::mutex> lk(mu);
        for (;;) {
            auto it = by_size.lower_bound({device, bytes});
            if (it == by_size.end() || it->first.first != device || it->first.second > bytes + bytes / 4 + 4096)
                return nullptr;
            void* p = it->second;
            const PoolBlock b = remove(p);
            if (allocation_id(p) != b.id) continue;  // freed past the library
            live[p] = b;
            return p;
        }
    }
    size_t idle_on(int device) {
        std::lock_guard<std::mutex> lk(mu);
        size_t bytes = 0;
        for (auto& kv : idle)
            if (kv.second.device == device) bytes += kv.second.bytes;
        return bytes;
    }
    void release() {
        std::lock_guard<std::mutex> lk(mu);
        for (auto& kv : idle) give_back(kv.first, kv.second);
        idle.clear();
        by_size.clear();
        by_age.clear();
        idle_bytes = 0;
    }
};
Pool& pool() {
    static Pool* p = new Pool();  // outlives every object; the context's end frees its blocks
    return *p;
}
}  // namespace

void* pool_alloc(size_t bytes) {
    const size_t size = bytes > SIZE_MAX - 511 ? bytes : (bytes + 511) & ~size_t(511);  // the former fails below
    int device = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    if (void* p = pool().take(device, size)) return p;
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, size);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        pool().release();
        e = cudaMalloc(&p, size);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        fail(e == cudaErrorMemoryAllocation ? HN_ERR_OUT_OF_MEMORY : HN_ERR_CUDA,
             std::string("cudaMalloc of ") + std::to_string(bytes) + " bytes failed: " + cudaGetErrorString(e));
    }
    const PoolBlock b{size, device, allocation_id(p)};
    std::lock_guard<std::mutex> lk(pool().mu);
    pool().live[p] = b;
    return p;
}

// What cudaFree does beside freeing: it waits for the work on every stream, and
// is refused where a stream capture forbids it. cudaDeviceSynchronize is
// refused beside any capture, and breaks it, so an allocation of no use is made
// and freed: 2.7 us (1.6 the synchronisation), once for blocks freed together.
cudaError_t wait_as_free() {
    void* q = nullptr;
    const cudaError_t e = cudaMalloc(&q, 512);
    return e == cudaSuccess ? cudaFree(q) : e;
}

cudaError_t pool_free(void* const* ps, size_t n) {
    Pool& P = pool();
    cudaError_t e = cudaSuccess;
    auto done = [&](cudaError_t one) {
        if (e == cudaSuccess) e = one;
    };
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess) cudaGetLastError();
    std::vector<std::pair<void*, PoolBlock>> keep, out;  // for the cache; for the driver
    for (size_t i = 0; i < n; ++i) {
        void* p = ps[i];
        if (!p) continue;
        const unsigned long long id = allocation_id(p);
        PoolBlock b{0, -1, 0};
        std::lock_guard<std::mutex> lk(P.mu);
        auto free_one = P.idle.find(p);
        if (free_one != P.idle.end()) {
            if (free_one->second.id == id) {  // freed before
                done(cudaErrorInvalidValue);
                continue;
            }
            P.remove(p);
        }
        auto it = P.live.find(p);
        if (it != P.live.end()) {
            if (it->second.id == id) b = it->second;
            P.live.erase(it);
        }
        (b.id != 0 && b.device == device && b.bytes <= kPoolBlock ? keep : out).emplace_back(p, b);
    }
    if (!keep.empty() && wait_as_free() != cudaSuccess) {
        cudaGetLastError();  // the results are cudaFree's
        out.insert(out.end(), keep.begin(), keep.end());
        keep.clear();
    }
    for (auto& o : out) {
        const cudaError_t one = cudaFree(o.first);
        done(one);
        if (one != cudaSuccess && o.second.id != 0) {
            std::lock_guard<std::mutex> lk(P.mu);
            P.live.emplace(o);
        }
    }
    std::vector<std::pair<void*, PoolBlock>> old;
    {
        std::lock_guard<std::mutex> lk(P.mu);
        for (auto& [p, b] : keep) {
            while (P.idle_bytes + b.bytes > kPoolBytes) {
                void* o = P.by_age.begin()->second;
                old.emplace_back(o, P.remove(o));
            }
            b.freed = P.frees++;
            P.idle[p] = b;
            P.by_size.emplace(std::pair{b.device, b.bytes}, p);
            P.by_age[b.freed] = p;
            P.idle_bytes += b.bytes;
        }
    }
    for (auto& o : old) done(give_back(o.first, o.second));
    return e;
}

void pool_release() { pool().release(); }

// ---------------------------------------------------------------- pinned host words
// Handles that read a count back each have a word of pinned memory. They come
// from slabs (4 KB per 1,024 handles at a time) that hn_shutdown gives back: a
// pinned allocation and its end take 2 ms, the rest of a small batch's handle
// 0.13 ms.
namespace {
constexpr int kSlabWords = 1024;
struct HostWords {
    std::mutex mu;
    std::vector<int32_t*> slabs, free;  // the slabs, their free words
};
HostWords& host_words() {
    static HostWords* w = new HostWords();  // outlives every object
    return *w;
}
}  // namespace

int32_t* host_word() {
    HostWords& W = host_words();
    std::lock_guard<std::mutex> lk(W.mu);
    if (W.free.empty()) {
        W.slabs.reserve(W.slabs.size() + 1);
        W.free.reserve((W.slabs.size() + 1) * kSlabWords);  // room for every word that comes back
        void* slab = nullptr;
        check_cuda(cudaHostAlloc(&slab, kSlabWords * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped),
                   "cudaHostAlloc");
        W.slabs.push_back(static_cast<int32_t*>(slab));
        for (int i = kSlabWords; i-- > 0;) W.free.push_back(W.slabs.back() + i);
    }
    int32_t* w = W.free.back();
    W.free.pop_back();
    return w;
}

void host_word_free(int32_t* w) {
    HostWords& W = host_words();
    std::lock_guard<std::mutex> lk(W.mu);
    if (w) W.free.push_back(w);
}

void host_words_release() {
    HostWords& W = host_words();
    std::lock_guard<std::mutex> lk(W.mu);
    if (W.free.size() < W.slabs.size() * kSlabWords) return;  // a handle has one
    for (int32_t* slab : W.slabs) cudaFreeHost(slab);
    W.slabs.clear();
    W.free.clear();
}

Workspace& workspace(cudaStream_t s) {
    std::lock_guard<std::mutex> lk(g_ctx.mu);
    auto it = g_ctx.ws.find(s);
    if (it != g_ctx.ws.end()) return it->second;
    Workspace w;
    w.partials = dmalloc<double>(4 * kMaxReduceBlocks + 8);
    w.counter = dmalloc<unsigned>(4);
    w.select = dmalloc<unsigned long long>(kSelectWords);
    w.price = dmalloc<unsigned long long>(kPriceWords);
    check_cuda(cudaMemsetAsync(w.counter, 0, 4 * sizeof(unsigned), s), "workspace init");
    check_cuda(cudaMemsetAsync(w.select, 0, kSelectWords * sizeof(unsigned long long), s), "workspace init");
    check_cuda(cudaStreamSynchronize(s), "workspace init sync");
    return g_ctx.ws.emplace(s, w).first->second;
}

void ensure_staging(Workspace& w, size_t bytes, cudaStream_t s) {
    if (w.staging_bytes < bytes) {
        check_cuda(cudaStreamSynchronize(s), "staging sync");
        if (w.staging_h) cudaFreeHost(w.staging_h);
        w.staging_h = nullptr;
        w.staging_bytes = 0;
        check_cuda(cudaMallocHost(reinterpret_cast<void**>(&w.staging_h), bytes),
                   "cudaMallocHost staging");
        w.staging_bytes = bytes;
    }
    if (w.staging_d_bytes < bytes) {
        check_cuda(cudaStreamSynchronize(s), "staging sync");
        dfree(w.staging_d);
        w.staging_d = nullptr;
        w.staging_d_bytes = 0;
        w.staging_d = dmalloc<double>((bytes + 7) / 8);
        w.staging_d_bytes = bytes;
    }
}

// ---------------------------------------------------------------- scans
namespace {
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int64_t kScanTile = kScanThreads * kScanItems;

template <class T>
__global__ void __launch_bounds__(kScanThreads) scan_tile_kernel(const T* in, T* out, int64_t n,
                                                                  int64_t* tile_sums) {
    if (!after_previous()) return;
    __shared__ int64_t sh[32];
    const int64_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int64_t v[kScanItems];
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = (base + i < n) ? static_cast<int64_t>(in[base + i]) : 0;
        s += v[i];
    }
    int64_t total;
    int64_t pre = block_exclusive_scan_i64<kScanThreads>(s, sh, &total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (base + i < n) out[base + i] = static_cast<T>(pre);
        pre += v[i];
    }
    if (threadIdx.x == 0 && tile_sums) tile_sums[blockIdx.x] = total;
}

template <class T>
__global__ void scan_add_kernel(T* out, int64_t n, const int64_t* tile_offsets) {
    if (!after_previous()) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] += static_cast<T>(tile_offsets[i / kScanTile]);
}

template <class T>
void scan_exclusive_impl(const T* in, T* out, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles == 1) {
        launch_next(scan_tile_kernel<T>, 1, kScanThreads, 0, s, in, out, n, nullptr);
        launched("scan_tile_kernel");
        return;
    }
    int64_t* sums = dmalloc<int64_t>(tiles);
    launch_next(scan_tile_kernel<T>, (unsigned)tiles, kScanThreads, 0, s, in, out, n, sums);
    launched("scan_tile_kernel");
    scan_exclusive_impl<int64_t>(sums, sums, tiles, s);
    launch_next(scan_add_kernel<T>, (unsigned)((n + 255) / 256), 256, 0, s, out, n, sums);
    launched("scan_add_kernel");
    check_cuda(cudaStreamSynchronize(s), "scan sync");
    dfree(sums);
}
}  // namespace

void scan_exclusive_i64(const int64_t* in, int64_t* out, int64_t n, cudaStream_t s) {
    scan_exclusive_impl<int64_t>(in, out, n, s);
}
void scan_exclusive_i32(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s) {
    scan_exclusive_impl<int32_t>(in, out, n, s);
}

// ---------------------------------------------------------------- BLAS-1
namespace {
constexpr int kRedThreads = 256;

enum RedOp { kDot = 0, kSumSq = 1, kMaxAbs = 2 };

// Deterministic grid reduction: each block folds a fixed, grid-strided slice
// in index order, reduces it with a fixed tree into partials[block]; the last
// block to finish folds the partials in block order. The grid size depends
// only on n, so the bits do not change from run to run.
template <int OP>
__global__ void __launch_bounds__(kRedThreads) reduce_kernel(int64_t n, const double* __restrict__ a,
                                                             const double* __restrict__ b,
                                                             double* partials, unsigned* counter,
                                                             double* out) {
    if (!after_previous()) return;
    __shared__ double sh[32];
    __shared__ bool last;
    double acc = 0.0;
    const int64_t stride = (int64_t)gridDim.x * kRedThreads;
    for (int64_t i = blockIdx.x * (int64_t)kRedThreads + threadIdx.x; i < n; i += stride) {
        if (OP == kDot) acc += a[i] * b[i];
        else if (OP == kSumSq) acc += a[i] * a[i];
        else acc = fmax(acc, fabs(a[i]));
    }
    double r = (OP == kMaxAbs) ? block_max<kRedThreads>(acc, sh) : block_sum<kRedThreads>(acc, sh);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = r;
        __threadfence();
        const unsigned t = atomicAdd(counter, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double v = (OP == kMaxAbs) ? 0.0 : 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kRedThreads) {
        const double p = __ldcg(partials + i);
        v = (OP == kMaxAbs) ? fmax(v, p) : v + p;
    }
    r = (OP == kMaxAbs) ? block_max<kRedThreads>(v, sh) : block_sum<kRedThreads>(v, sh);
    if (threadIdx.x == 0) {
        *out = (OP == kSumSq) ? sqrt(r) : r;
        *counter = 0u;
    }
}

__global__ void axpy_kernel(int64_t n, double alpha, const double* __restrict__ x,
                            double* __restrict__ y) {
    if (!after_previous()) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride)
        y[i] += alpha * x[i];
}

template <int OP>
void run_reduce(int64_t n, const double* a, const double* b, double* out, cudaStream_t s) {
    Workspace& w = workspace(s);
    const int grid = grid_for(n, kRedThreads * 4, kMaxReduceBlocks);
    launch_next(reduce_kernel<OP>, grid, kRedThreads, 0, s, n, a, b, w.partials, w.counter, out);
    launched("reduce_kernel");
}
}  // namespace

void reduce_dot(int64_t n, const double* a, const double* b, double* out, cudaStream_t s) {
    run_reduce<kDot>(n, a, b, out, s);
}
void reduce_nrm2(int64_t n, const double* a, double* out, cudaStream_t s) {
    run_reduce<kSumSq>(n, a, nullptr, out, s);
}
void reduce_maxabs(int64_t n, const double* a, double* out, cudaStream_t s) {
    run_reduce<kMaxAbs>(n, a, nullptr, out, s);
}

}  // namespace hn

using namespace hn;

// ================================================================ C ABI
extern "C" {

int hn_init(int device) {
    return guard("hn_init", [&] {
        if (device >= 0 && device == ctx().device) {  // known already: the queries below take milliseconds
            check_cuda(cudaSetDevice(device), "cudaSetDevice");
            return;
        }
        int count = 0;
        check_cuda(cudaGetDeviceCount(&count), "cudaGetDeviceCount");
        if (device < 0 || device >= count)
            fail(HN_ERR_INVALID_ARG, "device " + std::to_string(device) + " out of range (" +
                                         std::to_string(count) + " devices)");
        cudaDeviceProp p;
        check_cuda(cudaGetDeviceProperties(&p, device), "cudaGetDeviceProperties");
        if (p.major != 10 || p.minor != 0)
            fail(HN_ERR_UNSUPPORTED, std::string("device is sm_") + std::to_string(p.major) +
                                         std::to_string(p.minor) +
                                         "; this library is built for sm_100a only");
        check_cuda(cudaSetDevice(device), "cudaSetDevice");
        check_cuda(cudaFree(nullptr), "context creation");
        ctx().device = device;
        ctx().sm_count = p.multiProcessorCount;
    });
}

int hn_shutdown(void) {
    return guard("hn_shutdown", [&] {
        Context& c = ctx();
        if (c.device < 0) return;
        cudaDeviceSynchronize();
        std::lock_guard<std::mutex> lk(c.mu);
        for (auto& kv : c.ws) {
            dfree({kv.second.partials, kv.second.counter, kv.second.select, kv.second.price, kv.second.staging_d});
            if (kv.second.staging_h) cudaFreeHost(kv.second.staging_h);
        }
        c.ws.clear();
        pool_release();
        host_words_release();
    });
}

const char* hn_last_error(void) { return g_last_error.c_str(); }

int hn_device_info(hn_device_info_t* out) {
    return guard("hn_device_info", [&] {
        require_init();
        if (!out) fail(HN_ERR_INVALID_ARG, "null output");
        cudaDeviceProp p;
        check_cuda(cudaGetDeviceProperties(&p, ctx().device), "cudaGetDeviceProperties");
        std::memset(out, 0, sizeof(*out));
        std::strncpy(out->name, p.name, sizeof(out->name) - 1);
        out->device = ctx().device;
        out->sm_count = p.multiProcessorCount;
        out->cc_major = p.major;
        out->cc_minor = p.minor;
        check_cuda(cudaMemGetInfo(&out->free_mem, &out->total_mem), "cudaMemGetInfo");
        out->free_mem += pool().idle_on(out->device);  // the next hn_malloc's
    });
}

int hn_stats(uint64_t* kernel_launches, uint64_t* api_calls) {
    if (kernel_launches) *kernel_launches = ctx().launches.load();
    if (api_calls) *api_calls = ctx().calls.load();
    return HN_OK;
}

int hn_reset_stats(void) {
    ctx().launches.store(0);
    ctx().calls.store(0);
    return HN_OK;
}

int hn_fault_inject(int64_t after_calls, int status) {
    ctx().inject_status.store(status);
    ctx().inject_after.store(after_calls < 0 ? -1 : after_calls);
    return HN_OK;
}

int hn_malloc(void** ptr_dev, size_t bytes) {
    return guard("hn_malloc", [&] {
        require_init();
        if (!ptr_dev) fail(HN_ERR_INVALID_ARG, "null output");
        *ptr_dev = dmalloc<char>(bytes);
    });
}

int hn_free(void* p) {
    return guard("hn_free", [&] {
        require_init();
        check_cuda(pool_free(&p, 1), "cudaFree");
    });
}

int hn_trim(void) {
    return guard("hn_trim", [&] {
        require_init();
        pool_release();
    });
}

int hn_memcpy_h2d(void* dst, const void* src, size_t bytes, void* stream) {
    return guard("hn_memcpy_h2d", [&] {
        require_init();
        check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, as_stream(stream)),
                   "cudaMemcpyAsync H2D");
    });
}

int hn_memcpy_d2h(void* dst, const void* src, size_t bytes, void* stream) {
    return guard("hn_memcpy_d2h", [&] {
        require_init();
        check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, as_stream(stream)),
                   "cudaMemcpyAsync D2H");
        check_cuda(cudaStreamSynchronize(as_stream(stream)), "D2H sync");
    });
}

int hn_memcpy_d2d(void* dst, const void* src, size_t bytes, void* stream) {
    return guard("hn_memcpy_d2d", [&] {
        require_init();
        check_cuda(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, as_stream(stream)),
                   "cudaMemcpyAsync D2D");
    });
}

int hn_memset(void* p, int byte, size_t bytes, void* stream) {
    return guard("hn_memset", [&] {
        require_init();
        check_cuda(cudaMemsetAsync(p, byte, bytes, as_stream(stream)), "cudaMemsetAsync");
    });
}

int hn_stream_sync(void* stream) {
    return guard("hn_stream_sync", [&] {
        require_init();
        check_cuda(cudaStreamSynchronize(as_stream(stream)), "cudaStreamSynchronize");
    });
}

int hn_dot(int64_t n, const double* a, const double* b, double* result, void* stream) {
    return guard("hn_dot", [&] {
        require_init();
        if (n < 0 || !result || (n > 0 && (!a || !b))) fail(HN_ERR_INVALID_ARG, "bad arguments");
        reduce_dot(n, a, b, result, as_stream(stream));
    });
}

int hn_axpy(int64_t n, double alpha, const double* x, double* y, void* stream) {
    return guard("hn_axpy", [&] {
        require_init();
        if (n < 0 || (n > 0 && (!x || !y))) fail(HN_ERR_INVALID_ARG, "bad arguments");
        if (n == 0) return;
        launch_next(axpy_kernel, grid_for(n, 256, ctx().sm_count * 16), 256, 0, as_stream(stream), n, alpha, x, y);
        launched("axpy_kernel");
    });
}

int hn_nrm_inf(int64_t n, const double* v, double* result, void* stream) {
    return guard("hn_nrm_inf", [&] {
        require_init();
        if (n < 0 || !result || (n > 0 && !v)) fail(HN_ERR_INVALID_ARG, "bad arguments");
        reduce_maxabs(n, v, result, as_stream(stream));
    });
}

int hn_nrm2(int64_t n, const double* v, double* result, void* stream) {
    return guard("hn_nrm2", [&] {
        require_init();
        if (n < 0 || !result || (n > 0 && !v)) fail(HN_ERR_INVALID_ARG, "bad arguments");
        reduce_nrm2(n, v, result, as_stream(stream));
    });
}

}  // extern "C"
