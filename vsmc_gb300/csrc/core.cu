// Status strings, error bookkeeping, grid sizing and stream-ordered scratch.
#include "common.cuh"

#include <atomic>
#include <cuda.h>
#include <mutex>
#include <vector>

namespace vsmc_cuda
{

static std::atomic<int> g_last_cuda_error{0};

void set_last_cuda_error(cudaError_t e)
{
    g_last_cuda_error.store(static_cast<int>(e));
}

int num_sms()
{
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return 152;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) !=
                cudaSuccess ||
            n <= 0)
            n = 152;
        cached[dev] = n;
    }
    return cached[dev];
}

int grid_for(
    size_t work_items, int block, int items_per_thread, int blocks_per_sm)
{
    const size_t per_block =
        static_cast<size_t>(block) * static_cast<size_t>(items_per_thread);
    size_t need = (work_items + per_block - 1) / per_block;
    const size_t cap =
        static_cast<size_t>(num_sms()) * static_cast<size_t>(blocks_per_sm);
    if (need > cap)
        need = cap;
    if (need < 1)
        need = 1;
    return static_cast<int>(need);
}

// The scratch pool of a device: the library's own, so that no setting of the
// process's default pool changes.  The default pool gives its memory back at
// every synchronization, and mapping it again cost 0.2 to 2.4 ms a call
// (with the GPU idle around it, a resampling call took 300 us at n = 1000
// and 3.3 ms at 2^24; 70 us and 0.35 ms from this pool).  It keeps at most
// kScratchKeep of what no call uses (a resampling call takes about 24 bytes
// per particle, 0.4 GB at 2^24); anything above goes back at the next
// synchronization, and all of it when a device allocation of the library's
// fails or vsmc_cuda_trim_scratch is called.
// Allocations and frees are stream-ordered, from any thread.  A device reset
// (cudaDeviceReset) ends the pool with the context, so a pool belongs to the
// context that made it: its id is never used again, where the handle is.
constexpr uint64_t kScratchKeep = 1ull << 30;

struct ScratchPool {
    int dev;
    unsigned long long context;
    cudaMemPool_t pool;
};

static std::mutex g_pool_mutex;
static std::vector<ScratchPool> g_pools;

// id of a stream's context (0: none, or no driver call that tells)
static unsigned long long context_id(cudaStream_t st)
{
    using StreamCtx = CUresult (*)(CUstream, CUcontext *);
    using CtxId = CUresult (*)(CUcontext, unsigned long long *);
    static const auto entry = [](const char *name) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion(name, &f, 12000,
                cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return f;
    };
    static const auto stream_ctx =
        reinterpret_cast<StreamCtx>(entry("cuStreamGetCtx"));
    static const auto ctx_id = reinterpret_cast<CtxId>(entry("cuCtxGetId"));
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!stream_ctx || !ctx_id || stream_ctx(st, &ctx) != CUDA_SUCCESS ||
        ctx_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

// the pool of a stream's device in its context; null: the default pool
static cudaMemPool_t scratch_pool(cudaStream_t st)
{
    int dev = -1;
    const unsigned long long id = context_id(st);
    if (id == 0 || cudaStreamGetDevice(st, &dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (const ScratchPool &p : g_pools)
        if (p.dev == dev && p.context == id)
            return p.pool;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    uint64_t keep = kScratchKeep;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    g_pools.push_back({dev, id, pool});
    return pool;
}

// the pools of the current context
static cudaError_t scratch_trim()
{
    const unsigned long long id = context_id(nullptr);
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (const ScratchPool &p : g_pools) {
        const cudaError_t e = id != 0 && p.context == id
            ? cudaMemPoolTrimTo(p.pool, 0)
            : cudaSuccess;
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

cudaError_t device_malloc(void **p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        scratch_trim();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

Scratch::~Scratch()
{
    // stream-ordered: each block is released after the work queued before
    for (void *p : ptrs_)
        cudaFreeAsync(p, stream_);
}

void *Scratch::alloc(size_t bytes)
{
    void *p = nullptr;
    if (!found_) {
        // a stream under capture gets the graph's own allocation nodes
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
        if (cudaStreamIsCapturing(stream_, &cap) == cudaSuccess &&
            cap == cudaStreamCaptureStatusNone)
            pool_ = scratch_pool(stream_);
        else
            cudaGetLastError();
        found_ = true;
    }
    cudaError_t e = pool_
        ? cudaMallocFromPoolAsync(&p, bytes ? bytes : 1, pool_, stream_)
        : cudaMallocAsync(&p, bytes ? bytes : 1, stream_);
    if (pool_ && e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        scratch_trim();
        e = cudaMallocFromPoolAsync(&p, bytes ? bytes : 1, pool_, stream_);
    }
    if (e != cudaSuccess) {
        set_last_cuda_error(e);
        return nullptr;
    }
    ptrs_.push_back(p);
    return p;
}

} // namespace vsmc_cuda

extern "C" {

const char *vsmc_cuda_status_string(int status)
{
    switch (status) {
        case VSMC_CUDA_OK: return "ok";
        case VSMC_CUDA_ERR_ARG: return "invalid argument";
        case VSMC_CUDA_ERR_SIZE: return "length out of the supported range";
        case VSMC_CUDA_ERR_NONFINITE:
            return "non-finite or negative weight";
        case VSMC_CUDA_ERR_TIMEOUT: return "bounded device wait gave up";
        case VSMC_CUDA_ERR_CUDA: return "CUDA runtime error";
        case VSMC_CUDA_ERR_ALLOC: return "device allocation failed";
        case VSMC_CUDA_ERR_INTERNAL: return "internal consistency check failed";
        default: return "unknown status";
    }
}

int vsmc_cuda_last_cuda_error(void)
{
    return vsmc_cuda::g_last_cuda_error.load();
}

int vsmc_cuda_version(void) { return 100; }

int vsmc_cuda_trim_scratch(void)
{
    VSMC_CUDA_TRY(vsmc_cuda::scratch_trim());
    return VSMC_CUDA_OK;
}

} // extern "C"
