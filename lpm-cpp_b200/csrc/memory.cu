// Device memory of the problems and of their set-up, and the small pinned records they read scalars
// from.
//
// A problem holds about 60 device arrays and its set-up some 25 temporaries; cudaMalloc and cudaFree
// of each cost 12 + 8 ms per 18,000-particle problem, most of a small problem's whole life (and every
// load step paid for a temporary of the default pool, which gives its memory back at each
// synchronisation).  All come from one stream-ordered pool per device instead, which belongs to this
// library: the device's default pool and its settings are left alone.  The pool keeps at most
// kPoolKeep bytes that no handle uses (the rest goes back at the next synchronisation after a
// destroy), hands a stream only memory whose last use it can order before it, and gives everything
// unused back when an allocation fails.  The driver serialises its calls, so any thread may create and
// destroy problems.
//
// The pool and the pinned blocks belong to the device's context.  A host program may end that
// (cudaDeviceReset) once its handles are gone and create problems again; each use therefore compares the
// context's id, which no other context of the process ever has, and forgets what belonged to another.
#include <cuda.h>

#include <mutex>
#include <vector>

#include "lpm_internal.cuh"

namespace lpm
{

constexpr uint64_t kPoolKeep = uint64_t(512) << 20;
constexpr int kMaxDevices = 64;
constexpr size_t kPinnedBlock = 256;  // one problem's pinned records
constexpr size_t kPinnedKeep = 1024;  // blocks kept per device for later problems

struct DeviceMemory
{
    uint64_t ctx = 0; // the context that the rest belongs to
    cudaMemPool_t pool = nullptr;
    std::vector<void *> pinned;
};

static std::mutex g_mu;
static DeviceMemory g_dev[kMaxDevices];

// Id of the current device's context, which is created if there is none (after a reset); g_mu is held.
static cudaError_t context_id(uint64_t *id)
{
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static void *current = nullptr, *get_id = nullptr;
    if (!current || !get_id)
    {
        cudaDriverEntryPointQueryResult found;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &current, 12000, cudaEnableDefault, &found);
        if (e == cudaSuccess)
            e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &get_id, 12000, cudaEnableDefault, &found);
        if (e != cudaSuccess)
            return e;
        if (!current || !get_id)
            return cudaErrorNotSupported;
    }
    for (int attempt = 0; attempt < 2; ++attempt)
    {
        CUcontext ctx = nullptr;
        unsigned long long v = 0;
        if (reinterpret_cast<GetCurrent>(current)(&ctx) == CUDA_SUCCESS && ctx &&
            reinterpret_cast<GetId>(get_id)(ctx, &v) == CUDA_SUCCESS)
        {
            *id = v;
            return cudaSuccess;
        }
        const cudaError_t e = cudaFree(nullptr);
        if (e != cudaSuccess)
            return e;
    }
    return cudaErrorContextIsDestroyed;
}

// The current device's entry, as its context has it; g_mu is held.
static cudaError_t device_memory(DeviceMemory **out)
{
    int dev = 0;
    uint64_t ctx = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= kMaxDevices)
        return cudaErrorInvalidDevice;
    if ((e = context_id(&ctx)) != cudaSuccess)
        return e;
    DeviceMemory &m = g_dev[dev];
    if (m.ctx != ctx)
    { // what it held ended with its context
        m.ctx = ctx;
        m.pool = nullptr;
        m.pinned.clear();
    }
    *out = &m;
    return cudaSuccess;
}

static cudaError_t device_pool(cudaMemPool_t *out)
{
    std::lock_guard<std::mutex> lk(g_mu);
    DeviceMemory *m = nullptr;
    cudaError_t e = device_memory(&m);
    if (e != cudaSuccess)
        return e;
    if (!m->pool)
    {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        if ((e = cudaGetDevice(&props.location.id)) != cudaSuccess)
            return e;
        cudaMemPool_t p = nullptr;
        if ((e = cudaMemPoolCreate(&p, &props)) != cudaSuccess)
            return e;
        uint64_t keep = kPoolKeep;
        if ((e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess)
        {
            cudaMemPoolDestroy(p);
            return e;
        }
        m->pool = p;
    }
    *out = m->pool;
    return cudaSuccess;
}

cudaError_t pool_alloc_bytes(void **ptr, size_t bytes, cudaStream_t st)
{
    cudaMemPool_t pool = nullptr;
    cudaError_t e = device_pool(&pool);
    if (e != cudaSuccess)
        return e;
    e = cudaMallocFromPoolAsync(ptr, bytes ? bytes : 1, pool, st);
    if (e == cudaErrorMemoryAllocation)
    {
        (void)cudaGetLastError();
        cudaStreamSynchronize(st);
        cudaMemPoolTrimTo(pool, 0);
        e = cudaMallocFromPoolAsync(ptr, bytes ? bytes : 1, pool, st);
    }
    return e;
}

// a block for one problem's pinned records (Scalars, then 8 status words), and the context it belongs to
cudaError_t pinned_take(void **ptr, uint64_t *ctx)
{
    static_assert(sizeof(Scalars) <= 128, "the status words start at byte 128");
    {
        std::lock_guard<std::mutex> lk(g_mu);
        DeviceMemory *m = nullptr;
        const cudaError_t e = device_memory(&m);
        if (e != cudaSuccess)
            return e;
        *ctx = m->ctx;
        if (!m->pinned.empty())
        {
            *ptr = m->pinned.back();
            m->pinned.pop_back();
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(ptr, kPinnedBlock, cudaHostAllocPortable);
}

void pinned_give(void *ptr, uint64_t ctx)
{
    {
        std::lock_guard<std::mutex> lk(g_mu);
        DeviceMemory *m = nullptr;
        if (device_memory(&m) != cudaSuccess || m->ctx != ctx)
            return; // the block ended with its context
        if (m->pinned.size() < kPinnedKeep)
        {
            m->pinned.push_back(ptr);
            return;
        }
    }
    cudaFreeHost(ptr);
}

} // namespace lpm
