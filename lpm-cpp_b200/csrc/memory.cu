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
#include <mutex>
#include <vector>

#include "lpm_internal.cuh"

namespace lpm
{

constexpr uint64_t kPoolKeep = uint64_t(512) << 20;
constexpr int kMaxDevices = 64;
constexpr size_t kPinnedBlock = 256;  // one problem's pinned records
constexpr size_t kPinnedKeep = 1024;  // blocks kept for later problems

static std::mutex g_mu;
static cudaMemPool_t g_pool[kMaxDevices] = {};
static std::vector<void *> g_pinned;

static cudaError_t device_pool(cudaMemPool_t *out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev < 0 || dev >= kMaxDevices)
        return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_pool[dev])
    {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if ((e = cudaMemPoolCreate(&p, &props)) != cudaSuccess)
            return e;
        uint64_t keep = kPoolKeep;
        if ((e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess)
        {
            cudaMemPoolDestroy(p);
            return e;
        }
        g_pool[dev] = p;
    }
    *out = g_pool[dev];
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

// a block for one problem's pinned records (Scalars, then 8 status words)
cudaError_t pinned_take(void **ptr)
{
    static_assert(sizeof(Scalars) <= 128, "the status words start at byte 128");
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_pinned.empty())
        {
            *ptr = g_pinned.back();
            g_pinned.pop_back();
            return cudaSuccess;
        }
    }
    return cudaHostAlloc(ptr, kPinnedBlock, cudaHostAllocPortable);
}

void pinned_give(void *ptr)
{
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_pinned.size() < kPinnedKeep)
        {
            g_pinned.push_back(ptr);
            return;
        }
    }
    cudaFreeHost(ptr);
}

} // namespace lpm
