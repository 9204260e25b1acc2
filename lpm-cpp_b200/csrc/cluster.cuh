// Exchanges between the CTAs of one thread-block cluster by asynchronous stores and copies that count
// bytes on the receiver's mbarrier: a wait there orders the data without fences, and takes 366 cycles
// from store to wake-up whatever the cluster's size (a release/acquire cluster barrier with remote
// stores takes 1,070 at 16 CTAs).
#pragma once

#include <cstdint>

#include "cg_device.cuh"

namespace lpm
{

constexpr size_t kClusterSmem = 232448; // shared memory of one CTA on sm_100

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned mapa(unsigned a, unsigned rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void push(unsigned dst, unsigned bar, double v)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(dst), "d"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void push2(unsigned dst, unsigned bar, double a, double b)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst), "d"(a),
                 "d"(b), "r"(bar)
                 : "memory");
}
// bytes (a multiple of 16) of this CTA's shared memory to the same place in another CTA's; what they
// hold is written before the writers' fence_async and a block synchronisation
__device__ __forceinline__ void push_bulk(const void *src, unsigned rank, unsigned bar, unsigned bytes)
{
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     mapa(smem_addr(src), rank)),
                 "r"(smem_addr(src)), "r"(bytes), "r"(mapa(bar, rank))
                 : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(const void *bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init_done() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void expect_bytes(unsigned bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Waits until the phase `parity` of an mbarrier of this CTA is complete; false once the limit passed.
__device__ __forceinline__ bool cluster_wait(unsigned bar, unsigned parity, unsigned long long wait_ns)
{
    unsigned long long t0 = 0;
    while (true)
    {
        unsigned done;
        if (wait_ns >= 100000ull)
            asm volatile("{\n.reg .pred p;\n"
                         "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                         "selp.u32 %0, 1, 0, p;\n}"
                         : "=r"(done)
                         : "r"(bar), "r"(parity)
                         : "memory");
        else // a try may sleep past a limit this short
            asm volatile("{\n.reg .pred p;\n"
                         "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                         "selp.u32 %0, 1, 0, p;\n}"
                         : "=r"(done)
                         : "r"(bar), "r"(parity)
                         : "memory");
        if (done)
            return true;
        const unsigned long long now = gtimer();
        if (t0 == 0)
            t0 = now;
        else if (now - t0 > wait_ns)
            return false;
    }
}

// After a failed wait, before the cluster's last synchronisation (which orders no asynchronous store): what
// this CTA still has on its way to others, and nobody waits for any more, lands while it pauses.  An
// exchange takes 0.2 us; the pause is 50 us.
__device__ __forceinline__ void drain_pushes()
{
    const unsigned long long t0 = gtimer();
    while (gtimer() - t0 < 50000ull)
        __nanosleep(1000);
}

// Largest cluster the device runs of `kernel` with a CTA's whole shared memory: 16, else 8, else 0.
int max_cluster(const void *kernel);
// Launches `kernel` as one cluster of nc CTAs.
cudaError_t launch_cluster(const void *kernel, int nc, int threads, size_t smem, void **args, cudaStream_t st);

} // namespace lpm
