// How the slices of a small system are dealt to the CTAs of one cluster (cg_cluster.cu).  Compiles as host
// code too: the tests run these functions on the CPU.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define LPM_SHARE_HD __host__ __device__ __forceinline__
#else
#define LPM_SHARE_HD inline
#endif

namespace lpm
{

// CTAs for n slices where `limit` (a power of two) may be used: none of them without a slice
LPM_SHARE_HD int share_ctas(int n, int limit)
{
    while (limit > n)
        limit /= 2;
    return limit;
}

// First slice of CTA k of nc: shares of n / nc or one more, none empty when n >= nc
LPM_SHARE_HD int share_begin(int n, int nc, int k) { return (int)((int64_t)k * n / nc); }

// Slices of the largest share
LPM_SHARE_HD int share_most(int n, int nc) { return (n + nc - 1) / nc; }

} // namespace lpm
