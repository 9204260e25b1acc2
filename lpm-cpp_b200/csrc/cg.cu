// Linear solve of the Newton step: the replacement for Solver::LPM_CG (include/solver.h:277-354),
// i.e. MKL's RCI dcg with mkl_sparse_d_mv on the symmetric upper CSR.
//
// Elastic and J2 problems solve on the bond form of K (bond_op.cu), small ones of the other types in one
// cluster (cg_cluster.cu).  This file routes them and holds the CG on the assembled matrix.
//
// One persistent cooperative launch runs the whole unpreconditioned CG (x0 = 0, stop when
// ||r||^2 <= rtol*||r0||^2 + atol, cap = problem size, the squared-norm test of MKL's dcg with
// dpar[0] = dpar[1] = 1e-12 set at solver.h:312-313).  Per iteration:
//   phase A  q = K p_new, with p_new = r + beta*p_old formed on the fly from the gathered
//            r and p_old (so the direction update needs no pass of its own); partial p.q
//   barrier
//   phase B  x += alpha p_new, r -= alpha q; partial r.r
//   barrier
// Every reduction is a fixed tree, and every block reduces the per-block partials in the same
// order, so all blocks take identical decisions and a run is bit-reproducible.  The grid
// barrier is a sense-counting barrier with a time limit: a wait that exceeds it records
// LPMGPU_ERR_TIMEOUT and the kernel returns.
//
// The SpMV runs on the sliced-ELL layout (lpm_internal.cuh): one thread per particle row, a
// warp per slice of 32 rows.  For block column k every matrix plane load is 256 contiguous
// bytes (cache-streaming: the matrix is read once per iteration) and the x gathers of the 32
// rows hit neighbouring particles, so they coalesce and stay in L2 with the vectors.  k_cg's RES form keeps
// the matrix in shared memory where it fits; k_cg_stream brings a large FP32 3D matrix there by bulk copies.
//
// Mixed precision (LPMGPU_MIXED): the same kernel on an FP32 copy of K with FP32 Krylov
// vectors (dot products in FP64), inside an FP64 iterative refinement that recomputes the
// true residual b - K x with the FP64 matrix and stops on the same squared-norm rule.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include <string>

#include "bond_op.cuh"
#include "bulk_copy.cuh"
#include "cg_cluster.cuh"
#include "cg_device.cuh"

namespace lpm
{

struct CGState
{
    int n;              // particle rows
    int nslices;
    int64_t ndof;
    const int *__restrict__ rowptr;     // connection CSR (row lengths)
    const int *__restrict__ perm;       // slice position -> particle
    const int64_t *__restrict__ slice_off;
    const int *__restrict__ col_sell;
    double rtol, atol, abs_stop; // abs_stop >= 0 overrides rtol/atol
    int64_t maxit;
    unsigned *bar;      // [0] arrivals, [1] generation
    double *part;       // [grid][2]
    int64_t *info;      // [0] iterations, [1] status bits (1 maxit, 2 timeout, 4 breakdown), [2..3] rr0/rr bits
    unsigned long long wait_ns; // limit of each grid-barrier wait
    int steps;          // RES: columns of a warp at most
};


// The column split of spmv_block for a block of ns slices: warps per slice.
__host__ __device__ __forceinline__ int column_split(int ns, int nw)
{
    int S = 2;
    while (S < kMaxColumnSplit && ns * S * 2 <= nw)
        S *= 2;
    return S;
}

// RES: a warp's columns and values are the same in every iteration, so they are copied to shared memory
// once, and its row and row length stay in registers; per iteration only r and p are read from L2.
// Otherwise the chain perm -> rowptr -> column -> r, p starts at L2 again after each grid sum, which
// empties L1.  The sums are spmv_block's, so the bits are too.  us per iteration, without -> with: FP64 hex
// 18,000 rows 9.30 -> 7.92, 9,000 8.25 -> 7.03, 3,900 7.78 -> 6.58, square 17,550 8.06 -> 6.76; FP32 hex
// 18,000 8.39 -> 6.96.  What is left is the two grid sums (2.0 us each) and the latency of the gathers.
// s.steps: the most columns of a warp.
template <typename TK, typename TV, int D, bool RES>
__global__ void __launch_bounds__(kCGThreads, kCGMinBlocks) k_cg(CGState s, const TK *__restrict__ K, const TV *__restrict__ b,
                                                   TV *__restrict__ x, TV *__restrict__ r, TV *__restrict__ pa,
                                                   TV *__restrict__ pb, TV *__restrict__ q)
{
    extern __shared__ __align__(16) unsigned char cg_sm[];
    __shared__ double sh[32];
    __shared__ int s_fail;
    __shared__ TV red[32 * D * 32];
    if (threadIdx.x == 0)
        s_fail = 0;
    __syncthreads();
    unsigned epoch = 0;
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    // each block owns a contiguous, equal share of the slices (balanced, neighbours share L1)
    const int s0 = (int)((int64_t)blockIdx.x * s.nslices / gridDim.x);
    const int s1 = (int)((int64_t)(blockIdx.x + 1) * s.nslices / gridDim.x);
    const int warp = threadIdx.x >> 5;
    const uint64_t pf = l2_evict_first(), pl = l2_evict_last();

    int ri = -1, rn_ = 0, part = 0, split = 1; // RES: the lane's row, its columns here, the warp's part
    TK *kS = reinterpret_cast<TK *>(cg_sm) + (size_t)warp * s.steps * D * D * kSlice + (threadIdx.x & 31);
    int *cS = reinterpret_cast<int *>(reinterpret_cast<TK *>(cg_sm) + (size_t)(blockDim.x >> 5) * s.steps * D * D * kSlice) +
              warp * s.steps * kSlice + (threadIdx.x & 31);
    if constexpr (RES)
    {
        split = column_split(s1 - s0, blockDim.x >> 5);
        part = warp % split;
        const int sl = s0 + warp / split, pos = sl * kSlice + (threadIdx.x & 31);
        if (sl < s1 && pos < s.n)
        {
            ri = s.perm[pos];
            const int myn = s.rowptr[ri + 1] - s.rowptr[ri];
            const int64_t off = s.slice_off[sl];
            for (int k = part; k < myn; k += split, ++rn_)
            {
                const int64_t at = (off + k) * kSlice + (threadIdx.x & 31);
                cS[rn_ * kSlice] = s.col_sell[at];
#pragma unroll
                for (int e = 0; e < D * D; ++e)
                    kS[(rn_ * D * D + e) * kSlice] = K[((off + k) * D * D + e) * kSlice + (threadIdx.x & 31)];
            }
        }
    }

    double loc = 0;
    for (int64_t k = gt; k < s.ndof; k += T)
    {
        const TV v = b[k];
        st_keep(r + k, v, pl);
        st_keep(x + k, TV(0), pl);
        st_keep(pa + k, TV(0), pl);
        loc += (double)v * (double)v;
    }
    double rr;
    if (!grid_sum(loc, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rr, s.wait_ns))
        return;
    const double stop = (s.abs_stop >= 0) ? s.abs_stop : s.rtol * rr + s.atol;
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        s.info[0] = 0;
        reinterpret_cast<double *>(s.info)[2] = rr;
        reinterpret_cast<double *>(s.info)[3] = rr;
    }
    if (rr <= stop)
        return;
    TV beta = TV(0);
    TV *pold = pa, *pnew = pb;
    for (int64_t it = 1;; ++it)
    {
        double lpq = 0.0;
        if constexpr (RES)
        {
            TV acc[D], pn[D];
#pragma unroll
            for (int c = 0; c < D; ++c)
            {
                acc[c] = TV(0);
                if (part == 0 && ri >= 0)
                    pn[c] = ld_keep(r + (int64_t)ri * D + c, pl) + beta * ld_keep(pold + (int64_t)ri * D + c, pl);
            }
#pragma unroll 4
            for (int t = 0; t < rn_; ++t)
            {
                const int j = cS[t * kSlice];
                TV xv[D];
#pragma unroll
                for (int c = 0; c < D; ++c)
                    xv[c] = ld_keep(r + (int64_t)j * D + c, pl) + beta * ld_keep(pold + (int64_t)j * D + c, pl);
#pragma unroll
                for (int rr = 0; rr < D; ++rr)
#pragma unroll
                    for (int c = 0; c < D; ++c)
                        acc[rr] += kS[(t * D * D + rr * D + c) * kSlice] * xv[c];
            }
            if (part > 0)
#pragma unroll
                for (int c = 0; c < D; ++c)
                    red[(warp * D + c) * 32 + (threadIdx.x & 31)] = acc[c];
            __syncthreads();
            if (part == 0 && ri >= 0)
            {
                for (int p = 1; p < split; ++p)
#pragma unroll
                    for (int c = 0; c < D; ++c)
                        acc[c] += red[((warp + p) * D + c) * 32 + (threadIdx.x & 31)];
#pragma unroll
                for (int c = 0; c < D; ++c)
                {
                    st_keep(pnew + (int64_t)ri * D + c, pn[c], pl);
                    st_keep(q + (int64_t)ri * D + c, acc[c], pl);
                    lpq += (double)pn[c] * (double)acc[c];
                }
            }
        }
        else
            lpq = spmv_block<TK, TV, D>(s0, s1, s.n, s.rowptr, s.perm, s.slice_off, s.col_sell, K, r, pold, pnew, q, beta,
                                        pf, pl, red);
        double pq;
        if (!grid_sum(lpq, s.bar, epoch, s.info, &s_fail, s.part, 1, sh, &pq, s.wait_ns))
            return;
        if (pq == 0.0)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                s.info[0] = it - 1;
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 4ull);
            }
            return;
        }
        const double alpha = rr / pq;
        const TV al = (TV)alpha;
        double lrr = 0;
        for (int64_t k = gt; k < s.ndof; k += T)
        {
            const TV pn = ld_keep(pnew + k, pl);
            st_keep(x + k, ld_keep(x + k, pl) + al * pn, pl);
            const TV rv = ld_keep(r + k, pl) - al * ld_keep(q + k, pl);
            st_keep(r + k, rv, pl);
            lrr += (double)rv * (double)rv;
        }
        double rn;
        if (!grid_sum(lrr, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rn, s.wait_ns))
            return;
        const bool done = rn <= stop;
        const bool capped = it >= s.maxit;
        if (done || capped)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                s.info[0] = it;
                reinterpret_cast<double *>(s.info)[3] = rn;
                if (!done)
                    atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 1ull);
            }
            return;
        }
        beta = (TV)(rn / rr);
        rr = rn;
        TV *t = pold;
        pold = pnew;
        pnew = t;
    }
}

// The FP32 CG of a 3D problem large enough that a warp owns whole slices in every block (k_cg's rule on
// column splits): the same sums in the same order, so the same bits, with the matrix streamed to shared
// memory by bulk copies.  k_cg holds a step's nine matrix loads and six gathers per lane in registers,
// which bounds it by the latency of the gathers at two steps in flight (DRAM at 55 % of its peak).  Here a
// warp's matrix comes in chunks of kStreamCols block columns (1,152 bytes each), refilled as soon as a
// chunk is used, over the ends of slices and over the grid sums, and the registers hold the gathers of a
// whole chunk.  Chunks of 1 / 2 / 3 / 4 / 5 columns: 131 / 115.5 / 112.2 / 114.2 / 120 us per iteration
// at 410,286 BCC rows (672 MB of matrix; more chunks per warp measure the same: a copy is never waited
// for long).  k_cg -> this: BCC 410,286 rows 123 -> 112 us, BCC 182,250 75.0 -> 60.3, FCC 131,072 60.1 ->
// 55.6, SC 127,500 59.2 -> 52.5.  A direction formed by its own pass before the product, which halves
// the gathers for a third grid sum: 111.6, 61.3, 56.7, 53.1.
constexpr int kStreamCols = 3;
constexpr size_t kStreamSmem = (size_t)32 * kStreamCols * 9 * kSlice * sizeof(float);

__global__ void __launch_bounds__(kCGThreads, kCGMinBlocks)
    k_cg_stream(CGState s, const float *__restrict__ K, const float *__restrict__ b, float *__restrict__ x,
                float *__restrict__ r, float *__restrict__ pa, float *__restrict__ pb, float *__restrict__ q)
{
    constexpr int D = 3, E = 9, C = kStreamCols;
    extern __shared__ __align__(128) float ring[];
    __shared__ uint64_t full[32];
    __shared__ double sh[32];
    __shared__ int s_fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s0 = (int)((int64_t)blockIdx.x * s.nslices / gridDim.x);
    const int s1 = (int)((int64_t)(blockIdx.x + 1) * s.nslices / gridDim.x);
    const int64_t T = (int64_t)gridDim.x * blockDim.x;
    const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t pf = l2_evict_first(), pl = l2_evict_last();
    const bool has = s0 + warp < s1;
    float *mine = ring + (size_t)warp * C * E * kSlice;
    uint64_t *bar = full + warp;
    if (threadIdx.x == 0)
        s_fail = 0;
    if (lane == 0)
    {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    // the next chunk to fetch (lane 0): columns [pk, pk + C) of slice psl, which has pw columns at pkp
    int psl = s0 + warp, pk = 0, pw = 0;
    const float *pkp = K;
    auto slice_of = [&]() {
        const int64_t off = s.slice_off[psl];
        pw = (int)(s.slice_off[psl + 1] - off);
        pkp = K + off * E * kSlice;
        pk = 0;
    };
    auto issue = [&]() {
        const uint32_t bytes = (uint32_t)(min(C, pw - pk) * E * kSlice * sizeof(float));
        bulk_refill(mine, pkp + (int64_t)pk * E * kSlice, bytes, bar, pf);
        pk += C;
        if (pk >= pw)
        {
            psl += 32;
            if (psl >= s1)
                psl = s0 + warp;
            slice_of();
        }
    };
    if (has && lane == 0)
    {
        slice_of();
        issue();
    }
    uint32_t parity = 0;
    bool dead = false; // a copy did not come in time: nothing more is used or fetched

    double loc = 0;
    for (int64_t k = gt; k < s.ndof; k += T)
    {
        const float v = b[k];
        st_keep(r + k, v, pl);
        st_keep(x + k, 0.0f, pl);
        st_keep(pa + k, 0.0f, pl);
        loc += (double)v * (double)v;
    }
    unsigned epoch = 0;
    double rr = 0.0, stop = 0.0;
    bool go = grid_sum(loc, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rr, s.wait_ns);
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    if (go)
    {
        stop = (s.abs_stop >= 0) ? s.abs_stop : s.rtol * rr + s.atol;
        if (lead)
        {
            s.info[0] = 0;
            reinterpret_cast<double *>(s.info)[2] = rr;
            reinterpret_cast<double *>(s.info)[3] = rr;
        }
        go = !(rr <= stop);
    }
    float beta = 0.0f;
    float *pold = pa, *pnew = pb;
    for (int64_t it = 1; go; ++it)
    {
        double lpq = 0.0;
        for (int sl = s0 + warp; sl < s1 && !dead; sl += 32)
        {
            const int pos = sl * kSlice + lane;
            const int i = pos < s.n ? s.perm[pos] : -1;
            const int myn = i >= 0 ? s.rowptr[i + 1] - s.rowptr[i] : 0;
            const int64_t off = s.slice_off[sl];
            const int w = (int)(s.slice_off[sl + 1] - off);
            const int *cp = s.col_sell + off * kSlice + lane;
            float acc[D] = {0.0f, 0.0f, 0.0f};
            int jn[C];
#pragma unroll
            for (int u = 0; u < C; ++u)
                jn[u] = u < myn ? ld_stream(cp + u * kSlice, pf) : 0;
            for (int k = 0; k < w; k += C)
            {
                float xv[C][D], pv[C][D];
#pragma unroll
                for (int u = 0; u < C; ++u)
                    if (k + u < myn)
#pragma unroll
                        for (int c = 0; c < D; ++c)
                        {
                            xv[u][c] = ld_keep(r + (int64_t)jn[u] * D + c, pl);
                            pv[u][c] = ld_keep(pold + (int64_t)jn[u] * D + c, pl);
                        }
#pragma unroll
                for (int u = 0; u < C; ++u)
                    jn[u] = k + C + u < myn ? ld_stream(cp + (int64_t)(k + C + u) * kSlice, pf) : 0;
                if (!mbar_wait_bounded(bar, parity, s.wait_ns))
                {
                    atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 2ull);
                    s_fail = 1;
                    dead = true;
                }
                dead = __any_sync(0xffffffffu, dead);
                if (dead)
                    break;
                const float *kb = mine + lane;
#pragma unroll
                for (int u = 0; u < C; ++u)
                    if (k + u < myn)
                    {
#pragma unroll
                        for (int c = 0; c < D; ++c)
                            xv[u][c] = xv[u][c] + beta * pv[u][c];
#pragma unroll
                        for (int a = 0; a < D; ++a)
#pragma unroll
                            for (int c = 0; c < D; ++c)
                                acc[a] += kb[(u * E + a * D + c) * kSlice] * xv[u][c];
                    }
                __syncwarp();
                if (lane == 0)
                    issue();
                parity ^= 1;
            }
            if (i >= 0)
#pragma unroll
                for (int c = 0; c < D; ++c)
                {
                    const int64_t k = (int64_t)i * D + c;
                    const float pn = ld_keep(r + k, pl) + beta * ld_keep(pold + k, pl);
                    st_keep(pnew + k, pn, pl);
                    st_keep(q + k, acc[c], pl);
                    lpq += (double)pn * (double)acc[c];
                }
        }
        double pq;
        if (!grid_sum(lpq, s.bar, epoch, s.info, &s_fail, s.part, 1, sh, &pq, s.wait_ns))
            break;
        if (pq == 0.0)
        {
            if (lead)
            {
                s.info[0] = it - 1;
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 4ull);
            }
            break;
        }
        const float al = (float)(rr / pq);
        double lrr = 0;
        for (int64_t k = gt; k < s.ndof; k += T)
        {
            const float pn = ld_keep(pnew + k, pl);
            st_keep(x + k, ld_keep(x + k, pl) + al * pn, pl);
            const float rv = ld_keep(r + k, pl) - al * ld_keep(q + k, pl);
            st_keep(r + k, rv, pl);
            lrr += (double)rv * (double)rv;
        }
        double rn;
        if (!grid_sum(lrr, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rn, s.wait_ns))
            break;
        const bool done = rn <= stop;
        if (done || it >= s.maxit)
        {
            if (lead)
            {
                s.info[0] = it;
                reinterpret_cast<double *>(s.info)[3] = rn;
                if (!done)
                    atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 1ull);
            }
            break;
        }
        beta = (float)(rn / rr);
        rr = rn;
        float *t = pold;
        pold = pnew;
        pnew = t;
    }
    // the copy in flight ends before the block's shared memory is given back
    if (has)
        mbar_wait_bounded(bar, parity, kBarrierTimeoutNs);
}

// ---- helpers for the mixed-precision refinement
template <typename TA, typename TB>
__global__ void k_convert(int64_t m, const TA *__restrict__ a, TB *__restrict__ b)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        b[k] = (TB)a[k];
}

__global__ void k_add_f32(int64_t m, const float *__restrict__ d, double *__restrict__ x)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        x[k] += (double)d[k];
}

// r = b - K x (FP64), partial ||r||^2 per block
template <int D>
__global__ void __launch_bounds__(256) k_residual64(int n, int nslices, const int *__restrict__ rowptr,
                                                    const int *__restrict__ perm, const int64_t *__restrict__ slice_off,
                                                    const int *__restrict__ col_sell, const double *__restrict__ K,
                                                    const double *__restrict__ b, const double *__restrict__ x,
                                                    double *__restrict__ r, double *__restrict__ part)
{
    __shared__ double sh[32];
    const int W = (gridDim.x * blockDim.x) >> 5;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    double loc = 0;
    for (int sl = gw; sl < nslices; sl += W)
    {
        double acc[D];
        const int i = spmv_slice<double, double, D>(sl, n, rowptr, perm, slice_off, col_sell, K, x, x, 0.0, acc,
                                                    l2_evict_first(), l2_evict_last());
        if (i >= 0)
            for (int c = 0; c < D; ++c)
            {
                const int64_t k = (int64_t)i * D + c;
                const double v = b[k] - acc[c];
                r[k] = v;
                loc += v * v;
            }
    }
    block_partial(loc, part, 0, sh);
}

__global__ void k_sum_partials(int nblk, const double *__restrict__ part, double *__restrict__ out)
{
    __shared__ double sh[32];
    double v = 0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x)
        v += part[2 * b];
    v = wsum(v);
    if ((threadIdx.x & 31) == 0)
        sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32)
    {
        double t = (threadIdx.x < blockDim.x / 32) ? sh[threadIdx.x] : 0.0;
        t = wsum(t);
        if (threadIdx.x == 0)
            *out = t;
    }
}

// The default CG grid: one block per SM (kCGMinBlocks per SM when they fit), at most one block per
// slice.  Every grid up to it is co-resident, as the cooperative launch needs.
template <typename TK, typename TV, int D>
static cudaError_t cg_grid_rule(const Problem &p, int *grid_out)
{
    static int occ_cache[2][2][4] = {};
    int &occ = occ_cache[sizeof(TK) == 8][sizeof(TV) == 8][D];
    if (occ == 0)
    {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_cg<TK, TV, D, false>, kCGThreads, 0);
        if (e != cudaSuccess)
            return e;
        if (occ < 1)
            occ = 1;
    }
    int grid = p.num_sms * std::min(occ, kCGMinBlocks);
    if (grid > p.nslices)
        grid = std::max(1, p.nslices);
    if (grid > kMaxGridBlocks)
        grid = kMaxGridBlocks;
    *grid_out = grid;
    return cudaSuccess;
}

// k_cg's RES form on `grid` blocks: columns of a warp at most, 0 where it does not serve, which is where
// a block has more than half a slice per warp or its matrix does not fit (2D FP64: above four slices a
// block, 18,900 rows).  It is the faster form wherever it fits.
template <typename TK, int D>
static size_t resident_bytes(int steps)
{
    return (size_t)(kCGThreads / 32) * steps * kSlice * (D * D * sizeof(TK) + sizeof(int));
}
template <typename TK, int D>
static int resident_steps(const Problem &p, int grid)
{
    const int nw = kCGThreads / 32, most = div_up(p.nslices, grid);
    if (2 * most > nw)
        return 0;
    const int steps = div_up(p.max_conns, column_split(most, nw));
    return resident_bytes<TK, D>(steps) <= kDynamicSmem ? steps : 0;
}

// Waits for the CG launch between the handle's two events and reads its status words.
static cudaError_t finish_cg(Problem &p, const char *what, CGResult &out, double *rr_final, bool *declined)
{
    cudaError_t e;
    if ((e = cudaEventRecord(p.cg_ev[1], p.stream)) != cudaSuccess)
        return e;
    if ((e = cudaMemcpyAsync(p.cg_info_host, p.cg_info, 4 * sizeof(int64_t), cudaMemcpyDeviceToHost, p.stream)) !=
        cudaSuccess)
        return e;
    if ((e = cudaStreamSynchronize(p.stream)) != cudaSuccess)
        return e;
    if (declined && (p.cg_info_host[1] & kBondDeclined))
    {
        *declined = true;
        p.bo_valid = false; // so does every other solve with this K
        return cudaSuccess;
    }
    out.iters += p.cg_info_host[0];
    p.ctr.cg_iters += p.cg_info_host[0];
    {
        float ms = 0;
        if (cudaEventElapsedTime(&ms, p.cg_ev[0], p.cg_ev[1]) == cudaSuccess)
            p.ctr.cg_kernel_seconds += ms * 1e-3;
        static const bool log = std::getenv("LPMGPU_LOG") != nullptr;
        if (log)
            std::fprintf(stderr, "lpmgpu cg launch %lld: %s %s/%dd n=%d iters=%lld ms=%.3f\n",
                         (long long)p.ctr.cg_launches, what, p.cg_form, p.dim, p.n, (long long)p.cg_info_host[0], ms);
    }
    if (p.cg_info_host[1] & 1)
        out.maxit_hits++;
    if (p.cg_info_host[1] & 2)
        out.timeout = true;
    if (p.cg_info_host[1] & 4)
        out.breakdown = true;
    if (rr_final)
        *rr_final = reinterpret_cast<double *>(p.cg_info_host)[3];
    return cudaSuccess;
}

template <typename TK, typename TV, int D>
static cudaError_t run_cg(Problem &p, const TK *K, const TV *b, TV *x, TV *r, TV *pa, TV *pb, TV *q, double rtol,
                          double atol, double abs_stop, int64_t maxit, CGResult &out, double *rr_final)
{
    cudaError_t e;
    int grid = 0;
    if ((e = cg_grid_rule<TK, TV, D>(p, &grid)) != cudaSuccess)
        return e;
    if (p.cg_grid > 0 && p.cg_grid < grid)
        grid = p.cg_grid; // a tuned grid only ever lowers the default, so it stays co-resident
    CGState s;
    s.n = p.n;
    s.nslices = p.nslices;
    s.ndof = (int64_t)p.n * D;
    s.rowptr = p.cstart;
    s.perm = p.perm;
    s.slice_off = p.slice_off;
    s.col_sell = p.col_sell;
    s.rtol = rtol;
    s.atol = atol;
    s.abs_stop = abs_stop;
    s.maxit = maxit;
    s.bar = p.barrier;
    s.part = p.partials;
    s.info = p.cg_info;
    s.wait_ns = p.wait_ns;
    s.steps = 0;
    if ((e = cudaMemsetAsync(p.barrier, 0, 2 * sizeof(unsigned), p.stream)) != cudaSuccess)
        return e;
    if ((e = cudaMemsetAsync(p.cg_info, 0, 4 * sizeof(int64_t), p.stream)) != cudaSuccess)
        return e;
    void *args[] = {&s, &K, &b, &x, &r, &pa, &pb, &q};
    if ((e = cudaEventRecord(p.cg_ev[0], p.stream)) != cudaSuccess)
        return e;
    // the streamed form where every block has more than half a slice per warp, so no columns are split
    if (sizeof(TV) == 4 && D == 3 && 2 * (p.nslices / grid) > kCGThreads / 32)
    {
        p.cg_form = "streamed";
        if ((e = cudaFuncSetAttribute(k_cg_stream, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStreamSmem)) !=
            cudaSuccess)
            return e;
        e = cudaLaunchCooperativeKernel((const void *)k_cg_stream, dim3(grid), dim3(kCGThreads), args, kStreamSmem,
                                        p.stream);
    }
    else if (resident_steps<TK, D>(p, grid) > 0)
    {
        p.cg_form = "resident";
        s.steps = resident_steps<TK, D>(p, grid);
        const size_t smem = resident_bytes<TK, D>(s.steps);
        if ((e = allow_dynamic_smem((const void *)k_cg<TK, TV, D, true>)) != cudaSuccess)
            return e;
        e = cudaLaunchCooperativeKernel((const void *)k_cg<TK, TV, D, true>, dim3(grid), dim3(kCGThreads), args, smem,
                                        p.stream);
    }
    else
    {
        p.cg_form = "general";
        e = cudaLaunchCooperativeKernel((const void *)k_cg<TK, TV, D, false>, dim3(grid), dim3(kCGThreads), args, 0,
                                        p.stream);
    }
    if (e != cudaSuccess)
        return e;
    p.ctr.kernel_launches++;
    p.ctr.cg_launches++;
    return finish_cg(p, sizeof(TK) == 8 ? "assembled fp64" : "assembled fp32", out, rr_final, nullptr);
}

// K x = b on the bond form of the K assembled last (bond_op.cu), in one cluster when the problem fits
// one, else on the whole grid.  *declined: this K has no bond form, nothing was solved.
template <typename TV>
static cudaError_t run_bond(Problem &p, const TV *b, TV *x, TV *r, TV *pa, TV *pb, double rtol, double atol,
                            double abs_stop, int64_t maxit, CGResult &out, double *rr_final, bool *declined)
{
    cudaError_t e;
    *declined = false;
    if ((e = cudaEventRecord(p.cg_ev[0], p.stream)) != cudaSuccess)
        return e;
    const char *what = sizeof(TV) == 8 ? "bond fp64" : "bond fp32";
    if constexpr (sizeof(TV) == 8)
    {
        if (bond_cluster_fits(p))
            e = enqueue_bond_cluster(p, b, x, rtol, atol, abs_stop, maxit);
        else
            e = enqueue_bond_grid<TV>(p, b, x, r, pa, pb, rtol, atol, abs_stop, maxit);
    }
    else
        e = enqueue_bond_grid<TV>(p, b, x, r, pa, pb, rtol, atol, abs_stop, maxit);
    if (e != cudaSuccess)
        return e;
    return finish_cg(p, what, out, rr_final, declined);
}

// K x = b on the assembled matrix: small 2D FP64 problems in one cluster, the others on the grid
template <typename TK, typename TV, int D>
static cudaError_t run_assembled(Problem &p, const TK *K, const TV *b, TV *x, TV *r, TV *pa, TV *pb, TV *q, double rtol,
                                 double atol, double abs_stop, int64_t maxit, CGResult &out, double *rr_final)
{
    if constexpr (D == 2 && sizeof(TV) == 8)
        if (sell_cluster_fits(p))
        {
            cudaError_t e = cudaEventRecord(p.cg_ev[0], p.stream);
            if (e == cudaSuccess)
                e = enqueue_sell_cluster(p, b, x, rtol, atol, abs_stop, maxit);
            return e != cudaSuccess ? e : finish_cg(p, "assembled fp64", out, rr_final, nullptr);
        }
    return run_cg<TK, TV, D>(p, K, b, x, r, pa, pb, q, rtol, atol, abs_stop, maxit, out, rr_final);
}

template <int D>
static cudaError_t solve_dim(Problem &p, CGResult &out)
{
    const int64_t ndof = (int64_t)p.n * D;
    const int64_t maxit = p.desc.cg_maxit > 0 ? p.desc.cg_maxit : ndof;
    bool declined = false;
    if (p.bo_valid && (p.desc.precision != LPMGPU_MIXED || bond_cluster_fits(p)))
    {
        // Mixed precision in the cluster form: its bonds are in shared memory and its iterations are
        // bound by latency, not by bytes, so the correction is solved for in FP64 at once.  The caller's
        // cap, though, holds for each inner solve of a refinement, which goes on from one that reached it:
        // then the refinement below is run instead, as if this solve had not been.
        CGResult at_once;
        double rr = 0.0;
        const cudaError_t e = run_bond<double>(p, p.res, p.x, p.r, p.p0, p.p1, p.desc.cg_rtol, p.desc.cg_atol, -1.0,
                                               maxit, at_once, &rr, &declined);
        if (e != cudaSuccess)
            return e;
        const bool mixed = p.desc.precision == LPMGPU_MIXED;
        if (!declined && !(mixed && at_once.maxit_hits > 0 && std::isfinite(rr)))
        {
            out = at_once;
            out.refinements += mixed ? 1 : 0;
            return cudaSuccess;
        }
    }
    if (p.desc.precision != LPMGPU_MIXED)
        return run_assembled<double, double, D>(p, p.K, p.res, p.x, p.r, p.p0, p.p1, p.q, p.desc.cg_rtol,
                                                p.desc.cg_atol, -1.0, maxit, out, nullptr);
    // FP32 Krylov solve inside FP64 iterative refinement on the same stopping rule
    cudaError_t e;
    // rr0 = ||b||^2 via r = b - K*0
    if ((e = cudaMemsetAsync(p.x, 0, sizeof(double) * ndof, p.stream)) != cudaSuccess)
        return e;
    auto true_residual = [&](double &val) -> cudaError_t {
        cudaError_t e2 = enqueue_true_residual(p);
        if (e2 == cudaSuccess)
            e2 = cudaStreamSynchronize(p.stream);
        val = true_residual_result(p);
        return e2;
    };
    double rr0 = 0, rr = 0;
    if ((e = true_residual(rr0)) != cudaSuccess)
        return e;
    const double stop = p.desc.cg_rtol * rr0 + p.desc.cg_atol;
    rr = rr0;
    // The refinement's last step leaves a smooth error of up to 4e-9 of the solution in 3D (and below
    // 3e-10 in 2D) that depends on every rounding of its inner solves; 3D keeps the matrix that its
    // callers' results are reproducible with.
    bool bond = D == 2 && p.bo_valid && !declined;
    for (int ref = 0; ref < 30 && !(rr <= stop); ++ref)
    {
        if ((e = enqueue_r_to_b32(p)) != cudaSuccess)
            return e;
        // the inner solve aims a little below the outer target, measured on its own residual
        CGResult inner;
        double rr_in = 0;
        bool off = !bond;
        if constexpr (D == 2)
            if (bond && (e = run_bond<float>(p, p.b32, p.x32, p.r32, p.pa32, p.pb32, 0.0, 0.0, 0.25 * stop, maxit,
                                             inner, &rr_in, &off)) != cudaSuccess)
                return e;
        bond = !off;
        if (off && (e = run_cg<float, float, D>(p, p.K32, p.b32, p.x32, p.r32, p.pa32, p.pb32, p.q32, 0.0, 0.0, 0.25 * stop,
                                         maxit, inner, &rr_in)) != cudaSuccess)
            return e;
        out.iters += inner.iters;
        out.maxit_hits += inner.maxit_hits;
        out.timeout = out.timeout || inner.timeout;
        out.breakdown = out.breakdown || inner.breakdown;
        out.refinements++;
        if (inner.timeout)
            break;
        if ((e = enqueue_add_x32(p)) != cudaSuccess)
            return e;
        if ((e = true_residual(rr)) != cudaSuccess)
            return e;
        if (inner.iters == 0)
            break;
    }
    return cudaSuccess;
}

// r = b - K x (FP64 matrix) and ||r||^2 -> the pinned slot read by true_residual_result
cudaError_t enqueue_true_residual(Problem &p)
{
    const int64_t ndof = (int64_t)p.n * p.dim;
    const int nb_res = std::min(div_up(ndof, 256), 4 * p.num_sms);
    double *dst = reinterpret_cast<double *>(p.cg_info) + 5;
    if (p.dim == 2)
        k_residual64<2><<<nb_res, 256, 0, p.stream>>>(p.n, p.nslices, p.cstart, p.perm, p.slice_off, p.col_sell, p.K,
                                                      p.res, p.x, p.r, p.partials);
    else
        k_residual64<3><<<nb_res, 256, 0, p.stream>>>(p.n, p.nslices, p.cstart, p.perm, p.slice_off, p.col_sell, p.K,
                                                      p.res, p.x, p.r, p.partials);
    k_sum_partials<<<1, 256, 0, p.stream>>>(nb_res, p.partials, dst);
    p.ctr.kernel_launches += 2;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    return cudaMemcpyAsync(p.cg_info_host + 5, dst, sizeof(double), cudaMemcpyDeviceToHost, p.stream);
}

double true_residual_result(const Problem &p)
{
    return reinterpret_cast<const double *>(p.cg_info_host)[5];
}

cudaError_t enqueue_r_to_b32(Problem &p)
{
    const int64_t ndof = (int64_t)p.n * p.dim;
    k_convert<double, float><<<std::min(div_up(ndof, 256), 8 * p.num_sms), 256, 0, p.stream>>>(ndof, p.r, p.b32);
    p.ctr.kernel_launches++;
    return cudaGetLastError();
}

cudaError_t enqueue_res_to_b32(Problem &p)
{
    const int64_t ndof = (int64_t)p.n * p.dim;
    k_convert<double, float><<<std::min(div_up(ndof, 256), 8 * p.num_sms), 256, 0, p.stream>>>(ndof, p.res, p.b32);
    p.ctr.kernel_launches++;
    return cudaGetLastError();
}

cudaError_t enqueue_add_x32(Problem &p)
{
    const int64_t ndof = (int64_t)p.n * p.dim;
    k_add_f32<<<std::min(div_up(ndof, 256), 8 * p.num_sms), 256, 0, p.stream>>>(ndof, p.x32, p.x);
    p.ctr.kernel_launches++;
    return cudaGetLastError();
}

__global__ void k_to_f32(int64_t m, const double *__restrict__ a, float *__restrict__ b)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        b[k] = (float)a[k];
}

cudaError_t launch_k_to_f32(Problem &p)
{
    const int64_t m = p.nsb * p.dim * p.dim * kSlice;
    k_to_f32<<<std::min(div_up(m, 256), 16 * p.num_sms), 256, 0, p.stream>>>(m, p.K, p.K32);
    p.ctr.kernel_launches++;
    return cudaGetLastError();
}

cudaError_t solve_linear(Problem &p, CGResult &out)
{
    return p.dim == 2 ? solve_dim<2>(p, out) : solve_dim<3>(p, out);
}

// ---- autotuner of the CG launch shape (no counterpart in the reference)
//
// A persistent CG's cost per iteration is its matrix or bond stream plus two grid sums (2.0 us each).  On
// large problems every SM streams and the default grid (one block per SM) is best; on small ones
// the barriers dominate and fewer, fuller blocks can be faster.  The tuner times `iterations` CG
// iterations of this problem's own matrix for each candidate grid (the default and its 3/4, 1/2,
// 1/4, 1/8, 1/16), twice each, and keeps the fastest by its second timing.  Candidates are never
// above the default, so every one is co-resident.  For a problem that runs in one cluster the grid is
// the cluster's CTAs (rounded down to a power of two that still holds the problem).
template <typename TK, typename TV, int D>
static cudaError_t tune_dim(Problem &p, int iterations, lpmgpu_tune_result *res, const TK *K, const TV *b, TV *x,
                            TV *r, TV *pa, TV *pb, TV *q)
{
    int g0 = 0;
    const int saved = p.cg_grid;
    p.cg_grid = 0;
    const bool cluster = p.bo_valid && bond_cluster_fits(p);
    bool bond = cluster || (p.bo_valid && (sizeof(TV) == 8 || D == 2));
    // the solve that solve_dim runs: the bond form (FP64 in one cluster whatever the precision), or the
    // assembled matrix for a K without one
    auto solve = [&](CGResult &cr) -> cudaError_t {
        bool off = !bond;
        cudaError_t e2 = cudaSuccess;
        if (bond && cluster)
            e2 = run_bond<double>(p, p.diag_raw, p.x, p.r, p.p0, p.p1, 0.0, 0.0, 0.0, iterations, cr, nullptr, &off);
        else if constexpr (sizeof(TV) == 8 || D == 2)
        {
            if (bond)
                e2 = run_bond<TV>(p, b, x, r, pa, pb, 0.0, 0.0, 0.0, iterations, cr, nullptr, &off);
        }
        if (e2 == cudaSuccess && off)
            e2 = run_assembled<TK, TV, D>(p, K, b, x, r, pa, pb, q, 0.0, 0.0, 0.0, iterations, cr, nullptr);
        return e2;
    };
    cudaError_t e = cudaSuccess;
    if (bond)
    { // whether this K has a bond form is known once a launch has looked at its flags
        int flag = 0;
        e = cudaMemcpyAsync(&flag, &p.scal->bond_flag, sizeof(int), cudaMemcpyDeviceToHost, p.stream);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(p.stream);
        bond = (flag & bond_flags_bad(p)) == 0;
    }
    if (e == cudaSuccess)
        e = bond ? bond_default_grid<TV>(p, &g0) : cg_grid_rule<TK, TV, D>(p, &g0);
    p.cg_grid = saved;
    if (e != cudaSuccess)
        return e;
    std::vector<int> cand;
    for (int f : {16, 12, 8, 4, 2, 1}) // 16/16, 12/16, ... of the default
    {
        const int g = std::max(1, g0 * f / 16);
        if (std::find(cand.begin(), cand.end(), g) == cand.end() && (int)cand.size() < LPMGPU_TUNE_MAX)
            cand.push_back(g);
    }
    const lpmgpu_counters ctr = p.ctr;
    int best = g0;
    double best_us = 0;
    res->ncandidates = (int32_t)cand.size();
    for (size_t k = 0; k < cand.size(); ++k)
    {
        p.cg_grid = cand[k] == g0 ? 0 : cand[k]; // the default's own form is the one timed for it
        double us = 0;
        for (int rep = 0; rep < 2 && e == cudaSuccess; ++rep)
        {
            CGResult cr;
            e = solve(cr);
            float ms = 0;
            if (e == cudaSuccess && (e = cudaEventElapsedTime(&ms, p.cg_ev[0], p.cg_ev[1])) == cudaSuccess)
                us = cr.iters > 0 ? 1e3 * ms / (double)cr.iters : 0.0;
            if (cr.timeout)
            {
                set_last_error("a device-side barrier wait timed out while tuning the CG kernel");
                e = cudaErrorLaunchTimeout;
            }
        }
        if (e != cudaSuccess)
            break;
        res->grid[k] = cand[k];
        res->us_per_iter[k] = us;
        if (us > 0 && (best_us == 0 || us < best_us))
        {
            best_us = us;
            best = cand[k];
        }
    }
    p.ctr = ctr; // tuning launches do not count as solves
    p.cg_grid = (e == cudaSuccess) ? (best == g0 ? 0 : best) : saved;
    res->grid_default = g0;
    res->grid_chosen = best;
    return e;
}

} // namespace lpm

extern "C" {

int32_t lpmgpu_set_cg_grid(lpmgpu_solver *h, int32_t grid)
{
    if (!h || grid < 0)
        return LPMGPU_ERR_INVALID_ARG;
    h->p.cg_grid = grid;
    return LPMGPU_OK;
}

int32_t lpmgpu_set_wait_limit_ns(lpmgpu_solver *h, int64_t ns)
{
    if (!h)
        return LPMGPU_ERR_INVALID_ARG;
    h->p.wait_ns = ns > 0 ? (unsigned long long)ns : lpm::kBarrierTimeoutNs;
    return LPMGPU_OK;
}

int32_t lpmgpu_autotune(lpmgpu_solver *h, int32_t iterations, lpmgpu_tune_result *out)
{
    using namespace lpm;
    if (!h || !out || iterations < 1 || iterations > 100000)
        return LPMGPU_ERR_INVALID_ARG;
    *out = lpmgpu_tune_result{};
    Problem &p = h->p;
    cudaError_t e = cudaSetDevice(p.device);
    // K from the current state, as the next load step assembles it; the right-hand side is the
    // diagonal before the BC elimination, which is nonzero for every row
    if (e == cudaSuccess)
        e = enqueue_assemble(p, true);
    const int64_t ndof = (int64_t)p.n * p.dim;
    if (e == cudaSuccess && p.desc.precision == LPMGPU_MIXED)
    {
        k_convert<double, float><<<std::min(div_up(ndof, 256), 8 * p.num_sms), 256, 0, p.stream>>>(ndof, p.diag_raw,
                                                                                                   p.b32);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
    {
        out->precision = p.desc.precision;
        if (p.desc.precision == LPMGPU_MIXED)
            e = p.dim == 2 ? tune_dim<float, float, 2>(p, iterations, out, p.K32, p.b32, p.x32, p.r32, p.pa32, p.pb32,
                                                       p.q32)
                           : tune_dim<float, float, 3>(p, iterations, out, p.K32, p.b32, p.x32, p.r32, p.pa32, p.pb32,
                                                       p.q32);
        else
            e = p.dim == 2 ? tune_dim<double, double, 2>(p, iterations, out, p.K, p.diag_raw, p.x, p.r, p.p0, p.p1, p.q)
                           : tune_dim<double, double, 3>(p, iterations, out, p.K, p.diag_raw, p.x, p.r, p.p0, p.p1, p.q);
    }
    if (e == cudaErrorLaunchTimeout)
        return LPMGPU_ERR_TIMEOUT;
    if (e != cudaSuccess)
    {
        set_last_error(std::string("lpmgpu_autotune: ") + cudaGetErrorString(e));
        return LPMGPU_ERR_CUDA;
    }
    return LPMGPU_OK;
}

} // extern "C"

// ---------------------------------------------------------------------------------------
// Allocation-free CG on a caller-supplied block-CSR matrix.
//
// Some callers cannot allocate device memory.  A plugin that runs inside a host program which
// owns all device memory through its own pool or arena may not call cudaMalloc behind that
// allocator's back, and a latency-bound loop cannot afford cudaMalloc/cudaFree, which may
// synchronise the whole device.  For them the solve below takes every input and output from
// the caller and keeps its own work vectors, reduction partials and barrier words in the
// file-scope array g_noalloc_scratch, which every GPU that loads this library holds (about
// 8 MiB) until the process exits.
//
// Limits and caveats:
//  * at most kNoAllocMaxDof unknowns (rows * dim); larger systems are rejected;
//  * all calls on a device share the one array and it keeps the last call's contents, so
//    calls that overlap on the GPU (two streams, two host threads) race; serialise them;
//  * the first call on a device looks up the array's device address (set-up) and should
//    come before any stream capture begins; a cudaDeviceReset of that device invalidates the
//    looked-up address, so the entry point must not be used after one;
//  * the call waits for its stream before returning, and reports a solve that reached its
//    iteration cap (LPMGPU_ERR_CG_MAXIT) or broke down with p.Ap == 0 (LPMGPU_ERR_CG_BREAKDOWN).
namespace lpm
{

constexpr int64_t kNoAllocMaxDof = int64_t(1) << 18; // 262,144 unknowns
constexpr int kNoAllocMaxBlocks = 1024;
// r, p_a, p_b, q | per-block partials [2*blocks] | status words [4] | barrier [2]
constexpr int64_t kNoAllocDoubles = 4 * kNoAllocMaxDof + 2 * kNoAllocMaxBlocks + 4 + 2;
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

struct CGBsr
{
    int nrows;
    int64_t ndof;
    const int *__restrict__ rowptr;
    const int *__restrict__ col;
    const double *__restrict__ val; // row-major d x d blocks
    double rtol, atol;
    int64_t maxit;
    unsigned *bar;
    double *part;
    int64_t *info;
};

// One row of q = A (r + beta p_old), by a warp.  The row's blocks are contiguous, so the lanes read
// its values in order: lane l holds entry l % 4 of every eighth block.  kBsrUnroll blocks of a lane are in
// flight, their columns fetched one group ahead.  Lane c < D returns q's component c.
constexpr int kBsrUnroll = 4;
__device__ __forceinline__ double bsr_row(const CGBsr &s, int row, const double *r, const double *pold, double beta,
                                          uint64_t pm, uint64_t pl)
{
    constexpr int D = 2, E = 4, KB = 8;
    const int lane = threadIdx.x & 31, e = lane % E, kb = lane / E, c = e % D;
    const int end = s.rowptr[row + 1];
    int bk = s.rowptr[row] + kb;
    double acc = 0.0;
    int jn[kBsrUnroll];
#pragma unroll
    for (int u = 0; u < kBsrUnroll; ++u)
        jn[u] = (bk + u * KB < end) ? ld_stream(s.col + bk + u * KB, pm) : 0;
    for (; bk < end; bk += kBsrUnroll * KB)
    {
        double v[kBsrUnroll], xr[kBsrUnroll], xp[kBsrUnroll];
#pragma unroll
        for (int u = 0; u < kBsrUnroll; ++u)
        {
            const int k = bk + u * KB, j = jn[u], k2 = k + kBsrUnroll * KB;
            v[u] = xr[u] = xp[u] = 0.0;
            if (k < end)
            {
                v[u] = ld_stream(s.val + (int64_t)k * E + e, pm);
                xr[u] = ld_keep(r + (int64_t)j * D + c, pl);
                xp[u] = ld_keep(pold + (int64_t)j * D + c, pl);
            }
            jn[u] = (k2 < end) ? ld_stream(s.col + k2, pm) : 0;
        }
#pragma unroll
        for (int u = 0; u < kBsrUnroll; ++u)
            if (bk + u * KB < end)
                acc += v[u] * (xr[u] + beta * xp[u]);
    }
    // entry (i, c) of the KB lanes that share it, then the row i's D entries
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    return __shfl_sync(0xffffffffu, acc, (lane & 1) * 2);
}

// The CG of k_cg on a caller's block-CSR matrix in 2D: a warp per row, each block a contiguous share of
// the rows.  Bound by the two grid sums (2.0 us each) and the latency of the matrix loads (from L2 while
// it fits) at four blocks in flight per lane.  Serves what does not fit one cluster (cg_cluster.cu): 11,000
// hexagonal rows 5.7 ms a solve.
__global__ void __launch_bounds__(kCGThreads, kCGMinBlocks)
    k_cg_bsr_noalloc(CGBsr s, const double *__restrict__ b, double *__restrict__ x, double *r, double *pa, double *pb,
                     double *q)
{
    constexpr int D = 2;
    __shared__ double sh[32];
    __shared__ int s_fail;
    if (threadIdx.x == 0)
        s_fail = 0;
    __syncthreads();
    unsigned epoch = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int row0 = (int)((int64_t)blockIdx.x * s.nrows / gridDim.x),
              row1 = (int)((int64_t)(blockIdx.x + 1) * s.nrows / gridDim.x);
    const int64_t k0 = (int64_t)row0 * D, k1 = (int64_t)row1 * D;
    const int64_t bytes = (int64_t)s.rowptr[s.nrows] * (D * D * 8 + 4);
    const uint64_t pl = l2_evict_last(), pm = bytes <= ((int64_t)90 << 20) ? pl : l2_evict_first();
    double loc = 0;
    for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x)
    {
        const double v = b[k];
        st_keep(r + k, v, pl);
        x[k] = 0.0;
        st_keep(pa + k, 0.0, pl);
        loc += v * v;
    }
    double rr;
    if (!grid_sum(loc, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rr, kBarrierTimeoutNs))
        return;
    const double stop = s.rtol * rr + s.atol;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        s.info[0] = 0;
    if (rr <= stop)
        return;
    double beta = 0.0;
    double *pold = pa, *pnew = pb;
    for (int64_t it = 1;; ++it)
    {
        double lpq = 0;
        for (int row = row0 + warp; row < row1; row += nw)
        {
            const double qv = bsr_row(s, row, r, pold, beta, pm, pl);
            if (lane < D)
            {
                const int64_t k = (int64_t)row * D + lane;
                const double pn = ld_keep(r + k, pl) + beta * ld_keep(pold + k, pl);
                st_keep(pnew + k, pn, pl);
                st_keep(q + k, qv, pl);
                lpq += pn * qv;
            }
        }
        double pq;
        if (!grid_sum(lpq, s.bar, epoch, s.info, &s_fail, s.part, 1, sh, &pq, kBarrierTimeoutNs))
            return;
        if (pq == 0.0)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                s.info[0] = it - 1;
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 4ull);
            }
            return;
        }
        const double alpha = rr / pq;
        double lrr = 0;
        for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) // the block's own rows
        {
            x[k] = x[k] + alpha * ld_keep(pnew + k, pl);
            const double rv = ld_keep(r + k, pl) - alpha * ld_keep(q + k, pl);
            st_keep(r + k, rv, pl);
            lrr += rv * rv;
        }
        double rn;
        if (!grid_sum(lrr, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rn, kBarrierTimeoutNs))
            return;
        if (rn <= stop || it >= s.maxit)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                s.info[0] = it;
                if (!(rn <= stop))
                    atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 1ull);
            }
            return;
        }
        beta = rn / rr;
        rr = rn;
        double *t = pold;
        pold = pnew;
        pnew = t;
    }
}

// 32 blocks of a row at most: row, first block, end of the row's blocks
struct BsrChunk
{
    int row, k, end;
    __device__ __forceinline__ int count() const { return min(32, end - k); }
    __device__ __forceinline__ bool last() const { return k + 32 >= end; }
    // the next chunk of rows [ra, rb), after the last one the first
    __device__ __forceinline__ BsrChunk next(const int *__restrict__ rowptr, int ra, int rb) const
    {
        BsrChunk c = *this;
        if (last())
        {
            const bool wrap = row + 1 >= rb;
            c.row = wrap ? ra : row + 1;
            c.k = wrap ? rowptr[ra] : end;
            c.end = rowptr[c.row + 1];
        }
        else
            c.k += 32;
        return c;
    }
};

// The CG on a caller's block-CSR matrix in 3D.  A block has a contiguous share of the rows, a warp a
// contiguous share of those, which it walks in chunks of at most 32 blocks of a row, a lane per block.  A
// chunk's values come by bulk copy into one of the warp's two buffers while the chunk before it is used,
// its columns a chunk earlier still; both go on over the grid sums, since the matrix stays.  r and p are
// gathered a chunk ahead in registers.  Bound by the shared-memory and L1 wavefronts of the values (18 a
// chunk, 8 bytes at a stride of 72) and of the gathers (36), 26,000 -> 20,000 cycles a product of 105 rows
// per SM.  Whole solves, lanes over a row's entries as in k_cg_bsr_noalloc -> here: SC 15,625 rows (68 MB)
// 12.3 -> 9.9 ms, SC 1,728 2.5 -> 1.95, FCC 7,488 6.2 -> 5.4, BCC 11,664 7.8 -> 7.4.  Threads 384 / 512 /
// 640 / 768: 11.8 / 10.0 / 9.9 / 10.3 ms; asynchronous copies by the lanes in place of the bulk copies
// 10.9; gathers and copies two chunks ahead 10.7.  In 2D, with 8 to 31 blocks a row, a chunk leaves lanes
// idle: 5,700 -> 6,240 us at 11,000 hexagonal rows, so 2D keeps k_cg_bsr_noalloc.
constexpr int kBsrThreads = 640;
constexpr int kBsrBuf = 32 * 9 + 2; // doubles of a chunk and its odd start
constexpr size_t kBsrSmem = sizeof(double) * 2 * kBsrBuf * (kBsrThreads / 32);

__global__ void __launch_bounds__(kBsrThreads, 1)
    k_cg_bsr_chunks(CGBsr s, const double *__restrict__ b, double *__restrict__ x, double *r, double *pa, double *pb,
                    double *q)
{
    constexpr int D = 3, E = 9;
    extern __shared__ __align__(16) double bsr_sm[];
    __shared__ uint64_t full[2 * (kBsrThreads / 32)];
    __shared__ double sh[32];
    __shared__ int s_fail;
    if (threadIdx.x == 0)
        s_fail = 0;
    unsigned epoch = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = (int)((int64_t)blockIdx.x * s.nrows / gridDim.x),
              row1 = (int)((int64_t)(blockIdx.x + 1) * s.nrows / gridDim.x);
    const int ra = row0 + (row1 - row0) * warp / (kBsrThreads / 32),
              rb = row0 + (row1 - row0) * (warp + 1) / (kBsrThreads / 32);
    double *buf = bsr_sm + 2 * kBsrBuf * warp;
    uint64_t *bar = full + 2 * warp;
    if (lane == 0)
    {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        mbar_init_fence();
    }
    __syncthreads();
    const int64_t k0 = (int64_t)row0 * D, k1 = (int64_t)row1 * D;
    const int64_t bytes = (int64_t)s.rowptr[s.nrows] * (E * 8 + 4);
    const uint64_t pl = l2_evict_last(), pm = bytes <= ((int64_t)90 << 20) ? pl : l2_evict_first();
    // the warp's chunks go round its rows: c0 is used next and its copy is in flight, c1 follows it
    auto phase = [&](const BsrChunk &c) { return (int)((reinterpret_cast<uintptr_t>(s.val + (int64_t)c.k * E) >> 3) & 1); };
    // the entry of chunk c that this lane fetches by itself (the 16-byte copies leave out odd ends), or -1
    auto odd_entry = [&](const BsrChunk &c) {
        const int nd = c.count() * E, ph = phase(c);
        return lane == 0 ? (ph && nd > 0 ? 0 : -1) : lane == 1 && nd > ph && ((nd - ph) & 1) ? nd - 1 : -1;
    };
    double odd = 0.0;
    auto copy = [&](const BsrChunk &c, int to) {
        const double *src = s.val + (int64_t)c.k * E;
        const int ph = phase(c), oe = odd_entry(c), np = c.count() > 0 ? (c.count() * E - ph) >> 1 : 0;
        if (oe >= 0)
            odd = ld_stream(src + oe, pm);
        if (lane == 0)
            bulk_refill(buf + to * kBsrBuf + 2 * ph, src + ph, (uint32_t)(16 * np), bar + to, pm);
    };
    auto column = [&](const BsrChunk &c) { return lane < c.count() ? ld_stream(s.col + c.k + lane, pm) : 0; };
    BsrChunk c0 = {0, 0, 0}, c1 = c0;
    int j0 = 0, j1 = 0, flip = 0;
    unsigned parity = 0; // bit f: the parity that buffer f completes next
    bool dead = false;   // a copy did not come in time
    if (ra < rb)
    {
        c0 = {ra, s.rowptr[ra], s.rowptr[ra + 1]};
        copy(c0, 0);
        c1 = c0.next(s.rowptr, ra, rb);
        j0 = column(c0);
        j1 = column(c1);
    }
    double loc = 0;
    for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x)
    {
        const double v = b[k];
        st_keep(r + k, v, pl);
        x[k] = 0.0;
        st_keep(pa + k, 0.0, pl);
        loc += v * v;
    }
    double rr = 0.0;
    bool go = grid_sum(loc, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rr, kBarrierTimeoutNs);
    const double stop = s.rtol * rr + s.atol;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        s.info[0] = 0;
    go = go && !(rr <= stop);
    double beta = 0.0;
    double *pold = pa, *pnew = pb;
    for (int64_t it = 1; go; ++it)
    {
        double lpq = 0;
        if (ra < rb && !dead)
        {
            double gr[D], gp[D], xv[D], acc[D];
            auto gather = [&](const BsrChunk &c, int j) {
                if (lane < c.count())
#pragma unroll
                    for (int a = 0; a < D; ++a)
                    {
                        gr[a] = ld_keep(r + (int64_t)j * D + a, pl);
                        gp[a] = ld_keep(pold + (int64_t)j * D + a, pl);
                    }
            };
#pragma unroll
            for (int a = 0; a < D; ++a)
                gr[a] = gp[a] = acc[a] = 0.0;
            gather(c0, j0);
            for (;;)
            {
#pragma unroll
                for (int a = 0; a < D; ++a)
                    xv[a] = gr[a] + beta * gp[a];
                const bool more = !(c0.last() && c0.row + 1 >= rb);
                const double odd0 = odd;
                copy(c1, flip ^ 1);
                if (more)
                    gather(c1, j1);
                // p of the row, for the lanes that will store it
                const int comp = lane >> 3;
                const bool owner = c0.last() && (lane & 7) == 0 && comp < D;
                const int64_t ok = (int64_t)c0.row * D + comp;
                double ro = 0.0, po = 0.0;
                if (owner)
                {
                    ro = ld_keep(r + ok, pl);
                    po = ld_keep(pold + ok, pl);
                }
                const BsrChunk c2 = c1.next(s.rowptr, ra, rb);
                const int j2 = column(c2);
                if (!mbar_wait_bounded(bar + flip, (parity >> flip) & 1, kBarrierTimeoutNs))
                    dead = true;
                dead = __any_sync(0xffffffffu, dead);
                if (dead)
                {
                    atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 2ull);
                    s_fail = 1;
                    break;
                }
                parity ^= 1 << flip;
                const int oe = odd_entry(c0);
                if (oe >= 0)
                    buf[flip * kBsrBuf + phase(c0) + oe] = odd0;
                __syncwarp();
                if (lane < c0.count())
                {
                    const double *v = buf + flip * kBsrBuf + phase(c0) + lane * E;
#pragma unroll
                    for (int a = 0; a < D; ++a)
#pragma unroll
                        for (int e = 0; e < D; ++e)
                            acc[a] += v[a * D + e] * xv[e];
                }
                if (c0.last())
                {
                    // sums over the lanes: lane 8 h ends with component h
                    const bool up = lane & 16, up2 = lane & 8;
                    double u0 = up ? acc[2] : acc[0], u1 = up ? 0.0 : acc[1];
                    u0 += __shfl_xor_sync(0xffffffffu, up ? acc[0] : acc[2], 16);
                    u1 += __shfl_xor_sync(0xffffffffu, up ? acc[1] : 0.0, 16);
                    double t = (up2 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, up2 ? u0 : u1, 8);
                    t += __shfl_xor_sync(0xffffffffu, t, 4);
                    t += __shfl_xor_sync(0xffffffffu, t, 2);
                    t += __shfl_xor_sync(0xffffffffu, t, 1);
                    if (owner)
                    {
                        const double pn = ro + beta * po;
                        st_keep(pnew + ok, pn, pl);
                        st_keep(q + ok, t, pl);
                        lpq += pn * t;
                    }
#pragma unroll
                    for (int a = 0; a < D; ++a)
                        acc[a] = 0.0;
                }
                __syncwarp();
                c0 = c1;
                j0 = j1;
                c1 = c2;
                j1 = j2;
                flip ^= 1;
                if (!more)
                    break;
            }
        }
        double pq;
        if (!grid_sum(lpq, s.bar, epoch, s.info, &s_fail, s.part, 1, sh, &pq, kBarrierTimeoutNs))
            break;
        if (pq == 0.0)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                s.info[0] = it - 1;
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 4ull);
            }
            break;
        }
        const double alpha = rr / pq;
        double lrr = 0;
        for (int64_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) // the block's own rows
        {
            x[k] = x[k] + alpha * ld_keep(pnew + k, pl);
            const double rv = ld_keep(r + k, pl) - alpha * ld_keep(q + k, pl);
            st_keep(r + k, rv, pl);
            lrr += rv * rv;
        }
        double rn;
        if (!grid_sum(lrr, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rn, kBarrierTimeoutNs))
            break;
        if (rn <= stop || it >= s.maxit)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
            {
                s.info[0] = it;
                if (!(rn <= stop))
                    atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 1ull);
            }
            break;
        }
        beta = rn / rr;
        rr = rn;
        double *t = pold;
        pold = pnew;
        pnew = t;
    }
    // the copy in flight ends before the block's shared memory is given back
    if (ra < rb)
    {
        mbar_wait_bounded(bar + flip, (parity >> flip) & 1, kBarrierTimeoutNs);
        if (dead)
            mbar_wait_bounded(bar + (flip ^ 1), (parity >> (flip ^ 1)) & 1, kBarrierTimeoutNs);
    }
}

// The device address of the array in the current device's context, looked up on every call (the
// lookup allocates nothing): a cached address would dangle after the host application resets the
// device or re-creates its context, which reloads the module.
static cudaError_t noalloc_scratch(int dev, double **out)
{
    if (dev < 0)
        return cudaErrorInvalidDevice;
    double *ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_noalloc_scratch);
    if (e != cudaSuccess)
        return e;
    *out = ptr;
    return cudaSuccess;
}

template <int D>
static cudaError_t noalloc_launch(double *scr, int grid, const CGBsr &s0, const double *b, double *x,
                                  cudaStream_t stream, int64_t *status)
{
    CGBsr s = s0;
    double *r = scr, *pa = scr + kNoAllocMaxDof, *pb = scr + 2 * kNoAllocMaxDof, *q = scr + 3 * kNoAllocMaxDof;
    s.part = scr + 4 * kNoAllocMaxDof;
    s.info = reinterpret_cast<int64_t *>(s.part + 2 * kNoAllocMaxBlocks);
    s.bar = reinterpret_cast<unsigned *>(s.info + 4);
    // the barrier words and status must start at zero; the vectors are written before use
    cudaError_t e = cudaMemsetAsync(s.info, 0, 4 * sizeof(int64_t) + 2 * sizeof(double), stream);
    if (e != cudaSuccess)
        return e;
    void *args[] = {&s, &b, &x, &r, &pa, &pb, &q};
    if constexpr (D == 2)
        e = cudaLaunchCooperativeKernel((const void *)k_cg_bsr_noalloc, dim3(grid), dim3(kCGThreads), args, 0, stream);
    else if ((e = cudaFuncSetAttribute(k_cg_bsr_chunks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBsrSmem)) ==
             cudaSuccess)
        e = cudaLaunchCooperativeKernel((const void *)k_cg_bsr_chunks, dim3(grid), dim3(kBsrThreads), args, kBsrSmem, stream);
    if (e != cudaSuccess)
        return e;
    e = cudaMemcpyAsync(status, s.info, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess)
        return e;
    return cudaStreamSynchronize(stream);
}

} // namespace lpm

extern "C" int32_t lpmgpu_cg_bsr_noalloc(int32_t dim, int32_t nrows, const int32_t *rowptr, const int32_t *colidx,
                                         const double *values, const double *b, double *x, double rtol, double atol,
                                         int64_t maxit, void *stream, int64_t *iterations)
{
    using namespace lpm;
    if ((dim != 2 && dim != 3) || nrows <= 0 || !rowptr || !colidx || !values || !b || !x)
        return LPMGPU_ERR_INVALID_ARG;
    if ((int64_t)nrows * dim > kNoAllocMaxDof)
    {
        set_last_error("lpmgpu_cg_bsr_noalloc: more than 262144 unknowns (the size of its static scratch)");
        return LPMGPU_ERR_INVALID_ARG;
    }
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    double *scr = nullptr;
    if (e == cudaSuccess)
        e = noalloc_scratch(dev, &scr);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess)
    {
        set_last_error(std::string("lpmgpu_cg_bsr_noalloc: ") + cudaGetErrorString(e));
        return e == cudaErrorNoDevice ? LPMGPU_ERR_NO_DEVICE : LPMGPU_ERR_CUDA;
    }
    const int warps = (dim == 2 ? kCGThreads : kBsrThreads) / 32;
    int grid = std::min(sms, kNoAllocMaxBlocks); // one block per SM
    grid = std::min(grid, (nrows + warps - 1) / warps); // a row per warp
    grid = std::max(grid, 1);
    CGBsr s{};
    s.nrows = nrows;
    s.ndof = (int64_t)nrows * dim;
    s.rowptr = rowptr;
    s.col = colidx;
    s.val = values;
    s.rtol = rtol;
    s.atol = atol;
    s.maxit = maxit > 0 ? maxit : s.ndof;
    int64_t status[2] = {0, 0};
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    bool solved = false;
    if (bsr_cluster_may_fit(dim, nrows))
    {
        int64_t *info = reinterpret_cast<int64_t *>(scr + 4 * kNoAllocMaxDof + 2 * kNoAllocMaxBlocks);
        e = cudaMemsetAsync(info, 0, 4 * sizeof(int64_t), st);
        if (e == cudaSuccess)
            e = enqueue_bsr_cluster(dim, nrows, rowptr, colidx, values, b, x, rtol, atol, s.maxit, info, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(status, info, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
        solved = e != cudaSuccess || !(status[1] & kCgDeclined);
    }
    if (!solved)
        e = (dim == 2) ? noalloc_launch<2>(scr, grid, s, b, x, st, status) : noalloc_launch<3>(scr, grid, s, b, x, st, status);
    if (e != cudaSuccess)
    {
        set_last_error(std::string("lpmgpu_cg_bsr_noalloc: ") + cudaGetErrorString(e));
        return LPMGPU_ERR_CUDA;
    }
    if (iterations)
        *iterations = status[0];
    // status bits of k_cg_bsr_noalloc: 2 a barrier wait timed out, 4 p.Ap == 0, 1 cap reached
    if (status[1] & 2)
    {
        set_last_error("lpmgpu_cg_bsr_noalloc: a device-side barrier wait timed out");
        return LPMGPU_ERR_TIMEOUT;
    }
    if (status[1] & 4)
    {
        set_last_error("lpmgpu_cg_bsr_noalloc: CG broke down (p.Ap == 0: the matrix is singular or indefinite)");
        return LPMGPU_ERR_CG_BREAKDOWN;
    }
    if (status[1] & 1)
    {
        set_last_error("lpmgpu_cg_bsr_noalloc: CG reached its iteration cap without meeting the tolerance");
        return LPMGPU_ERR_CG_MAXIT;
    }
    return LPMGPU_OK;
}
