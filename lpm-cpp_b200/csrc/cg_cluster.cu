// CGs of small systems inside one thread-block cluster: the matrix rows of a CTA stay in its shared
// memory, every CTA holds all of r and p, and an iteration exchanges the CTAs' parts of r (one bulk copy
// to each of the others) and their sums.  Both kernels run the loop of k_cg (cg.cu) with its stopping
// rule and status words.
//
// k_cg on the grid pays two barriers of 2 us per iteration whatever the size; here an exchange takes
// about 0.4 us.  The solves are bound by the chain of exchanges, block synchronisations and warp sums.
#include <algorithm>
#include <atomic>

#include "cg_cluster.cuh"
#include "cluster.cuh"
#include "shares.cuh"

namespace lpm
{

// ---- host helpers of cluster.cuh
int max_cluster(const void *kernel)
{
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    {
        (void)cudaGetLastError();
        return 0;
    }
    for (int nc = 16; nc >= 8; nc /= 2)
    {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(nc);
        cfg.blockDim = dim3(1024);
        cfg.dynamicSmemBytes = kClusterSmem;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nc;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int k = 0;
        if (cudaOccupancyMaxActiveClusters(&k, kernel, &cfg) == cudaSuccess && k > 0)
            return nc;
        (void)cudaGetLastError();
    }
    return 0;
}

cudaError_t launch_cluster(const void *kernel, int nc, int threads, size_t smem, void **args, cudaStream_t st)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = nc;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

constexpr int kThreads = 1024;
constexpr int kMaxCtas = 16;

// ---- the assembled 2D system
//
// The sums are k_cg's on its default grid for these sizes, one slice per block: there 16 warps share a
// slice, part t taking its block columns t, t + 16, ..., and the 16 partial rows are added in order; a
// slice's p.q is a block's partial; r.r is summed over 32 consecutive unknowns, 32 of those, and blocks.
// Every value is formed by the same operations in the same order, so the solve keeps its bits.
//
// Every CTA has slices (shares.cuh), which is what orders the exchanges: a CTA stores into another's pq, g
// and r and counts bytes on its mbarriers only after that CTA's own slices' sums of the phase before, so
// none is ever a phase behind what arrives.
//
// Bound by shared-memory bandwidth (the product reads 36 bytes per block, its 16 partial rows go
// through memory, p and r are whole vectors) and by 60 cycles per level of each warp sum.  A plate of
// 1,840 particles: 6.9 us per iteration on the grid, 5.7 here; 1,050: 6.3 and 4.6.
struct SellCG
{
    int n, nslices, per, width; // most slices of a CTA, most block columns of a slice
    const int *rowptr, *perm, *iperm, *col;
    const int64_t *slice_off;
    const double *K, *b;
    double *x;
    double rtol, atol, abs_stop;
    int64_t maxit;
    int64_t *info;
    unsigned long long wait_ns;
};

constexpr int kSellParts = 16;      // kMaxColumnSplit: the parts of a slice alone in its block
constexpr int kSellMaxSlices = 128; // their sums and those of their unknowns fit the arrays below
static_assert(kSellParts == kMaxColumnSplit, "the parts of k_cg's column split");

struct SellShared
{
    unsigned long long mbar[3]; // [0] r of the other CTAs, [1] the slices' p.q, [2] the groups' r.r
    double pq[kSellMaxSlices];
    double g[kSellMaxSlices * 2]; // sums over 32 consecutive unknowns
    double alpha;
    double tot;
    int fail;
};
constexpr size_t kSellFixed = (sizeof(SellShared) + 127) / 128 * 128;

static size_t sell_smem(int nslices, int per, int width)
{
    const size_t rows = (size_t)nslices * 32;
    const size_t red = (size_t)per * kSellParts * 64 * 8, vec = rows * 16;
    return kSellFixed + (size_t)per * width * 32 * (32 + 2) + std::max(red, vec) + vec + rows * 2 + (size_t)per * 32;
}

// ||r||^2 from the r that every CTA holds, into tot: each CTA sums its share of the groups of 32
// consecutive unknowns and sends them to all
__device__ __forceinline__ void sell_rr(SellShared *sh, const double *r, const unsigned short *pos, int ndof, unsigned par,
                                        unsigned long long wait_ns)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned nc = gridDim.x, bar = smem_addr(&sh->mbar[2]);
    const int ng = (ndof + 31) / 32, nb = (ng + 31) / 32, share = (ng + nc - 1) / nc;
    const int g0 = min(ng, (int)blockIdx.x * share), g1 = min(ng, g0 + share);
    for (int g = g0 + warp; g < g1; g += nw)
    {
        const int k = g * 32 + lane;
        double e = 0.0;
        if (k < ndof)
        {
            const double v = r[2 * pos[k >> 1] + (k & 1)];
            e += v * v;
        }
        e = wsum(e);
        if (lane < (int)nc)
            push(mapa(smem_addr(&sh->g[g]), lane), mapa(bar, lane), e);
    }
    if (warp == 0)
    {
        if (lane == 0)
            expect_bytes(bar, 8u * ng);
        __syncwarp();
        const bool ok = __all_sync(0xffffffffu, cluster_wait(bar, par, wait_ns));
        double mine = 0.0; // lane b: the sum of block b of 1,024 unknowns
        for (int b0 = 0; b0 < nb; b0 += 4)
        {
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = 32 * (b0 + u) + lane < ng ? sh->g[32 * (b0 + u) + lane] : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = wsum(v[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (lane == b0 + u)
                    mine = v[u];
        }
        mine = wsum(mine);
        if (lane == 0)
        {
            sh->tot = 0.0 + mine;
            if (!ok)
                sh->fail = 1;
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads, 1) k_cg_sell_cluster(SellCG s)
{
    extern __shared__ __align__(128) unsigned char csm[];
    SellShared *sh = reinterpret_cast<SellShared *>(csm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned nc = gridDim.x, rank = blockIdx.x; // the grid is one cluster
    const int rows = s.nslices * 32, ndof = 2 * s.n;
    const int sl0 = share_begin(s.nslices, nc, rank), ns = share_begin(s.nslices, nc, rank + 1) - sl0;
    // shared memory: the slices' blocks, r (whose place the partial rows take during the product), p,
    // the blocks' columns, each particle's position
    const size_t red_bytes = (size_t)s.per * kSellParts * 64 * 8, vec_bytes = (size_t)rows * 16;
    double *Ks = reinterpret_cast<double *>(csm + kSellFixed);
    double *r = Ks + (size_t)s.per * s.width * 32 * 4, *red = r;
    double *p = r + (red_bytes > vec_bytes ? red_bytes : vec_bytes) / 8;
    unsigned short *cS = reinterpret_cast<unsigned short *>(p + (size_t)rows * 2);
    unsigned short *pos = cS + (size_t)s.per * s.width * 32;
    unsigned char *cnt = reinterpret_cast<unsigned char *>(pos + rows); // blocks of the own rows
    const unsigned barR = smem_addr(&sh->mbar[0]), barP = smem_addr(&sh->mbar[1]);
    if (threadIdx.x == 0)
    {
        sh->fail = 0;
        for (int k = 0; k < 3; ++k)
            mbar_init(&sh->mbar[k]);
        mbar_init_done();
    }
    for (int i = threadIdx.x; i < s.n; i += blockDim.x)
        pos[i] = (unsigned short)s.iperm[i];
    for (int q = threadIdx.x; q < rows; q += blockDim.x)
    {
        const int i = q < s.n ? s.perm[q] : -1;
#pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            r[2 * q + c] = i >= 0 ? s.b[2 * (int64_t)i + c] : 0.0;
            p[2 * q + c] = 0.0;
        }
    }
    for (int e = threadIdx.x; e < ns * s.width * 32; e += blockDim.x)
    {
        const int l = e & 31, t = (e >> 5) % s.width, ls = (e >> 5) / s.width;
        const int64_t off = s.slice_off[sl0 + ls];
        const int w = (int)(s.slice_off[sl0 + ls + 1] - off);
        if (t >= w)
            continue;
        cS[e] = (unsigned short)s.iperm[s.col[(off + t) * 32 + l]];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            Ks[(size_t)(e >> 5) * 128 + k * 32 + l] = s.K[((off + t) * 4 + k) * 32 + l];
    }
    for (int q = threadIdx.x; q < ns * 32; q += blockDim.x)
    {
        const int i = sl0 * 32 + q < s.n ? s.perm[sl0 * 32 + q] : -1;
        cnt[q] = (unsigned char)(i >= 0 ? s.rowptr[i + 1] - s.rowptr[i] : 0);
    }
    // the rows of this warp's slice, when it closes one
    const int own = warp < ns ? (sl0 + warp) * 32 + lane : rows;
    const int oi = own < s.n ? s.perm[own] : -1;
    double rv[2] = {0.0, 0.0}, xv[2] = {0.0, 0.0};
    if (oi >= 0)
    {
        rv[0] = s.b[2 * (int64_t)oi];
        rv[1] = s.b[2 * (int64_t)oi + 1];
    }
    cluster_sync();
    unsigned par2 = 0;
    sell_rr(sh, r, pos, ndof, par2, s.wait_ns);
    double rr = sh->tot;
    const double stop = (s.abs_stop >= 0) ? s.abs_stop : s.rtol * rr + s.atol;
    const bool lead = rank == 0 && threadIdx.x == 0;
    if (lead)
    {
        s.info[0] = 0;
        reinterpret_cast<double *>(s.info)[2] = rr;
        reinterpret_cast<double *>(s.info)[3] = rr;
    }
    double beta = 0.0;
    unsigned par = 0;
    for (int64_t it = 1; !sh->fail && !(rr <= stop); ++it, par ^= 1)
    {
        for (int q = threadIdx.x; q < 2 * rows; q += blockDim.x)
            p[q] = r[q] + beta * p[q];
        __syncthreads();
        // the parts of the slices' rows
        for (int task = warp; task < ns * kSellParts; task += nw)
        {
            const int ls = task / kSellParts, part = task % kSellParts;
            const int m = cnt[ls * 32 + lane];
            double a0 = 0.0, a1 = 0.0;
            for (int k = part; k < m; k += kSellParts)
            {
                const int e = (ls * s.width + k) * 32;
                const double2 v = reinterpret_cast<const double2 *>(p)[cS[e + lane]];
                const double *kb = Ks + (size_t)e * 4 + lane;
                a0 += kb[0] * v.x;
                a0 += kb[32] * v.y;
                a1 += kb[64] * v.x;
                a1 += kb[96] * v.y;
            }
            red[task * 64 + lane] = a0;
            red[task * 64 + 32 + lane] = a1;
        }
        __syncthreads();
        double q0 = 0.0, q1 = 0.0, p0 = 0.0, p1 = 0.0;
        if (warp < ns)
        {
            const double *t = red + warp * kSellParts * 64 + lane;
            double v[2 * kSellParts];
#pragma unroll
            for (int k = 0; k < kSellParts; ++k)
            {
                v[2 * k] = t[k * 64];
                v[2 * k + 1] = t[k * 64 + 32];
            }
            q0 = v[0];
            q1 = v[1];
#pragma unroll
            for (int k = 1; k < kSellParts; ++k)
            {
                q0 += v[2 * k];
                q1 += v[2 * k + 1];
            }
            double lpq = 0.0;
            if (oi >= 0)
            {
                p0 = p[2 * own];
                p1 = p[2 * own + 1];
                lpq += p0 * q0;
                lpq += p1 * q1;
            }
            lpq = wsum(lpq);
            fence_async(); // the others' copies of r take the partial rows' place
            if (lane < (int)nc)
                push(mapa(smem_addr(&sh->pq[sl0 + warp]), lane), mapa(barP, lane), lpq);
        }
        if (warp == 0)
        {
            if (lane == 0)
            {
                expect_bytes(barP, 8u * s.nslices);
                expect_bytes(barR, 512u * (s.nslices - ns));
            }
            __syncwarp();
            const bool ok = __all_sync(0xffffffffu, cluster_wait(barP, par, s.wait_ns));
            double t = 0.0;
            for (int g = 0; g < s.nslices; g += 32)
                t += wsum(g + lane < s.nslices ? sh->pq[g + lane] : 0.0);
            if (lane == 0)
            {
                sh->tot = t;
                sh->alpha = rr / t;
                if (!ok)
                    sh->fail = 1;
            }
        }
        __syncthreads();
        if (sh->fail)
            break;
        if (sh->tot == 0.0)
        {
            if (lead)
            {
                s.info[0] = it - 1;
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 4ull);
            }
            break;
        }
        const double al = sh->alpha;
        if (warp < ns)
        {
            if (oi >= 0)
            {
                xv[0] = xv[0] + al * p0;
                xv[1] = xv[1] + al * p1;
                rv[0] = rv[0] - al * q0;
                rv[1] = rv[1] - al * q1;
            }
            reinterpret_cast<double2 *>(r)[own] = make_double2(rv[0], rv[1]);
            fence_async();
        }
        __syncthreads();
        if (warp == 0)
        {
            if (lane < (int)nc && lane != (int)rank)
                push_bulk(r + 64 * sl0, lane, barR, 512u * ns);
            __syncwarp();
            if (!__all_sync(0xffffffffu, cluster_wait(barR, par, s.wait_ns)) && lane == 0)
                sh->fail = 1;
        }
        __syncthreads();
        if (sh->fail)
            break;
        par2 ^= 1;
        sell_rr(sh, r, pos, ndof, par2, s.wait_ns);
        const double rn = sh->tot;
        if (sh->fail)
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
        beta = rn / rr;
        rr = rn;
    }
    if (sh->fail && threadIdx.x == 0)
        atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 2ull);
    if (sh->fail)
        drain_pushes();
    if (oi >= 0)
    {
        s.x[2 * (int64_t)oi] = xv[0];
        s.x[2 * (int64_t)oi + 1] = xv[1];
    }
    cluster_sync(); // no CTA leaves while another may still write into its shared memory
}

static int sell_ctas()
{
    static std::atomic<int> known{-1};
    int v = known.load();
    if (v < 0)
    {
        v = max_cluster((const void *)k_cg_sell_cluster);
        known.store(v);
    }
    return v;
}

bool sell_cluster_fits(const Problem &p)
{
    const int nc = sell_ctas();
    if (p.dim != 2 || nc < 1 || p.cg_grid > 0 || p.nslices > std::min(kSellMaxSlices, p.num_sms) || p.n > 0xffff)
        return false;
    return sell_smem(p.nslices, share_most(p.nslices, share_ctas(p.nslices, nc)), p.max_conns) <= kClusterSmem;
}

cudaError_t enqueue_sell_cluster(Problem &p, const double *b, double *x, double rtol, double atol, double abs_stop,
                                 int64_t maxit)
{
    cudaError_t e = cudaMemsetAsync(p.cg_info, 0, 4 * sizeof(int64_t), p.stream);
    if (e != cudaSuccess)
        return e;
    SellCG s;
    const int nc = share_ctas(p.nslices, sell_ctas());
    s.n = p.n;
    s.nslices = p.nslices;
    s.per = share_most(p.nslices, nc);
    s.width = p.max_conns;
    s.rowptr = p.cstart;
    s.perm = p.perm;
    s.iperm = p.iperm;
    s.col = p.col_sell;
    s.slice_off = p.slice_off;
    s.K = p.K;
    s.b = b;
    s.x = x;
    s.rtol = rtol;
    s.atol = atol;
    s.abs_stop = abs_stop;
    s.maxit = maxit;
    s.info = p.cg_info;
    s.wait_ns = p.wait_ns;
    p.cg_form = "cluster";
    void *args[] = {&s};
    e = launch_cluster((const void *)k_cg_sell_cluster, nc, kThreads, sell_smem(s.nslices, s.per, s.width), args, p.stream);
    if (e == cudaSuccess)
    {
        p.ctr.kernel_launches++;
        p.ctr.cg_launches++;
    }
    return e;
}

// ---- the allocation-free CG
//
// CTA k owns `per` rows; every CTA holds all of r and p, sends its part of r to the others by one bulk
// copy each, and forms p itself.  Solve of 1,085 rows in 2D: 1.42 ms on the grid, 0.95 ms here (1.36 ms
// with each row of r pushed only into the CTAs whose blocks reach it: a packet per row and target costs
// more than whole copies; 1.36 ms with 512 threads).
struct BsrCG
{
    int nrows, per; // rows, rows per CTA (even: the parts of r are whole 16-byte pieces)
    const int *rowptr, *col;
    const double *val, *b;
    double *x;
    double rtol, atol;
    int64_t maxit;
    int64_t *info;
};

struct BsrShared
{
    unsigned long long mbar[2]; // [0] r and r.r of the CTAs, [1] their p.q
    double part[2][kMaxCtas];
    double sum[32];
    double tot[2];
    int fail;
};
constexpr size_t kBsrFixed = (sizeof(BsrShared) + 127) / 128 * 128;

// the sum of v over the cluster: warp 0 exchanges the CTAs' sums (and waits for `halo` bytes of copies on
// the same mbarrier); every thread must call it, and finds the sum in tot[which]
template <typename F>
__device__ __forceinline__ void bsr_exchange(BsrShared *sh, unsigned nc, unsigned rank, int which, unsigned par,
                                             unsigned halo, double v, F copies)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = wsum(v);
    if (lane == 0)
        sh->sum[warp] = v;
    __syncthreads();
    if (warp == 0)
    {
        const unsigned bar = smem_addr(&sh->mbar[which]);
        copies(bar);
        double t = lane < (int)(blockDim.x >> 5) ? sh->sum[lane] : 0.0;
        t = wsum(t);
        if (lane < (int)nc)
            push(mapa(smem_addr(&sh->part[which][rank]), lane), mapa(bar, lane), t);
        if (lane == 0)
            expect_bytes(bar, halo + 8u * nc);
        __syncwarp();
        const bool ok = __all_sync(0xffffffffu, cluster_wait(bar, par, kBarrierTimeoutNs));
        t = wsum(lane < (int)nc ? sh->part[which][lane] : 0.0);
        if (lane == 0)
        {
            sh->tot[which] = t;
            if (!ok)
                sh->fail = 1;
        }
    }
    __syncthreads();
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1) k_cg_bsr_cluster(BsrCG s)
{
    constexpr int E = D * D, KB = D == 2 ? 8 : 3;
    extern __shared__ __align__(128) unsigned char csm[];
    BsrShared *sh = reinterpret_cast<BsrShared *>(csm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned nc = gridDim.x, rank = blockIdx.x;
    const int all = (int)nc * s.per; // rows held, the last ones past the end zero
    const int a0 = min(s.nrows, (int)rank * s.per), a1 = min(s.nrows, a0 + s.per), ns = a1 - a0;
    // the matrix's most blocks of a CTA; every CTA looks at all shares, so all decide alike
    int most = 0;
    for (unsigned k = 0; k < nc; ++k)
        most = max(most, s.rowptr[min(s.nrows, (int)(k + 1) * s.per)] - s.rowptr[min(s.nrows, (int)k * s.per)]);
    if (kBsrFixed + 8 * (2 * (size_t)all * D + 2 * (size_t)s.per * D) + (size_t)most * (8 * E + 4) + 4 * ((size_t)s.per + 1) >
        kClusterSmem)
    {
        if (rank == 0 && threadIdx.x == 0)
            s.info[1] = kCgDeclined;
        return;
    }
    double *r = reinterpret_cast<double *>(csm + kBsrFixed), *p = r + (size_t)all * D;
    double *xs = p + (size_t)all * D, *qs = xs + (size_t)s.per * D;
    double *val = qs + (size_t)s.per * D;
    int *col = reinterpret_cast<int *>(val + (size_t)most * E), *rp = col + most;
    if (threadIdx.x == 0)
    {
        sh->fail = 0;
        mbar_init(&sh->mbar[0]);
        mbar_init(&sh->mbar[1]);
        mbar_init_done();
    }
    const int b0 = s.rowptr[a0], nblk = s.rowptr[a1] - b0;
    for (int k = threadIdx.x; k < nblk * E; k += blockDim.x)
        val[k] = s.val[(int64_t)b0 * E + k];
    for (int k = threadIdx.x; k < nblk; k += blockDim.x)
        col[k] = s.col[b0 + k] * D;
    for (int k = threadIdx.x; k <= ns; k += blockDim.x)
        rp[k] = s.rowptr[a0 + k] - b0;
    for (int k = threadIdx.x; k < all * D; k += blockDim.x)
    {
        r[k] = k < s.nrows * D ? s.b[k] : 0.0;
        p[k] = 0.0;
    }
    double loc = 0.0;
    for (int k = threadIdx.x; k < ns * D; k += blockDim.x)
    {
        xs[k] = 0.0;
        loc += s.b[a0 * D + k] * s.b[a0 * D + k];
    }
    cluster_sync();
    unsigned par0 = 0, par1 = 0;
    auto none = [](unsigned) {};
    // the sum of p.q tells the others that r may be overwritten: its reads come before their copies
    auto read = [](unsigned) { fence_async(); };
    bsr_exchange(sh, nc, rank, 0, par0, 0u, loc, none);
    par0 ^= 1;
    double rr = sh->tot[0];
    const double stop = s.rtol * rr + s.atol;
    const bool lead = rank == 0 && threadIdx.x == 0;
    if (lead)
        s.info[0] = 0;
    double beta = 0.0;
    const unsigned rbytes = 8u * D * s.per; // one CTA's part of r
    for (int64_t it = 1; !sh->fail && !(rr <= stop); ++it)
    {
        for (int k = threadIdx.x; k < all * D; k += blockDim.x)
            p[k] = r[k] + beta * p[k];
        __syncthreads();
        // q = A p, a warp per row: bsr_row's lanes (cg.cu)
        double lpq = 0.0;
        const int e = lane % E, kb = lane / E, c = e % D;
        for (int row = warp; row < ns; row += nw)
        {
            const int k1 = kb < KB ? rp[row + 1] : 0;
            double acc = 0.0;
#pragma unroll 4
            for (int k = rp[row] + kb; k < k1; k += KB)
                acc += val[k * E + e] * p[col[k] + c];
            if constexpr (D == 2)
            {
                acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                acc += __shfl_xor_sync(0xffffffffu, acc, 8);
                acc += __shfl_xor_sync(0xffffffffu, acc, 16);
                acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                acc = __shfl_sync(0xffffffffu, acc, (lane & 1) * 2);
            }
            else
            {
                acc = acc + __shfl_sync(0xffffffffu, acc, (lane + 9) & 31) + __shfl_sync(0xffffffffu, acc, (lane + 18) & 31);
                acc = acc + __shfl_sync(0xffffffffu, acc, (lane + 1) & 31) + __shfl_sync(0xffffffffu, acc, (lane + 2) & 31);
                acc = __shfl_sync(0xffffffffu, acc, (lane % 3) * 3);
            }
            if (lane < D)
            {
                qs[row * D + lane] = acc;
                lpq += p[(a0 + row) * D + lane] * acc;
            }
        }
        bsr_exchange(sh, nc, rank, 1, par1, 0u, lpq, read);
        par1 ^= 1;
        const double pq = sh->tot[1];
        if (sh->fail)
            break;
        if (pq == 0.0)
        {
            if (lead)
            {
                s.info[0] = it - 1;
                s.info[1] = 4;
            }
            break;
        }
        const double al = rr / pq;
        double lrr = 0.0;
        for (int k = threadIdx.x; k < ns * D; k += blockDim.x)
        {
            xs[k] = xs[k] + al * p[a0 * D + k];
            const double v = r[a0 * D + k] - al * qs[k];
            r[a0 * D + k] = v;
            lrr += v * v;
        }
        fence_async();
        bsr_exchange(sh, nc, rank, 0, par0, rbytes * (nc - 1), lrr, [&](unsigned bar) {
            // the places of r behind the last row are zero in every CTA: whole parts are copied
            if (lane < (int)nc && lane != (int)rank)
                push_bulk(r + (size_t)rank * s.per * D, lane, bar, rbytes);
        });
        par0 ^= 1;
        const double rn = sh->tot[0];
        if (sh->fail)
            break;
        if (rn <= stop || it >= s.maxit)
        {
            if (lead)
            {
                s.info[0] = it;
                s.info[1] = rn <= stop ? 0 : 1;
            }
            break;
        }
        beta = rn / rr;
        rr = rn;
    }
    for (int k = threadIdx.x; k < ns * D; k += blockDim.x)
        s.x[a0 * D + k] = xs[k];
    if (sh->fail)
        drain_pushes();
    cluster_sync();
    if (sh->fail && threadIdx.x == 0)
        atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 2ull);
}

static int bsr_ctas()
{
    static std::atomic<int> known{-1};
    int v = known.load();
    if (v < 0)
    {
        v = std::min(max_cluster((const void *)k_cg_bsr_cluster<2>), max_cluster((const void *)k_cg_bsr_cluster<3>));
        known.store(v);
    }
    return v;
}

static int bsr_rows(int nrows, int nc) { return std::max(2, (div_up(nrows, nc) + 1) / 2 * 2); }

bool bsr_cluster_may_fit(int dim, int nrows)
{
    const int nc = bsr_ctas();
    if (nc < 1)
        return false;
    // all rows' vectors, and 15 blocks for each own row (a sparser matrix is a matter of the grid)
    const size_t per = bsr_rows(nrows, nc);
    return kBsrFixed + 8 * dim * (2 * per * nc + 2 * per) + per * 15 * (8 * dim * dim + 4) <= kClusterSmem;
}

cudaError_t enqueue_bsr_cluster(int dim, int nrows, const int *rowptr, const int *col, const double *val, const double *b,
                                double *x, double rtol, double atol, int64_t maxit, int64_t *info, cudaStream_t st)
{
    const int nc = bsr_ctas();
    BsrCG s{nrows, bsr_rows(nrows, nc), rowptr, col, val, b, x, rtol, atol, maxit, info};
    void *args[] = {&s};
    return launch_cluster(dim == 2 ? (const void *)k_cg_bsr_cluster<2> : (const void *)k_cg_bsr_cluster<3>, nc, kThreads,
                          kClusterSmem, args, st);
}

} // namespace lpm
