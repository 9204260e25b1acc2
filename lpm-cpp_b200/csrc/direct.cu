// Direct solve of the Newton system: the device counterpart of Solver::LPM_PARDISO
// (include/solver.h:191-274), which the reference's SolverMode::PARDISO runs in place of its CG.
//
//   * Ordering (host, once per problem): reverse Cuthill-McKee over the particle connection graph
//     (the conns of assembly.h:237-266) narrows the band; particle i's unknowns become
//     d * rank(i) + r.  The half-bandwidth is kd = d * max |rank(i) - rank(j)| over connected
//     pairs + d - 1.
//   * Band fill (device): the BC-eliminated stiffness, read from its sliced-ELL blocks, into the
//     permuted lower band (band_chol.cuh's layout).
//   * Factorisation (device, once per assembled K: K is fixed through a load step's Newton
//     iterations, solver_static.h:107-118): blocked band Cholesky in column blocks of kBandNB in
//     one persistent launch.
//   * Solve (device, every Newton iteration): forward and backward substitution on the factor, in
//     one CTA.
// The band costs n * (kd + 1) doubles; 2D plates fit easily, wide 3D bands are rejected with
// LPMGPU_ERR_OUT_OF_MEMORY before anything is allocated.  A pivot that is not positive (a
// singular or indefinite K, e.g. a particle left without bonds) is LPMGPU_ERR_NOT_SPD.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "band_chol.cuh"
#include "bulk_copy.cuh"
#include "cg_device.cuh"
#include "cluster.cuh"

namespace lpm
{

constexpr int kBandNB = 32;                       // column block of the factorisation and solves
constexpr int64_t kBandMaxBytes = int64_t(32) << 30; // band storage limit per problem (32 GiB)

// Reverse Cuthill-McKee over a graph in CSR (rows ascending ids, self loops allowed): rank[i] is
// i's position.  Each connected component starts at a pseudo-peripheral vertex (the last vertex
// reached by two breadth-first sweeps from its lowest-degree vertex); neighbours join in
// ascending degree, then id.  When the given order (the identity) has a band at most as wide,
// it is kept instead.  Returns the largest |rank(i) - rank(j)| over the edges.
int64_t rcm_order(int n, const int *start, const int *adj, int *rank)
{
    std::vector<int> deg(n), order;
    order.reserve(n);
    for (int i = 0; i < n; ++i)
        deg[i] = start[i + 1] - start[i];
    std::vector<char> seen(n, 0);
    std::vector<int> level(n, -1), byid(n);
    for (int i = 0; i < n; ++i)
        byid[i] = i;
    std::stable_sort(byid.begin(), byid.end(), [&](int a, int b) { return deg[a] < deg[b]; });
    auto bfs_last = [&](int s) {
        // the last vertex of a breadth-first sweep from s inside its component
        std::vector<int> q{s};
        level[s] = 0;
        size_t h = 0;
        int last = s;
        while (h < q.size())
        {
            const int v = q[h++];
            last = v;
            for (int k = start[v]; k < start[v + 1]; ++k)
                if (level[adj[k]] < 0)
                {
                    level[adj[k]] = level[v] + 1;
                    q.push_back(adj[k]);
                }
        }
        for (int v : q)
            level[v] = -1;
        return last;
    };
    std::vector<int> nb;
    for (int s0 : byid)
    {
        if (seen[s0])
            continue;
        const int s = bfs_last(bfs_last(s0));
        size_t h = order.size();
        order.push_back(s);
        seen[s] = 1;
        while (h < order.size())
        {
            const int v = order[h++];
            nb.clear();
            for (int k = start[v]; k < start[v + 1]; ++k)
                if (!seen[adj[k]])
                {
                    seen[adj[k]] = 1;
                    nb.push_back(adj[k]);
                }
            std::sort(nb.begin(), nb.end(), [&](int a, int b) { return deg[a] != deg[b] ? deg[a] < deg[b] : a < b; });
            order.insert(order.end(), nb.begin(), nb.end());
        }
    }
    for (int p = 0; p < n; ++p)
        rank[order[n - 1 - p]] = p; // reversed
    int64_t bw = 0, bw_id = 0;
    for (int i = 0; i < n; ++i)
        for (int k = start[i]; k < start[i + 1]; ++k)
        {
            bw = std::max<int64_t>(bw, std::abs((int64_t)rank[i] - rank[adj[k]]));
            bw_id = std::max<int64_t>(bw_id, std::abs((int64_t)i - adj[k]));
        }
    // the lattice generators' own order (row by row along the longest side) is often as narrow:
    // keep whichever band is narrower
    if (bw_id <= bw)
    {
        for (int i = 0; i < n; ++i)
            rank[i] = i;
        bw = bw_id;
    }
    return bw;
}

// One thread per particle i: its stiffness block row (sliced ELL, BCs eliminated) into the
// permuted lower band, entries on or below the diagonal only; the full symmetric storage holds
// every lower entry exactly once.
template <int D>
__global__ void k_band_fill(int n, const int *__restrict__ rowptr, const int *__restrict__ iperm_sell,
                            const int64_t *__restrict__ slice_off, const int *__restrict__ col_sell,
                            const double *__restrict__ K, const int *__restrict__ rank, int64_t ldab,
                            double *__restrict__ AB)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int pos = iperm_sell[i], s = pos / kSlice, l = pos % kSlice;
    const int nc = rowptr[i + 1] - rowptr[i];
    const int64_t ri = (int64_t)D * rank[i];
    for (int k = 0; k < nc; ++k)
    {
        const int64_t b = slice_off[s] + k;
        const int j = col_sell[b * kSlice + l];
        const int64_t cj = (int64_t)D * rank[j];
        for (int r = 0; r < D; ++r)
            for (int c = 0; c < D; ++c)
            {
                const int64_t R = ri + r, C = cj + c;
                if (R >= C)
                    AB[(R - C) + C * ldab] = K[(b * D * D + r * D + c) * kSlice + l];
            }
    }
}

// ---- factorisation: one persistent launch
//
// Per 32-column block: the rows below are solved against the factored block (four rows per warp), and
// after a barrier the trailing window is updated with FP64 tensor instructions (the update is a product
// of two panels) while warp 0 of every CTA updates and factors the next diagonal block (repeating it
// costs less than another exchange); a second barrier ends the block.  Bound by the diagonal blocks'
// serial pivots, then by the latency of the window's entries and two grid barriers (2.5 us each).
// Factor and solve of the 50 x 58 hexagonal plate (5,800 unknowns, half-bandwidth 401) 46.0 -> 3.7 ms,
// 100 x 115 (23,000, 801) 330 -> 19.3 ms, against three launches per block and one warp per diagonal
// block.  One 16-CTA cluster, whose barrier takes 0.3 us, took 4.0 and 33.1 ms: its SMs hold too few
// window tiles in flight.
constexpr int kFactorThreads = 256;
constexpr int kFactorWarps = kFactorThreads / 32;

// All blocks of the cooperative launch: a counting barrier in global memory (bounded: false and
// *fail = -1 once a wait passed the limit).
__device__ __forceinline__ bool factor_barrier(unsigned *bar, unsigned &epoch, int *fail, int *s_stop,
                                               unsigned long long wait_ns)
{
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        atomicAdd(bar, 1u);
        const unsigned target = (epoch + 1u) * gridDim.x;
        const unsigned long long t0 = gtimer();
        while ((int)(ld_acquire(bar) - target) < 0)
            if (gtimer() - t0 > wait_ns)
            {
                atomicExch(fail, -1);
                *s_stop = 1;
                break;
            }
    }
    epoch++;
    __syncthreads();
    return *s_stop == 0;
}

// D += A B^T for 8 x 4 panels: lane l holds row l / 4, column l % 4 of each operand and the entries
// (l / 4, 2 (l % 4)) and the next one of D
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// The factor of a 32 x 32 block by one warp: lane i holds row i in v and gets the pivots in fours, after
// which its row moves down by four columns (straight-line code for all 32 would not fit the instruction
// caches, and every block runs it once).  Column j goes to L[j][.] (zero above the diagonal and behind
// row 31), the reciprocal of its diagonal to inv[j].  Returns 0, or 1 + the column of a pivot that is
// not positive.
constexpr int kLRow = 66; // doubles per column of L: 32 rows, 32 zeros, 2 to shift the banks
__device__ __forceinline__ int factor_block(double *v, double (*L)[kLRow], double *inv)
{
    const int lane = threadIdx.x & 31;
    int bad = 0;
    double d = __shfl_sync(0xffffffffu, v[0], 0);
#pragma unroll 1
    for (int j4 = 0; j4 < 32; j4 += 4)
    {
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const int j = j4 + u;
            if (bad == 0 && !(d > 0.0))
                bad = j + 1;
            const double is = rsqrt(d);
            v[u] *= is; // lane j: d / sqrt(d)
            // the next pivot is ready in its own lane before the column's other updates
            d = __shfl_sync(0xffffffffu, v[u + 1] - v[u] * v[u], (j + 1) & 31);
            L[j][lane] = lane >= j ? v[u] : 0.0;
            if (lane == j)
                inv[j] = is;
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 32; c += 2)
                if (c + 1 > u)
                {
                    const double2 w = *reinterpret_cast<const double2 *>(&L[j][j4 + c]);
                    if (c > u)
                        v[c] -= v[u] * w.x;
                    v[c + 1] -= v[u] * w.y;
                }
        }
#pragma unroll
        for (int c = 0; c < 32; ++c)
            v[c] = c < 28 ? v[c < 28 ? c + 4 : 31] : 0.0;
    }
    return bad;
}

__global__ void __launch_bounds__(kFactorThreads, 1) k_band_factor(double *AB, int64_t ldab, int64_t kd, int64_t n,
                                                                  int *fail, unsigned *bar,
                                                                  unsigned long long wait_ns)
{
    extern __shared__ __align__(16) unsigned char fsm[];
    double(*Lb)[32][kLRow] = reinterpret_cast<double(*)[32][kLRow]>(fsm); // this block's factor and the next one's
    double(*T)[33] = reinterpret_cast<double(*)[33]>(fsm + 2 * sizeof(double) * 32 * kLRow);
    __shared__ double inv[2][32];
    __shared__ int bad, s_stop;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gw = (int64_t)blockIdx.x * kFactorWarps + warp, nwarps = (int64_t)kFactorWarps * gridDim.x;
    const int r8 = lane >> 2, k4 = lane & 3;
    unsigned epoch = 0;
    if (threadIdx.x == 0)
        s_stop = bad = 0;
    for (int k = threadIdx.x; k < 2 * 32 * kLRow; k += blockDim.x)
        (&Lb[0][0][0])[k] = 0.0;
    __syncthreads();
    if (warp == 0) // the first block: lane i reads row i; a missing row or column is the identity's
    {
        const int jb = (int)min((int64_t)kBandNB, n);
        double v[33];
#pragma unroll
        for (int j = 0; j < 32; ++j)
            v[j] = (lane < jb && j <= lane && lane - j <= kd) ? AB[(lane - j) + j * ldab] : (j == lane && lane >= jb) ? 1.0 : 0.0;
        v[32] = 0.0;
        const int b = factor_block(v, Lb[0], inv[0]);
        if (lane == 0)
            bad = b;
    }
    __syncthreads();
    for (int64_t j0 = 0; j0 < n; j0 += kBandNB)
    {
        const int cur = (int)((j0 / kBandNB) & 1);
        const int jb = (int)min((int64_t)kBandNB, n - j0);
        const int64_t c0 = j0 + jb, end = band::below_end(n, kd, j0, jb), m2 = end - c0;
        if (bad)
        {
            if (blockIdx.x == 0 && threadIdx.x == 0)
                *fail = (int)(j0 + bad);
            return; // every CTA factored the same block
        }
        // the rows below against the factored block: four rows per warp, a lane per column
        const double(*L)[kLRow] = Lb[cur];
        for (int64_t q = gw; 4 * q < m2; q += nwarps)
        {
            const int64_t i0 = c0 + 4 * q;
            double *const col = AB + (j0 + lane) * ldab - (j0 + lane); // entry (i, j0 + lane) at col[i]
            double x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                x[u] = (i0 + u < end && lane < jb && i0 + u - (j0 + lane) <= kd) ? col[i0 + u] : 0.0;
#pragma unroll 4
            for (int j = 0; j < 32; ++j)
            {
                const double l = lane > j ? L[j][lane] : 0.0, ij = inv[cur][j];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    const double y = __shfl_sync(0xffffffffu, x[u], j) * ij;
                    x[u] = lane == j ? y : x[u] - y * l;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u < end && lane < jb && i0 + u - (j0 + lane) <= kd)
                    col[i0 + u] = x[u];
        }
        if (!factor_barrier(bar, epoch, fail, &s_stop, wait_ns))
            return;
        // the factor takes the block's place (every CTA has long read it)
        if (blockIdx.x == gridDim.x - 1 && warp == kFactorWarps - 1 && lane < jb)
            for (int j = 0; j <= lane; ++j)
                if (lane - j <= kd)
                    AB[(lane - j) + (j0 + j) * ldab] = L[j][lane];
        if (m2 <= 0)
            break; // the last block
        if (warp == 0)
        {
            // the next diagonal block: this block's update of it, then its factor, in every CTA
            const int nb = (int)min((int64_t)kBandNB, n - c0);
            double d[4][4][2];
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y)
                    d[x][y][0] = d[x][y][1] = 0.0;
            double v[33];
#pragma unroll
            for (int j = 0; j < 32; ++j)
                v[j] = (lane < nb && j <= lane && lane - j <= kd) ? AB[(lane - j) + (c0 + j) * ldab]
                       : (j == lane && lane >= nb)                ? 1.0
                                                                  : 0.0;
            v[32] = 0.0;
#pragma unroll
            for (int k = 0; k < kBandNB; k += 4)
            {
                const int64_t j = j0 + k + k4;
                const double *col = AB + j * ldab - j;
                double a[4];
#pragma unroll
                for (int x = 0; x < 4; ++x)
                {
                    const int64_t i = c0 + 8 * x + r8;
                    a[x] = (i < end && i - j <= kd) ? col[i] : 0.0;
                }
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y <= x; ++y)
                        dmma(d[x][y][0], d[x][y][1], a[x], a[y]);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y <= x; ++y)
                {
                    T[8 * x + r8][8 * y + 2 * k4] = d[x][y][0];
                    T[8 * x + r8][8 * y + 2 * k4 + 1] = d[x][y][1];
                }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (j <= lane)
                    v[j] -= T[lane][j];
            __syncwarp();
            const int b = factor_block(v, Lb[cur ^ 1], inv[cur ^ 1]);
            if (lane == 0)
                bad = b;
        }
        else
        {
            // trailing window below the next diagonal block, in tiles of 32 x 16, a warp each:
            // A(i, c) -= sum_k L(i, k) L(c, k)
            const int64_t tr = (m2 + 31) / 32, tc = (m2 + 15) / 16;
            const int64_t first = (int64_t)(warp - 1) * gridDim.x + blockIdx.x, step = (int64_t)(kFactorWarps - 1) * gridDim.x;
            for (int64_t t = first; t < (tr - 1) * tc; t += step)
            {
                const int64_t ti = 1 + t / tc, tj = t % tc, i0 = c0 + ti * 32, cc = c0 + tj * 16;
                if (cc > i0 + 31 || i0 - (cc + 15) > kd)
                    continue; // above the diagonal, or outside the band
                double d[4][2][2], w[4][2][2]; // the product; the window's entries, on their way meanwhile
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 2; ++y)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                        {
                            const int64_t i = i0 + 8 * x + r8, c = cc + 8 * y + 2 * k4 + e;
                            d[x][y][e] = 0.0;
                            w[x][y][e] = (c <= i && i < end && i - c <= kd) ? AB[(i - c) + c * ldab] : 0.0;
                        }
#pragma unroll
                for (int k = 0; k < kBandNB; k += 4) // rows below exist: the block has all its columns
                {
                    const int64_t j = j0 + k + k4;
                    const double *col = AB + j * ldab - j; // entry (i, j) at col[i]
                    double a[4], b[2];
#pragma unroll
                    for (int x = 0; x < 4; ++x)
                    {
                        const int64_t i = i0 + 8 * x + r8;
                        a[x] = (i < end && i - j <= kd) ? col[i] : 0.0;
                    }
#pragma unroll
                    for (int y = 0; y < 2; ++y)
                    {
                        const int64_t i = cc + 8 * y + r8;
                        b[y] = (i < end && i - j <= kd) ? col[i] : 0.0;
                    }
#pragma unroll
                    for (int x = 0; x < 4; ++x)
#pragma unroll
                        for (int y = 0; y < 2; ++y)
                            dmma(d[x][y][0], d[x][y][1], a[x], b[y]);
                }
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 2; ++y)
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                        {
                            const int64_t i = i0 + 8 * x + r8, c = cc + 8 * y + 2 * k4 + e;
                            if (c <= i && i < end && i - c <= kd)
                                AB[(i - c) + c * ldab] = w[x][y][e] - d[x][y][e];
                        }
            }
        }
        if (!factor_barrier(bar, epoch, fail, &s_stop, wait_ns))
            return;
    }
}

constexpr int kFactorSmem = 2 * 8 * 32 * kLRow + 8 * 32 * 33;

// ---- substitution: one CTA
//
// Forward, block by block: one warp solves the block's triangle (lane i holds y_i), then the rows
// below take their 32 products.  Backward: a warp per column of the block
// gathers the finished x below it, then one warp solves the transposed triangle.  Bound by the chain
// of 32 pivots per block, so more CTAs would only add barriers.  Both sweeps over 5,800 unknowns at
// half-bandwidth 401: 1.15 ms (2.74 ms without the panels; 25 ms with four launches per block).
constexpr int kSolveThreads = 1024;
constexpr int kSolvePanelBytes = 104 * 1024; // one panel; two are in shared memory
static_assert(2 * kSolvePanelBytes + 12 * 1024 <= 232448, "shared memory of the substitution");

// `panel` holds a block's 32 whole band columns (one contiguous piece of the band) when they fit,
// copied there ahead of their use; wider bands are read from global memory.
template <bool PANEL>
__global__ void __launch_bounds__(kSolveThreads, 1) k_band_solve(const double *AB, int64_t ldab, int64_t kd, int64_t n,
                                                                double *y, int *fail, unsigned long long wait_ns)
{
    extern __shared__ __align__(128) unsigned char dsm[];
    __shared__ double M[32][33]; // M[j][i]: column j, row i of the block, over the diagonal entry j
    __shared__ double inv[32], s[32];
    __shared__ int lost; // a copy did not arrive in time
    __shared__ uint64_t bar[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nblk = (n + kBandNB - 1) / kBandNB;
    if (threadIdx.x == 0)
    {
        lost = 0;
        for (int k = 0; k < 2; ++k)
            mbar_init(&bar[k], 1);
        mbar_init_fence();
    }
    __syncthreads();
    // the copies run through blocks 0 .. nblk - 1, then back to 0; copy q goes to buffer q % 2
    auto block_of = [&](int64_t q) { return q < nblk ? q : 2 * nblk - 1 - q; };
    auto fetch = [&](int64_t q) {
        if (!PANEL || threadIdx.x != 0 || q >= 2 * nblk)
            return;
        const int64_t j0 = block_of(q) * kBandNB, jb = min((int64_t)kBandNB, n - j0);
        // whole 16-byte pieces; the allocation has one spare entry behind an odd last column
        const unsigned bytes = (unsigned)((jb * ldab * 8 + 15) / 16 * 16);
        bulk_refill(dsm + (q & 1) * kSolvePanelBytes, AB + j0 * ldab, bytes, &bar[q & 1]);
    };
    // column j of block q, entry (i, j) at [i - j]
    auto column = [&](int64_t q, int64_t j0, int j) -> const double * {
        return PANEL ? reinterpret_cast<const double *>(dsm + (q & 1) * kSolvePanelBytes) + j * ldab
                     : AB + (j0 + j) * ldab;
    };
    auto arrive = [&](int64_t q) {
        if (!PANEL)
            return;
        const uint32_t parity = (uint32_t)((q >> 1) & 1);
        // a try may sleep past a limit below 100 us, which cluster_wait minds
        if (!(wait_ns >= 100000ull ? mbar_wait_bounded(&bar[q & 1], parity, wait_ns)
                                   : cluster_wait(smem_u32(&bar[q & 1]), parity, wait_ns)))
            lost = 1;
    };
    // After the block synchronisation that follows arrive(q): a copy that did not come in time ends the
    // kernel, and the host learns of it.  The copies in flight, q and q + 1, land before the block's shared
    // memory is given back.
    auto given_up = [&](int64_t q) {
        if (!PANEL || !lost)
            return false;
        if (threadIdx.x == 0)
        {
            for (int64_t w = q; w < min(q + 2, 2 * nblk); ++w)
                cluster_wait(smem_u32(&bar[w & 1]), (unsigned)((w >> 1) & 1), kBarrierTimeoutNs);
            *fail = -1;
        }
        return true;
    };
    auto stage = [&](int64_t q, int64_t j0, int jb, bool transposed) { // warp w: column w
        const double v = (warp < jb && lane < jb && lane >= warp && lane - warp <= kd) ? column(q, j0, warp)[lane - warp]
                                                                                        : (lane == warp ? 1.0 : 0.0);
        const double dj = 1.0 / __shfl_sync(0xffffffffu, v, warp);
        if (lane == warp)
            inv[warp] = dj;
        // forward: column j over its diagonal; backward: row i of L^T over the diagonal of i, which
        // column j's thread i learns from the other warps' diagonals
        if (!transposed)
            M[warp][lane] = v * dj;
        else
            M[lane][warp] = v;
    };
    fetch(0);
    fetch(1);
    for (int64_t q = 0; q < nblk; ++q)
    {
        const int64_t j0 = q * kBandNB;
        const int jb = (int)min((int64_t)kBandNB, n - j0);
        const int64_t c0 = j0 + jb, end = band::below_end(n, kd, j0, jb);
        arrive(q);
        stage(q, j0, jb, false);
        __syncthreads();
        if (given_up(q))
            return;
        if (warp == 0)
        {
            double v = lane < jb ? y[j0 + lane] : 0.0;
#pragma unroll
            for (int j = 0; j < 32; ++j)
            {
                const double x = __shfl_sync(0xffffffffu, v, j);
                v -= lane > j ? M[j][lane] * x : 0.0;
            }
            v *= inv[lane];
            s[lane] = v;
            if (lane < jb)
                y[j0 + lane] = v;
        }
        __syncthreads();
        for (int64_t i = c0 + threadIdx.x; i < end; i += blockDim.x)
        {
            double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
            for (int j = 0; j < jb; ++j)
                if (i - (j0 + j) <= kd)
                    t[j & 3] += column(q, j0, j)[i - j0 - j] * s[j];
            y[i] -= (t[0] + t[1]) + (t[2] + t[3]);
        }
        __syncthreads();
        fetch(q + 2);
    }
    for (int64_t q = nblk; q < 2 * nblk; ++q)
    {
        const int64_t j0 = block_of(q) * kBandNB;
        const int jb = (int)min((int64_t)kBandNB, n - j0);
        const int64_t c0 = j0 + jb, end = band::below_end(n, kd, j0, jb);
        arrive(q);
        stage(q, j0, jb, true);
        if (warp < jb)
        {
            const int64_t j = j0 + warp;
            const double *col = column(q, j0, warp) - j; // entry (i, j) at col[i]
            const int64_t last = min(end, j + kd + 1);
            double t0 = 0.0, t1 = 0.0;
            int64_t i = c0 + lane;
            for (; i + 32 < last; i += 64)
            {
                t0 += col[i] * y[i];
                t1 += col[i + 32] * y[i + 32];
            }
            if (i < last)
                t0 += col[i] * y[i];
            t0 = wsum(t0 + t1);
            if (lane == 0)
                s[warp] = y[j] - t0;
        }
        __syncthreads();
        if (given_up(q))
            return;
        if (warp == 0)
        {
            // M[j][i] = L(j, i): x_i = (s_i - sum_{j > i} L(j, i) x_j) / L(i, i)
            double v = lane < jb ? s[lane] : 0.0;
            const double di = inv[lane];
            v *= di;
#pragma unroll
            for (int j = 31; j >= 0; --j)
            {
                const double x = __shfl_sync(0xffffffffu, v, j);
                v -= lane < j ? M[j][lane] * di * x : 0.0;
            }
            if (lane < jb)
                y[j0 + lane] = v;
        }
        __syncthreads();
        fetch(q + 2);
    }
}

// y[d*rank(i)+r] = src[d*i+r]  /  dst[d*i+r] = y[d*rank(i)+r]
__global__ void k_band_perm(int n, int dim, const int *__restrict__ rank, const double *__restrict__ src,
                            double *__restrict__ dst, int inverse)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (int64_t)n * dim)
        return;
    const int i = (int)(q / dim), r = (int)(q % dim);
    const int64_t pq = (int64_t)dim * rank[i] + r;
    if (inverse)
        dst[q] = src[pq];
    else
        dst[pq] = src[q];
}

// The ordering, the band's size and its storage; once per problem.
static int32_t direct_setup(Problem &p)
{
    if (p.band_ab)
        return LPMGPU_OK;
    const int n = p.n;
    std::vector<int> start((size_t)n + 1), adj((size_t)p.nnzb), rank(n);
    cudaError_t e = cudaMemcpyAsync(start.data(), p.cstart, sizeof(int) * ((size_t)n + 1), cudaMemcpyDeviceToHost,
                                    p.stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(adj.data(), p.conns, sizeof(int) * (size_t)p.nnzb, cudaMemcpyDeviceToHost, p.stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(p.stream);
    if (e != cudaSuccess)
    {
        set_last_error(std::string("direct solver set-up: ") + cudaGetErrorString(e));
        return LPMGPU_ERR_CUDA;
    }
    const int64_t bw = rcm_order(n, start.data(), adj.data(), rank.data());
    const int64_t ndof = (int64_t)n * p.dim;
    const int64_t kd = std::min<int64_t>((int64_t)p.dim * bw + p.dim - 1, ndof - 1);
    const int64_t ldab = kd + 1;
    if (ldab * ndof * (int64_t)sizeof(double) > kBandMaxBytes)
    {
        set_last_error("direct solver: the band (" + std::to_string(ndof) + " unknowns, half-bandwidth " +
                       std::to_string(kd) + ") is larger than the 32 GiB the solver allows; use the CG");
        return LPMGPU_ERR_OUT_OF_MEMORY;
    }
    if ((e = dalloc(p, &p.band_rank, (size_t)n)) != cudaSuccess ||
        (e = dalloc(p, &p.band_y, (size_t)ndof)) != cudaSuccess ||
        (e = dalloc(p, &p.band_fail, 1)) != cudaSuccess ||
        (e = dalloc(p, &p.band_ab, (size_t)(ldab * ndof) + 1)) != cudaSuccess) // + 1: whole 16-byte copies
    {
        (void)cudaGetLastError(); // a failed allocation is reported here, not by a later launch check
        p.band_ab = nullptr;
        set_last_error(std::string("direct solver: ") + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? LPMGPU_ERR_OUT_OF_MEMORY : LPMGPU_ERR_CUDA;
    }
    if ((e = cudaMemcpyAsync(p.band_rank, rank.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, p.stream)) !=
            cudaSuccess ||
        (e = cudaStreamSynchronize(p.stream)) != cudaSuccess)
        return LPMGPU_ERR_CUDA;
    p.band_kd = kd;
    p.band_factored = -1;
    return LPMGPU_OK;
}

// Band fill + blocked factorisation of the current K.
template <int D>
static cudaError_t factor(Problem &p)
{
    const int64_t ndof = (int64_t)p.n * D, kd = p.band_kd, ldab = kd + 1;
    cudaError_t e = cudaMemsetAsync(p.band_ab, 0, sizeof(double) * (size_t)(ldab * ndof), p.stream);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(p.band_fail, 0, sizeof(int), p.stream);
    if (e != cudaSuccess)
        return e;
    k_band_fill<D><<<div_up(p.n, 128), 128, 0, p.stream>>>(p.n, p.cstart, p.iperm, p.slice_off, p.col_sell, p.K,
                                                          p.band_rank, ldab, p.band_ab);
    p.ctr.kernel_launches++;
    if ((e = cudaGetLastError()) != cudaSuccess)
        return e;
    if ((e = cudaMemsetAsync(p.barrier, 0, 2 * sizeof(unsigned), p.stream)) != cudaSuccess)
        return e;
    double *ab = p.band_ab;
    int64_t ld = ldab, k = kd, nn = ndof;
    int *fail = p.band_fail;
    unsigned *bar = p.barrier;
    unsigned long long wait_ns = p.wait_ns;
    void *args[] = {&ab, &ld, &k, &nn, &fail, &bar, &wait_ns};
    e = cudaLaunchCooperativeKernel((const void *)k_band_factor, dim3(p.num_sms), dim3(kFactorThreads), args,
                                    kFactorSmem, p.stream);
    p.ctr.kernel_launches++;
    return e;
}

// Forward and backward substitution of p.res into p.x.
template <int D>
static cudaError_t substitute(Problem &p)
{
    const int64_t ndof = (int64_t)p.n * D, kd = p.band_kd, ldab = kd + 1;
    const int nb = (int)div_up(ndof, 256);
    k_band_perm<<<nb, 256, 0, p.stream>>>(p.n, D, p.band_rank, p.res, p.band_y, 0);
    p.ctr.kernel_launches++;
    if (kBandNB * ldab * 8 <= kSolvePanelBytes)
    {
        const cudaError_t e = cudaFuncSetAttribute(k_band_solve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   2 * kSolvePanelBytes);
        if (e != cudaSuccess)
            return e;
        k_band_solve<true><<<1, kSolveThreads, 2 * kSolvePanelBytes, p.stream>>>(p.band_ab, ldab, kd, ndof, p.band_y,
                                                                              p.band_fail, p.wait_ns);
    }
    else
        k_band_solve<false><<<1, kSolveThreads, 0, p.stream>>>(p.band_ab, ldab, kd, ndof, p.band_y, p.band_fail,
                                                               p.wait_ns);
    p.ctr.kernel_launches++;
    k_band_perm<<<nb, 256, 0, p.stream>>>(p.n, D, p.band_rank, p.band_y, p.x, 1);
    p.ctr.kernel_launches++;
    return cudaGetLastError();
}

// K x = res into p.x by the band Cholesky; the factor is reused while K is unchanged.
int32_t solve_direct(Problem &p)
{
    int32_t s = direct_setup(p);
    if (s != LPMGPU_OK)
        return s;
    cudaError_t e = cudaSuccess;
    if (p.band_factored != p.k_version)
    {
        e = p.dim == 2 ? factor<2>(p) : factor<3>(p);
        int fail = 0;
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&fail, p.band_fail, sizeof(int), cudaMemcpyDeviceToHost, p.stream);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(p.stream);
        if (e != cudaSuccess)
        {
            set_last_error(std::string("direct solver: ") + cudaGetErrorString(e));
            return LPMGPU_ERR_CUDA;
        }
        if (fail < 0)
        {
            p.band_factored = -1;
            set_last_error("direct solver: a device-side barrier wait timed out");
            return LPMGPU_ERR_TIMEOUT;
        }
        if (fail)
        {
            p.band_factored = -1;
            set_last_error("direct solver: the stiffness is not positive definite (pivot " + std::to_string(fail) +
                           " of the reordered system)");
            return LPMGPU_ERR_NOT_SPD;
        }
        p.band_factored = p.k_version;
    }
    e = p.dim == 2 ? substitute<2>(p) : substitute<3>(p);
    int *fail = reinterpret_cast<int *>(p.cg_info_host + 6);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(fail, p.band_fail, sizeof(int), cudaMemcpyDeviceToHost, p.stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(p.stream);
    if (e != cudaSuccess)
    {
        set_last_error(std::string("direct solver: ") + cudaGetErrorString(e));
        return LPMGPU_ERR_CUDA;
    }
    if (*fail)
    {
        p.band_factored = -1; // the next call starts from the band
        set_last_error("direct solver: a device-side copy wait of the substitution timed out");
        return LPMGPU_ERR_TIMEOUT;
    }
    return LPMGPU_OK;
}

} // namespace lpm

extern "C" int32_t lpmgpu_band_order(int32_t n, const int32_t *start, const int32_t *adj, int32_t *rank,
                                     int64_t *bandwidth)
{
    if (n <= 0 || !start || !adj || !rank || !bandwidth || start[0] != 0)
        return LPMGPU_ERR_INVALID_ARG;
    for (int i = 0; i < n; ++i)
        if (start[i + 1] < start[i])
            return LPMGPU_ERR_INVALID_ARG;
    for (int k = 0; k < start[n]; ++k)
        if (adj[k] < 0 || adj[k] >= n)
            return LPMGPU_ERR_INVALID_ARG;
    *bandwidth = lpm::rcm_order(n, start, adj, rank);
    return LPMGPU_OK;
}
