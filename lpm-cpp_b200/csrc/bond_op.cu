// The bond form of the stiffness product (bond_op.cuh): its layout, its refresh at every assembly
// and the CG on it, which replaces Solver::LPM_CG (include/solver.h:277-354) as k_cg of cg.cu does:
// unpreconditioned, x0 = 0, stop when ||r||^2 <= rtol*||r0||^2 + atol, cap = problem size.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "bond_op.cuh"
#include "cluster.cuh"

namespace lpm
{

// ---------------------------------------------------------------------------- layout
// Columns and source bonds of every entry, and the lowest and highest row that each group touches;
// *bad is set for a bond list the form cannot take (a partner that appears twice in one particle's
// lists, or opposite bonds that are not a pairing).
__global__ void k_bo_fill(int n, int ng, int ls, int width, const int *__restrict__ bstart,
                          const int *__restrict__ nb0, const int *__restrict__ bp2, const int *__restrict__ brev,
                          int *__restrict__ col, int *__restrict__ src, int *__restrict__ reach, int *__restrict__ bad)
{
    const int lane = threadIdx.x & 31;
    const int g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (g >= ng)
        return;
    const int S = 1 << ls, i = g * (32 >> ls) + (lane >> ls), q = lane & (S - 1);
    const int b0 = i < n ? bstart[i] : 0, nb = i < n ? bstart[i + 1] - b0 : 0, n0 = i < n ? nb0[i] : 0;
    int lo = min(i, n - 1), hi = lo;
    for (int t = 0; t < width; ++t)
    {
        const int o = t * S + q;
        const int64_t e = ((int64_t)g * width + t) * 32 + lane;
        const bool have = o < nb;
        const int j = have ? bp2[b0 + o] : min(i, n - 1);
        col[e] = 2 * j + ((have && o >= n0) ? 1 : 0);
        src[e] = have ? b0 + o : -1;
        lo = min(lo, j);
        hi = max(hi, j);
        if (have)
        {
            bool odd = brev[brev[b0 + o]] != b0 + o;
            for (int k = 0; k < o; ++k)
                odd |= bp2[b0 + k] == j;
            if (odd)
                atomicExch(bad, 1);
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0)
    {
        reach[2 * g] = lo;
        reach[2 * g + 1] = hi;
    }
}

// ---------------------------------------------------------------------------- refresh
// One thread per entry: the cosines (and T, T - F) of the current state, and the flags of the
// bonds: coefficients that are not the layer's constants, or that differ between the directions.
template <int D, bool GEN>
__global__ void __launch_bounds__(256) k_bo_pack(int64_t entries, const int *__restrict__ src,
                                                 const int *__restrict__ brev, const double *__restrict__ cs,
                                                 const double *__restrict__ Kn, const double *__restrict__ Tv,
                                                 const double *__restrict__ bdamage, double *__restrict__ c,
                                                 float *__restrict__ c32, double *__restrict__ tm,
                                                 float *__restrict__ tm32, int *flag)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= entries)
        return;
    const int64_t t = e >> 5;
    const int lane = (int)(e & 31);
    const int b = src[e];
    double v[D], T = 0.0, M = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k)
        v[k] = b >= 0 ? cs[3 * (int64_t)b + k] : 0.0;
    int f = 0;
    if (b >= 0)
    {
        const int rb = brev[b];
        const double Da = bdamage[b], Dr = bdamage[rb];
        const bool broken = fabs(Da - 1.0) < kEps;
        if (broken != (fabs(Dr - 1.0) < kEps))
            f |= kBondUnsupported;
        if constexpr (GEN)
        {
            T = (1 - Da) * Tv[b];
            M = T - (1 - Da) * (2 * Kn[b] + Tv[b]);
            if (!(Da == Dr) || Kn[b] != Kn[rb] || Tv[b] != Tv[rb])
                f |= kBondUnsupported;
        }
        else if (!broken && !(Da == 0.0 && Dr == 0.0))
            f |= kBondGeneral;
    }
#pragma unroll
    for (int k = 0; k < D; ++k)
    {
        c[(t * D + k) * 32 + lane] = v[k];
        if (c32)
            c32[(t * D + k) * 32 + lane] = (float)v[k];
    }
    if constexpr (GEN)
    {
        tm[(2 * t) * 32 + lane] = T;
        tm[(2 * t + 1) * 32 + lane] = M;
        if (tm32)
        {
            tm32[(2 * t) * 32 + lane] = (float)T;
            tm32[(2 * t + 1) * 32 + lane] = (float)M;
        }
    }
    if (f)
        atomicOr(flag, f);
}

// One thread per particle: the constraint mask of this assembly, and with GEN the particle's S, U
// and self block (fdu2dxyz, derivative.h:8-45).  A particle whose bonds are all broken is
// constrained by the assembly whatever its residual: such a K keeps the assembled form.
template <int D, bool GEN>
__global__ void __launch_bounds__(128) k_bo_rows(int n, int apply_bc, const int *__restrict__ bstart,
                                                 const int *__restrict__ nb0, const int *__restrict__ cons,
                                                 const double *__restrict__ damage_visual,
                                                 const double *__restrict__ cs, const double *__restrict__ Kn,
                                                 const double *__restrict__ Tv, const double *__restrict__ bdamage,
                                                 const double *__restrict__ cs_sum, unsigned char *__restrict__ mask,
                                                 double *__restrict__ row, float *__restrict__ row32, int *flag)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    int m = 0;
    if (apply_bc)
    {
        for (int k = 0; k < D; ++k)
            m |= (cons[3 * i + k] == 1) << k;
        if (fabs(damage_visual[i] - 1.0) < kEps)
            atomicOr(flag, kBondUnsupported);
    }
    mask[i] = (unsigned char)m;
    if constexpr (GEN)
    {
        constexpr int RS = 4 * D + D * (D + 1) / 2;
        double v[RS];
#pragma unroll
        for (int k = 0; k < RS; ++k)
            v[k] = 0.0;
#pragma unroll
        for (int L = 0; L < 2; ++L)
        {
            const int lo = L == 0 ? bstart[i] : bstart[i] + nb0[i], hi = L == 0 ? bstart[i] + nb0[i] : bstart[i + 1];
#pragma unroll
            for (int k = 0; k < D; ++k)
                v[L * D + k] = cs_sum[6 * (int64_t)i + 3 * L + k];
            for (int b = lo; b < hi; ++b)
            {
                double c[D];
#pragma unroll
                for (int k = 0; k < D; ++k)
                    c[k] = cs[3 * (int64_t)b + k];
                const double T = (1 - bdamage[b]) * Tv[b], F = (1 - bdamage[b]) * (2 * Kn[b] + Tv[b]);
                int e = 4 * D;
#pragma unroll
                for (int r = 0; r < D; ++r)
                {
                    v[(2 + L) * D + r] += T * c[r];
#pragma unroll
                    for (int q = 0; q < D; ++q)
                        if (r <= q)
                            v[e++] += F * c[r] * c[q] + T * c[r] * v[L * D + q];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < RS; ++k)
        {
            row[(int64_t)k * n + i] = v[k];
            if (row32)
                row32[(int64_t)k * n + i] = (float)v[k];
        }
    }
}

// ---------------------------------------------------------------------------- vectors of the CG
// r and p are gathered: in 2D one pair per particle; in 3D the pairs (x, y) of all particles, then
// their z (a warp's gather of 32 neighbouring rows then touches each 128-byte line once).
template <typename TV, int D>
__device__ __forceinline__ void ld_vec(const TV *v, int n, int j, TV *out, uint64_t pl)
{
    const auto a = ld_keep2(v + 2 * (int64_t)j, pl);
    out[0] = a.x;
    out[1] = a.y;
    if constexpr (D == 3)
        out[2] = ld_keep(v + 2 * (int64_t)n + j, pl);
}
__device__ __forceinline__ void st_keep2(double *a, double2 v, uint64_t pol)
{
    asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;" ::"l"(a), "d"(v.x), "d"(v.y), "l"(pol)
                 : "memory");
}
template <typename TV, int D>
__device__ __forceinline__ void st_vec(TV *v, int n, int j, const TV *in, uint64_t pl)
{
    if constexpr (sizeof(TV) == 8)
        st_keep2(v + 2 * (int64_t)j, make_double2(in[0], in[1]), pl);
    else
        st_keep2(v + 2 * (int64_t)j, make_float2(in[0], in[1]), pl);
    if constexpr (D == 3)
        st_keep(v + 2 * (int64_t)n + j, in[2], pl);
}

// the sum of v over the lanes that share a row
template <typename TV>
__device__ __forceinline__ TV row_sum(TV v, int ls)
{
    for (int o = 1; o < (1 << ls); o <<= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Per-particle values of the general form: S, U per layer and the upper triangle of the self block.
template <typename TV, int D>
struct RowTerms
{
    static constexpr int N = 4 * D + D * (D + 1) / 2;
    TV v[N];
    __device__ __forceinline__ void load(const TV *row, int n, int i)
    {
#pragma unroll
        for (int k = 0; k < N; ++k)
            v[k] = row[(int64_t)k * n + i];
    }
    __device__ __forceinline__ TV dot(int at, const TV *x) const
    {
        TV t = v[at] * x[0];
#pragma unroll
        for (int k = 1; k < D; ++k)
            t += v[at + k] * x[k];
        return t;
    }
    __device__ __forceinline__ void self(const TV *x, TV *y) const
    {
#pragma unroll
        for (int r = 0; r < D; ++r)
        {
            TV t = TV(0);
#pragma unroll
            for (int q = 0; q < D; ++q)
            {
                const int a = r < q ? r : q, b = r < q ? q : r;
                t += v[4 * D + a * D - a * (a - 1) / 2 + (b - a)] * x[q];
            }
            y[r] = t;
        }
    }
};

// what a lane gathers from its bonds in the first pass; Z (uniform form): also the part of K x that needs
// no theta
template <typename TV, int D, bool GEN, bool Z = false>
struct Pass1
{
    TV th0 = TV(0), th1 = TV(0); // theta (GEN: G) per layer
    TV h0 = TV(0), h1 = TV(0);   // GEN: H per layer
    double en = 0.0;             // x . K x's bond terms
    TV z[D];                     // Z: sum of 2 Kn c d
    __device__ __forceinline__ Pass1()
    {
#pragma unroll
        for (int k = 0; k < D; ++k)
            z[k] = TV(0);
    }
    __device__ __forceinline__ void bond(const TV *xi, const TV *xj, const TV *c, int L, const TV *Kn, TV T, TV M)
    {
        if constexpr (!GEN)
        {
            TV d = c[0] * (xi[0] - xj[0]);
#pragma unroll
            for (int k = 1; k < D; ++k)
                d += c[k] * (xi[k] - xj[k]);
            th0 += L ? TV(0) : d;
            th1 += L ? d : TV(0);
            en += (double)(L ? Kn[1] : Kn[0]) * ((double)d * (double)d);
            if constexpr (Z)
            {
                const TV kd = 2 * (L ? Kn[1] : Kn[0]) * d;
#pragma unroll
                for (int k = 0; k < D; ++k)
                    z[k] += c[k] * kd;
            }
        }
        else
        {
            TV ci = c[0] * xi[0], cj = c[0] * xj[0];
#pragma unroll
            for (int k = 1; k < D; ++k)
            {
                ci += c[k] * xi[k];
                cj += c[k] * xj[k];
            }
            const TV h = 2 * T * cj;
            th0 += L ? TV(0) : cj;
            th1 += L ? cj : TV(0);
            h0 += L ? TV(0) : h;
            h1 += L ? h : TV(0);
            en += (double)(M * cj - T * ci) * (double)ci;
        }
    }
};

// The row's share of x . K x that needs its whole sums; GEN: alpha, beta per layer into ab.
template <typename TV, int D>
__device__ __forceinline__ double general_row(const RowTerms<TV, D> &rt, const TV *xi, TV G0, TV G1, TV H0, TV H1, TV *ab)
{
    TV y[D];
    rt.self(xi, y);
    double e = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k)
        e += (double)y[k] * (double)xi[k];
#pragma unroll
    for (int L = 0; L < 2; ++L)
    {
        const TV G = L ? G1 : G0, H = L ? H1 : H0;
        const TV sx = rt.dot(L * D, xi), ux = rt.dot((2 + L) * D, xi);
        ab[2 * L] = TV(0.75) * sx - TV(0.5) * G;
        ab[2 * L + 1] = TV(0.25) * (ux - H);
        e += -0.75 * (double)sx * (double)H - 0.5 * (double)ux * (double)G + 0.5 * (double)G * (double)H;
    }
    return e;
}

// the row's result from its own sums (second pass of the general form)
template <typename TV, int D>
__device__ __forceinline__ void general_close(const RowTerms<TV, D> &rt, const TV *xi, TV G0, TV G1, TV H0, TV H1, TV *y)
{
    TV sy[D];
    rt.self(xi, sy);
#pragma unroll
    for (int k = 0; k < D; ++k)
        y[k] += sy[k] - (TV(0.375) * (rt.v[k] * H0 + rt.v[D + k] * H1) +
                         TV(0.25) * (rt.v[2 * D + k] * G0 + rt.v[3 * D + k] * G1));
}

// The CG on the whole grid, one block per SM, each owning a contiguous share of the groups.  pq is known
// after pass 1, so x and r are updated in pass 2 and there is no vector pass.
//
// Large problems: bound by the bond stream (28 bytes per bond and pass in FP64 3D, twice per iteration,
// from L2 while it fits there) and its gathers, plus two grid sums of 2.0 us.  One bond in flight per lane
// at 1024 threads: the 64 registers hold no more without spills (two bonds spilled: 70 us per iteration on
// the cube below; 512 threads with two bonds: 25.1 us against 23.1 then).  51x50x50 simple cubic FP64,
// assembled matrix (584 MB at 93% of HBM) -> bonds (64 MB): 98.2 -> 20.2 us.
//
// ST (uniform coefficients, at most one group per warp, whose bonds fit kStagedSmem): the columns and
// cosines are copied to shared memory once, since each grid sum empties L1, so a gather no longer waits on
// a column from L2 and the registers hold three bonds' gathers per lane.  Without -> with ST, us per
// iteration: hexagonal 18,000 rows 7.76 -> 6.99, 40,000 9.07 -> 8.78, square 21,000 7.19 -> 6.80, simple
// cubic 8,000 9.06 -> 8.23, 27,000 11.2 -> 9.68, FCC 7,488 9.08 -> 8.17, BCC 16,000 9.01 -> 8.75.  At 1024
// threads with 1 / 2 / 3 bonds in flight (the latter two spill) hexagonal 18,000 takes 7.38 / 8.25 / 10.2;
// at 512 with 5, 7.37 and simple cubic 27,000 13.7.  Its registers also keep z, the part of K p without
// theta, from pass 1, so pass 2 gathers theta alone: hexagonal 18,000 6.99 -> 6.78, 40,000 8.78 -> 8.61,
// simple cubic 8,000 8.23 -> 7.72, 27,000 9.68 -> 8.84, FCC 7,488 8.17 -> 7.68.  The general form has no
// registers for z: it spills, and the cube above goes from 21.2 to 25.9.
constexpr int kBondThreads = 1024, kStagedThreads = 512;
constexpr size_t kStagedSmem = 128 * 1024;

template <typename TV, int D, bool GEN, bool ST>
__global__ void __launch_bounds__(ST ? kStagedThreads : kBondThreads, 1) k_cg_bond(BondCG<TV> s)
{
    extern __shared__ __align__(16) unsigned char bond_sm[];
    __shared__ double sh[32];
    __shared__ int s_fail;
    if (*s.flag & s.flag_bad)
    {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), (unsigned long long)kBondDeclined);
        return;
    }
    if (threadIdx.x == 0)
        s_fail = 0;
    __syncthreads();
    constexpr int U = ST ? 3 : 1; // bonds in flight per lane
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n = s.n, ls = s.ls, q = lane & ((1 << ls) - 1), rl = lane >> ls, R = 32 >> ls;
    const int g0 = (int)((int64_t)blockIdx.x * s.ng / gridDim.x), g1 = (int)((int64_t)(blockIdx.x + 1) * s.ng / gridDim.x);
    const uint64_t pl = l2_evict_last(), pb_ = s.keep ? l2_evict_last() : l2_evict_first();
    unsigned epoch = 0;
    // ST: the bonds of the warp's one group
    TV *cS = reinterpret_cast<TV *>(bond_sm) + (size_t)warp * s.width * D * 32 + lane;
    int *colS = reinterpret_cast<int *>(reinterpret_cast<TV *>(bond_sm) + (size_t)(g1 - g0) * s.width * D * 32) +
                warp * s.width * 32 + lane;
    if (ST && g0 + warp < g1)
        for (int t = 0; t < s.width; ++t)
        {
            const int64_t at = (int64_t)(g0 + warp) * s.width + t;
            colS[t * 32] = s.col[at * 32 + lane];
#pragma unroll
            for (int k = 0; k < D; ++k)
                cS[(t * D + k) * 32] = s.c[(at * D + k) * 32 + lane];
        }
    const int ts = (g0 + warp) * s.width; // ST: the group's first entry
    auto column = [&](int t) {
        if constexpr (ST)
            return colS[(t - ts) * 32];
        else
            return ld_stream(s.col + (int64_t)t * 32 + lane, pb_);
    };
    auto staged_cosines = [&](int t, TV *c) {
#pragma unroll
        for (int k = 0; k < D; ++k)
            c[k] = cS[((t - ts) * D + k) * 32];
    };

    double loc = 0;
    for (int g = g0 + warp; g < g1; g += nw)
    {
        const int i = g * R + rl;
        if (q == 0 && i < n)
        {
            TV bv[D], zero[D];
#pragma unroll
            for (int k = 0; k < D; ++k)
            {
                bv[k] = s.b[(int64_t)i * D + k];
                zero[k] = TV(0);
                s.x[(int64_t)i * D + k] = TV(0);
                loc += (double)bv[k] * (double)bv[k];
            }
            st_vec<TV, D>(s.r, n, i, bv, pl);
            st_vec<TV, D>(s.pa, n, i, zero, pl);
        }
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
    TV *pold = s.pa, *pnew = s.pb;
    for (int64_t it = 1;; ++it)
    {
        // pass 1: p = r + beta p_old on the fly; theta (GEN: alpha, beta) per particle; p . K p
        double lpq = 0;
        TV zS[D]; // ST: the warp's one group's share of z
        for (int g = g0 + warp; g < g1; g += nw)
        {
            const int i = g * R + rl, ii = min(i, n - 1);
            TV xi[D];
            {
                TV a[D], b[D];
                ld_vec<TV, D>(s.r, n, ii, a, pl);
                ld_vec<TV, D>(pold, n, ii, b, pl);
#pragma unroll
                for (int k = 0; k < D; ++k)
                    xi[k] = a[k] + beta * b[k];
            }
            Pass1<TV, D, GEN, ST> ps;
            const int t1 = (g + 1) * s.width;
            int t = g * s.width;
            int cn[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                cn[u] = (t + u < t1) ? column(t + u) : 0;
            for (; t < t1; t += U)
            {
                int co[U];
                TV rv[U][D], pv[U][D], cv[U][D], T[U], M[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    co[u] = cn[u];
                    cn[u] = (t + U + u < t1) ? column(t + U + u) : 0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (t + u < t1)
                    {
                        ld_vec<TV, D>(s.r, n, co[u] >> 1, rv[u], pl);
                        ld_vec<TV, D>(pold, n, co[u] >> 1, pv[u], pl);
                        if constexpr (!ST)
                        {
                            const TV *cb = s.c + ((int64_t)(t + u) * D) * 32 + lane;
#pragma unroll
                            for (int k = 0; k < D; ++k)
                                cv[u][k] = ld_stream(cb + k * 32, pb_);
                        }
                        if constexpr (GEN)
                        {
                            T[u] = ld_stream(s.tm + (int64_t)(2 * (t + u)) * 32 + lane, pb_);
                            M[u] = ld_stream(s.tm + (int64_t)(2 * (t + u) + 1) * 32 + lane, pb_);
                        }
                    }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (t + u < t1)
                    {
                        TV xj[D];
                        if constexpr (ST)
                            staged_cosines(t + u, cv[u]);
#pragma unroll
                        for (int k = 0; k < D; ++k)
                            xj[k] = rv[u][k] + beta * pv[u][k];
                        ps.bond(xi, xj, cv[u], co[u] & 1, s.Kn, GEN ? T[u] : TV(0), GEN ? M[u] : TV(0));
                    }
            }
            const TV a0 = row_sum(ps.th0, ls), a1 = row_sum(ps.th1, ls);
            lpq += ps.en;
            if constexpr (ST)
            {
#pragma unroll
                for (int k = 0; k < D; ++k)
                    zS[k] = ps.z[k];
            }
            if constexpr (GEN)
            {
                const TV h0 = row_sum(ps.h0, ls), h1 = row_sum(ps.h1, ls);
                if (q == 0 && i < n)
                {
                    RowTerms<TV, D> rt;
                    rt.load(s.row, n, i);
                    TV ab[4];
                    lpq += general_row<TV, D>(rt, xi, a0, a1, h0, h1, ab);
                    st_vec<TV, D>(pnew, n, i, xi, pl);
                    if constexpr (sizeof(TV) == 8)
                    {
                        st_keep2(s.th + 4 * (int64_t)i, make_double2(ab[0], ab[1]), pl);
                        st_keep2(s.th + 4 * (int64_t)i + 2, make_double2(ab[2], ab[3]), pl);
                    }
                    else
                    {
                        st_keep2(s.th + 4 * (int64_t)i, make_float2(ab[0], ab[1]), pl);
                        st_keep2(s.th + 4 * (int64_t)i + 2, make_float2(ab[2], ab[3]), pl);
                    }
                }
            }
            else if (q == 0 && i < n)
            {
                lpq += (double)s.T[0] * ((double)a0 * (double)a0) + (double)s.T[1] * ((double)a1 * (double)a1);
                st_vec<TV, D>(pnew, n, i, xi, pl);
                if constexpr (sizeof(TV) == 8)
                    st_keep2(s.th + 2 * (int64_t)i, make_double2(a0, a1), pl);
                else
                    st_keep2(s.th + 2 * (int64_t)i, make_float2(a0, a1), pl);
            }
        }
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
        const TV al = (TV)(rr / pq);
        // pass 2: K p row by row, x += alpha p, r -= alpha K p, r . r
        double lrr = 0;
        for (int g = g0 + warp; g < g1; g += nw)
        {
            const int i = g * R + rl, ii = min(i, n - 1);
            TV xi[D], y[D], ti0 = TV(0), ti1 = TV(0);
            ld_vec<TV, D>(pnew, n, ii, xi, pl);
            if constexpr (!GEN)
            {
                const auto v = ld_keep2(s.th + 2 * (int64_t)ii, pl);
                ti0 = v.x;
                ti1 = v.y;
            }
#pragma unroll
            for (int k = 0; k < D; ++k)
                y[k] = ST ? zS[k] : TV(0);
            Pass1<TV, D, GEN> ps; // GEN: the row's G and H again
            const int t1 = (g + 1) * s.width;
            int t = g * s.width;
            int cn[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                cn[u] = (t + u < t1) ? column(t + u) : 0;
            for (; t < t1; t += U)
            {
                int co[U];
                TV pv[U][D], cv[U][D], ta[U], tb[U], T[U], M[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    co[u] = cn[u];
                    cn[u] = (t + U + u < t1) ? column(t + U + u) : 0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (t + u < t1)
                    {
                        if constexpr (!ST)
                            ld_vec<TV, D>(pnew, n, co[u] >> 1, pv[u], pl);
                        if constexpr (GEN)
                        {
                            const auto v = ld_keep2(s.th + 2 * (int64_t)co[u], pl);
                            ta[u] = v.x;
                            tb[u] = v.y;
                            T[u] = ld_stream(s.tm + (int64_t)(2 * (t + u)) * 32 + lane, pb_);
                            M[u] = ld_stream(s.tm + (int64_t)(2 * (t + u) + 1) * 32 + lane, pb_);
                        }
                        else
                            ta[u] = ld_keep(s.th + co[u], pl);
                        if constexpr (!ST)
                        {
                            const TV *cb = s.c + ((int64_t)(t + u) * D) * 32 + lane;
#pragma unroll
                            for (int k = 0; k < D; ++k)
                                cv[u][k] = ld_stream(cb + k * 32, pb_);
                        }
                    }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (t + u < t1)
                    {
                        const int L = co[u] & 1;
                        if constexpr (ST)
                            staged_cosines(t + u, cv[u]);
                        TV w;
                        if constexpr (GEN)
                        {
                            ps.bond(xi, pv[u], cv[u], L, s.Kn, T[u], M[u]);
                            TV ci = cv[u][0] * xi[0], cj = cv[u][0] * pv[u][0];
#pragma unroll
                            for (int k = 1; k < D; ++k)
                            {
                                ci += cv[u][k] * xi[k];
                                cj += cv[u][k] * pv[u][k];
                            }
                            w = T[u] * (ta[u] - ci) + tb[u] + M[u] * cj;
                        }
                        else if constexpr (ST)
                            w = (L ? s.T[1] : s.T[0]) * (ta[u] + (L ? ti1 : ti0));
                        else
                        {
                            TV d = cv[u][0] * (xi[0] - pv[u][0]);
#pragma unroll
                            for (int k = 1; k < D; ++k)
                                d += cv[u][k] * (xi[k] - pv[u][k]);
                            w = (L ? s.T[1] : s.T[0]) * (ta[u] + (L ? ti1 : ti0)) + 2 * (L ? s.Kn[1] : s.Kn[0]) * d;
                        }
#pragma unroll
                        for (int k = 0; k < D; ++k)
                            y[k] += cv[u][k] * w;
                    }
            }
#pragma unroll
            for (int k = 0; k < D; ++k)
                y[k] = row_sum(y[k], ls);
            TV G0, G1, H0, H1;
            if constexpr (GEN)
            {
                G0 = row_sum(ps.th0, ls);
                G1 = row_sum(ps.th1, ls);
                H0 = row_sum(ps.h0, ls);
                H1 = row_sum(ps.h1, ls);
            }
            if (q == 0 && i < n)
            {
                if constexpr (GEN)
                {
                    RowTerms<TV, D> rt;
                    rt.load(s.row, n, i);
                    general_close<TV, D>(rt, xi, G0, G1, H0, H1, y);
                }
                const int m = s.mask[i];
                TV rv[D];
                ld_vec<TV, D>(s.r, n, i, rv, pl);
#pragma unroll
                for (int k = 0; k < D; ++k)
                {
                    if (!((m >> k) & 1))
                        rv[k] -= al * y[k];
                    lrr += (double)rv[k] * (double)rv[k];
                    TV *xp = s.x + (int64_t)i * D + k;
                    st_keep(xp, ld_keep(xp, pl) + al * xi[k], pl);
                }
                st_vec<TV, D>(s.r, n, i, rv, pl);
            }
        }
        double rn;
        if (!grid_sum(lrr, s.bar, epoch, s.info, &s_fail, s.part, 0, sh, &rn, s.wait_ns))
            return;
        const bool done = rn <= stop;
        if (done || it >= s.maxit)
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

// ---------------------------------------------------------------------------- cluster form
// A problem whose bonds and vectors fit the shared memory of one thread-block cluster runs its whole
// CG there.  CTA k owns the rows [k*rho, (k+1)*rho), one group per warp; a thread keeps its row's r, p
// and x in registers.  Shared memory holds p and theta of the CTA's own rows and of its halo (the
// other rows that its bonds reach), and r of the halo.  Owners push theta (pass 1) and r (pass 2) of
// each row into the halos that hold it, and every CTA forms its halo's p = r + beta p itself.  The
// pushes and the CTAs' partial sums are asynchronous stores that count bytes on the receiver's
// mbarriers, so an exchange needs one bounded wait, no fence and no load from another CTA.  The last
// warp owns no rows: it exchanges the sums, p . K p while the others run pass 2 (which needs theta,
// but alpha only at its end).
//
// Bound by latency below about 200 rows per CTA and by shared-memory bandwidth above.  Pass 1 keeps z in
// registers, so pass 2 reads theta alone of the partners.  Measured per iteration against k_cg on the
// assembled matrix: hexagonal plates of 725, 2,900 and 11,500 particles 7.9 -> 2.9, 8.3 -> 3.0 and 9.9 ->
// 5.2 us; simple-cubic cubes of 1,000 and 4,096 particles 9.8 -> 3.6 and 10.6 -> 4.8 us.  With p gathered
// again in pass 2: 2.9, 3.5 and 5.75 us on the plates, 3.9 and 5.9 on the cubes.  Gathering the neighbours
// from other CTAs' shared memory instead took 4.0, 5.2 and 7.8 us on the plates.
struct ClusterShared
{
    double part[2][16]; // partial sums of the CTAs: [0] r.r, [1] p.Kp
    double sh[2][32];
    double tot[2];
    unsigned long long mbar[3]; // arrivals: [0] sums of r.r and r of the halo, [1] sums of p.Kp, [2] theta of the halo
    int lo[16], hi[16]; // rows whose values each CTA holds
    int fail;           // the first section in which a wait passed its limit
    int pad;
};

// bytes of one held row: p, theta (GEN: alpha and beta per layer); of one halo row: r besides
template <int D, bool GEN>
constexpr int kHeldBytes = 8 * D + (GEN ? 32 : 16);
template <int D, bool GEN>
constexpr int kSlotBytes = 32 * (4 + 8 * D + (GEN ? 16 : 0));
constexpr size_t kClusterFixed = (sizeof(ClusterShared) + 127) / 128 * 128;

// The exchange of one sum by one warp: adds the CTA's `nw` warp sums sh[which][.], sends the total
// to every CTA, waits for theirs (and `halo` bytes of pushes on the same mbarrier) and leaves the
// cluster's total in tot[which].  A wait past its limit marks section `sec` as failed.
__device__ __forceinline__ void exchange_sum(ClusterShared *cs, unsigned nc, unsigned rank, int nw, int which,
                                             unsigned parity, unsigned halo, int sec, int64_t *info,
                                             unsigned long long wait_ns)
{
    const int l = threadIdx.x & 31;
    double t = l < nw ? cs->sh[which][l] : 0.0;
    t = wsum(t);
    const unsigned bar = smem_addr(&cs->mbar[which]);
    if (l < (int)nc)
        push(mapa(smem_addr(&cs->part[which][rank]), l), mapa(bar, l), t);
    if (l == 0)
        expect_bytes(bar, halo + 8u * nc);
    __syncwarp();
    const bool done = __all_sync(0xffffffffu, cluster_wait(bar, parity, wait_ns));
    t = (l < (int)nc) ? cs->part[which][l] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, o);
    if (l == 0)
    {
        cs->tot[which] = t;
        if (!done)
        {
            atomicOr(reinterpret_cast<unsigned long long *>(info + 1), 2ull);
            atomicMin(&cs->fail, sec);
        }
    }
}

template <int D, bool GEN>
__global__ void __launch_bounds__(1024, 1) k_cg_bond_cluster(BondCG<double> s, int G, int slots, int held)
{
    extern __shared__ __align__(128) unsigned char csm[];
    if (*s.flag & s.flag_bad)
    {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), (unsigned long long)kBondDeclined);
        return;
    }
    ClusterShared *cs = reinterpret_cast<ClusterShared *>(csm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5; // nw = G + 1
    const int n = s.n, ls = s.ls, R = 32 >> ls, q = lane & ((1 << ls) - 1), rho = G * R;
    const bool helper = warp == G;
    const unsigned nc = gridDim.x, rank = blockIdx.x; // the grid is one cluster
    // shared memory after the fixed part: p (x, y), theta, r of the halo (x, y), cosines, T and M,
    // p.z, r.z of the halo, columns; `held` rows, halo = held - rho
    const int nhalo = held - rho;
    double2 *pS = reinterpret_cast<double2 *>(csm + kClusterFixed);
    double2 *thS = pS + held, *th1S = thS + held;
    double2 *rS = thS + (GEN ? 2 : 1) * (size_t)held;
    double *cS = reinterpret_cast<double *>(rS + nhalo);
    double *tmS = cS + (size_t)slots * D * 32;
    double *pzS = tmS + (GEN ? (size_t)slots * 64 : 0);
    double *rzS = pzS + (D == 3 ? held : 0);
    unsigned *colS = reinterpret_cast<unsigned *>(rzS + (D == 3 ? nhalo : 0));
    const unsigned barR = smem_addr(&cs->mbar[0]), barT = smem_addr(&cs->mbar[2]);
    if (threadIdx.x == 0)
    {
        cs->fail = 1 << 30;
        for (int k = 0; k < 3; ++k)
            mbar_init(&cs->mbar[k]);
        mbar_init_done();
    }
    // the rows each CTA holds: its own and all that its bonds reach
    for (int k = warp; k < (int)nc; k += nw)
    {
        int lo = k * rho, hi = lo + rho - 1;
        for (int g = k * G + lane; g < min(s.ng, (k + 1) * G); g += 32)
        {
            lo = min(lo, s.reach[2 * g]);
            hi = max(hi, s.reach[2 * g + 1]);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0)
        {
            cs->lo[k] = lo;
            cs->hi[k] = min(hi + 1, max(n, k * rho + rho));
        }
    }
    __syncthreads();
    const int a0 = (int)rank * rho, lo = cs->lo[rank], hi = min(cs->hi[rank], n); // own rows, held rows
    const int below = a0 - lo, nh = below + max(0, hi - (a0 + rho));
    const int gfirst = min(s.ng, (int)rank * G), g = gfirst + warp;
    const bool act = !helper && g < s.ng;
    const int tfirst = gfirst * s.width;
    const int t0 = act ? g * s.width : tfirst, t1 = act ? t0 + s.width : tfirst;
    for (int t = t0; t < t1; ++t)
    {
        const int e = (t - tfirst) * 32 + lane;
        colS[e] = (unsigned)(s.col[(int64_t)t * 32 + lane] - 2 * lo); // 2 * held row + layer
        if constexpr (D == 2)
            reinterpret_cast<double2 *>(cS)[e] = make_double2(s.c[((int64_t)t * 2) * 32 + lane],
                                                              s.c[((int64_t)t * 2 + 1) * 32 + lane]);
        else
#pragma unroll
            for (int k = 0; k < D; ++k)
                cS[((t - tfirst) * D + k) * 32 + lane] = s.c[((int64_t)t * D + k) * 32 + lane];
        if constexpr (GEN)
            reinterpret_cast<double2 *>(tmS)[e] = make_double2(s.tm[((int64_t)t * 2) * 32 + lane],
                                                               s.tm[((int64_t)t * 2 + 1) * 32 + lane]);
    }
    // halo row h is particle lo + h below the own rows, a0 + rho + (h - below) above them
    for (int h = threadIdx.x; h < nh; h += blockDim.x)
    {
        const int j = h < below ? lo + h : a0 + rho + (h - below);
        rS[h] = make_double2(s.b[(int64_t)j * D], s.b[(int64_t)j * D + 1]);
        pS[j - lo] = make_double2(0.0, 0.0);
        if constexpr (D == 3)
        {
            rzS[h] = s.b[(int64_t)j * D + 2];
            pzS[j - lo] = 0.0;
        }
    }
    const int i = a0 + warp * R + (lane >> ls), li = i - lo; // this thread's row, its place among the held
    const bool valid = act && i < n, own = valid && q == 0;
    const int ir = min(i, n - 1);
    double r[D], p[D], x[D];
    double loc = 0;
    int m = 0;
    unsigned targets = 0; // CTAs whose halo has this row
    if (act)
    {
        m = s.mask[ir];
#pragma unroll
        for (int k = 0; k < D; ++k)
        {
            r[k] = valid ? s.b[(int64_t)ir * D + k] : 0.0;
            p[k] = 0.0;
            x[k] = 0.0;
            if (own)
                loc += r[k] * r[k];
        }
        if (own)
            for (unsigned k = 0; k < nc; ++k)
                if (k != rank && i >= cs->lo[k] && i < cs->hi[k])
                    targets |= 1u << k;
    }
    RowTerms<double, D> rt;
    if constexpr (GEN)
        rt.load(s.row, n, ir);
    cluster_sync();
    // Sections are numbered so that every warp takes the same decision on a failed wait: a warp that
    // is ahead marks a later section than the one the others are about to check.
    int sec = 0;
    unsigned parR = 0, parP = 0;
    const unsigned thBytes = (GEN ? 32u : 16u) * nh, rBytes = 8u * D * nh;
    loc = wsum(loc);
    if (lane == 0)
        cs->sh[0][warp] = loc;
    __syncthreads();
    if (helper)
        exchange_sum(cs, nc, rank, nw, 0, parR, 0u, sec, s.info, s.wait_ns);
    __syncthreads();
    double rr = cs->tot[0];
    bool ok = cs->fail > sec;
    parR ^= 1;
    const double stop = (s.abs_stop >= 0) ? s.abs_stop : s.rtol * rr + s.atol;
    const bool lead = rank == 0 && threadIdx.x == 0;
    if (lead)
    {
        s.info[0] = 0;
        reinterpret_cast<double *>(s.info)[2] = rr;
        reinterpret_cast<double *>(s.info)[3] = rr;
    }
    double beta = 0.0;
    const int e0 = t0 - tfirst, e1 = t1 - tfirst;
    for (int64_t it = 1; ok && !(rr <= stop); ++it)
    {
        // p of the own rows and of the halo
        if (act)
        {
#pragma unroll
            for (int k = 0; k < D; ++k)
                p[k] = r[k] + beta * p[k];
            if (q == 0) // rows past the end too: missing bonds point at the last row, with c = 0
            {
                pS[li] = make_double2(p[0], p[1]);
                if constexpr (D == 3)
                    pzS[li] = p[2];
            }
        }
        for (int h = threadIdx.x; h < nh; h += blockDim.x)
        {
            const int l = h < below ? h : rho + h;
            const double2 rv = rS[h], pv = pS[l];
            pS[l] = make_double2(rv.x + beta * pv.x, rv.y + beta * pv.y);
            if constexpr (D == 3)
                pzS[l] = rzS[h] + beta * pzS[l];
        }
        __syncthreads();
        double lpq = 0, y[D];
        double ti0 = 0.0, ti1 = 0.0, h0 = 0.0, h1 = 0.0;
        if (act)
        {
            Pass1<double, D, GEN, !GEN> ps;
#pragma unroll 2
            for (int e = e0; e < e1; ++e)
            {
                const unsigned co = colS[e * 32 + lane];
                double c[D], xj[D], T = 0.0, M = 0.0;
                const double2 pv = pS[co >> 1];
                xj[0] = pv.x;
                xj[1] = pv.y;
                if constexpr (D == 2)
                {
                    const double2 cv = reinterpret_cast<const double2 *>(cS)[e * 32 + lane];
                    c[0] = cv.x;
                    c[1] = cv.y;
                }
                else
                {
                    xj[2] = pzS[co >> 1];
#pragma unroll
                    for (int k = 0; k < D; ++k)
                        c[k] = cS[(e * D + k) * 32 + lane];
                }
                if constexpr (GEN)
                {
                    const double2 tv = reinterpret_cast<const double2 *>(tmS)[e * 32 + lane];
                    T = tv.x;
                    M = tv.y;
                }
                ps.bond(p, xj, c, (int)(co & 1u), s.Kn, T, M);
            }
            ti0 = row_sum(ps.th0, ls);
            ti1 = row_sum(ps.th1, ls);
            lpq = ps.en;
#pragma unroll
            for (int k = 0; k < D; ++k)
                y[k] = ps.z[k];
            double2 v0 = make_double2(ti0, ti1), v1 = make_double2(0.0, 0.0);
            if constexpr (GEN)
            {
                h0 = row_sum(ps.h0, ls);
                h1 = row_sum(ps.h1, ls);
                double ab[4];
                const double e = general_row<double, D>(rt, p, ti0, ti1, h0, h1, ab);
                if (own)
                    lpq += e;
                v0 = make_double2(ab[0], ab[1]);
                v1 = make_double2(ab[2], ab[3]);
            }
            else if (own)
                lpq += s.T[0] * (ti0 * ti0) + s.T[1] * (ti1 * ti1);
            if (q == 0)
            {
                thS[li] = v0;
                if constexpr (GEN)
                    th1S[li] = v1;
            }
            for (unsigned b = targets; b; b &= b - 1)
            {
                const unsigned k = __ffs(b) - 1, bar = mapa(barT, k);
                const int lk = i - cs->lo[k];
                push2(mapa(smem_addr(thS + lk), k), bar, v0.x, v0.y);
                if constexpr (GEN)
                    push2(mapa(smem_addr(th1S + lk), k), bar, v1.x, v1.y);
            }
        }
        lpq = wsum(lpq);
        if (lane == 0)
            cs->sh[1][warp] = lpq;
        ++sec;
        __syncthreads();
        if (helper)
        {
            if (lane == 0)
                expect_bytes(barT, thBytes);
            exchange_sum(cs, nc, rank, nw, 1, parP, 0u, sec, s.info, s.wait_ns);
        }
        // pass 2 up to alpha: K p row by row
        if (act)
        {
            if (!__all_sync(0xffffffffu, cluster_wait(barT, parP, s.wait_ns)) && lane == 0)
            {
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 2ull);
                atomicMin(&cs->fail, sec);
            }
#pragma unroll 4
            for (int e = e0; e < e1; ++e)
            {
                const unsigned co = colS[e * 32 + lane];
                const int L = (int)(co & 1u);
                double c[D], xj[D], w;
                if constexpr (GEN)
                {
                    const double2 pv = pS[co >> 1];
                    xj[0] = pv.x;
                    xj[1] = pv.y;
                    if constexpr (D == 3)
                        xj[2] = pzS[co >> 1];
                }
                if constexpr (D == 2)
                {
                    const double2 cv = reinterpret_cast<const double2 *>(cS)[e * 32 + lane];
                    c[0] = cv.x;
                    c[1] = cv.y;
                }
                else
                {
#pragma unroll
                    for (int k = 0; k < D; ++k)
                        c[k] = cS[(e * D + k) * 32 + lane];
                }
                if constexpr (GEN)
                {
                    const double2 tv = reinterpret_cast<const double2 *>(tmS)[e * 32 + lane];
                    const double2 ab = (L ? th1S : thS)[co >> 1];
                    double ci = c[0] * p[0], cj = c[0] * xj[0];
#pragma unroll
                    for (int k = 1; k < D; ++k)
                    {
                        ci += c[k] * p[k];
                        cj += c[k] * xj[k];
                    }
                    w = tv.x * (ab.x - ci) + ab.y + tv.y * cj;
                }
                else
                {
                    const double tj = reinterpret_cast<const double *>(thS)[co];
                    w = (L ? s.T[1] : s.T[0]) * (tj + (L ? ti1 : ti0));
                }
#pragma unroll
                for (int k = 0; k < D; ++k)
                    y[k] += c[k] * w;
            }
#pragma unroll
            for (int k = 0; k < D; ++k)
                y[k] = row_sum(y[k], ls);
            if constexpr (GEN)
                general_close<double, D>(rt, p, ti0, ti1, h0, h1, y);
        }
        __syncthreads();
        const double pq = cs->tot[1];
        if (!(ok = cs->fail > sec))
            break;
        parP ^= 1;
        if (pq == 0.0)
        {
            if (lead)
            {
                s.info[0] = it - 1;
                atomicOr(reinterpret_cast<unsigned long long *>(s.info + 1), 4ull);
            }
            break;
        }
        const double al = rr / pq;
        double lrr = 0;
        if (act)
        {
#pragma unroll
            for (int k = 0; k < D; ++k)
            {
                if (valid && !((m >> k) & 1))
                    r[k] -= al * y[k];
                x[k] += al * p[k];
                if (own)
                    lrr += r[k] * r[k];
            }
            for (unsigned b = targets; b; b &= b - 1)
            {
                const unsigned k = __ffs(b) - 1, bar = mapa(barR, k);
                const int h = i - cs->lo[k] - (k < rank ? rho : 0);
                push2(mapa(smem_addr(rS + h), k), bar, r[0], r[1]);
                if constexpr (D == 3)
                    push(mapa(smem_addr(rzS + h), k), bar, r[2]);
            }
        }
        lrr = wsum(lrr);
        if (lane == 0)
            cs->sh[0][warp] = lrr;
        ++sec;
        __syncthreads();
        if (helper)
            exchange_sum(cs, nc, rank, nw, 0, parR, rBytes, sec, s.info, s.wait_ns);
        __syncthreads();
        const double rn = cs->tot[0];
        if (!(ok = cs->fail > sec))
            break;
        parR ^= 1;
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
    if (own)
#pragma unroll
        for (int k = 0; k < D; ++k)
            s.x[(int64_t)i * D + k] = x[k];
    if (!ok)
        drain_pushes();
    cluster_sync(); // no CTA leaves while another may still push into its shared memory
}

// ---------------------------------------------------------------------------- host side
template <int D, bool GEN>
static size_t cluster_smem(int G, int R, int width, int held)
{
    return kClusterFixed + (size_t)kHeldBytes<D, GEN> * held + (size_t)8 * D * (held - G * R) +
           (size_t)kSlotBytes<D, GEN> * G * width;
}

static size_t cluster_smem_of(const Problem &p, int G, int held)
{
    const int R = 32 >> p.bo_ls;
    if (p.dim == 2)
        return p.bo_gen ? cluster_smem<2, true>(G, R, p.bo_width, held) : cluster_smem<2, false>(G, R, p.bo_width, held);
    return p.bo_gen ? cluster_smem<3, true>(G, R, p.bo_width, held) : cluster_smem<3, false>(G, R, p.bo_width, held);
}

// the most rows a CTA of an nc-CTA cluster holds: its own and those its bonds reach
static int held_rows(const Problem &p, int nc)
{
    const int R = 32 >> p.bo_ls, G = div_up(p.bo_ng, nc);
    int most = G * R;
    for (int k = 0; k < nc; ++k)
    {
        int lo = k * G * R, hi = lo + G * R - 1;
        for (int g = k * G; g < std::min(p.bo_ng, (k + 1) * G); ++g)
        {
            lo = std::min(lo, p.bo_reach_host[2 * (size_t)g]);
            hi = std::max(hi, p.bo_reach_host[2 * (size_t)g + 1]);
        }
        most = std::max(most, hi + 1 - lo);
    }
    return most;
}

static bool cluster_holds(const Problem &p, int nc)
{
    const int G = div_up(p.bo_ng, nc);
    return G <= 31 && cluster_smem_of(p, G, held_rows(p, nc)) <= kClusterSmem;
}

static const void *cluster_kernel(const Problem &p)
{
    if (p.dim == 2)
        return p.bo_gen ? (const void *)k_cg_bond_cluster<2, true> : (const void *)k_cg_bond_cluster<2, false>;
    return p.bo_gen ? (const void *)k_cg_bond_cluster<3, true> : (const void *)k_cg_bond_cluster<3, false>;
}

// largest cluster for the problem's kernel, asked once per kernel
static int cluster_limit(const Problem &p)
{
    static std::atomic<int> known[2][2]; // 1 + the answer
    std::atomic<int> &k = known[p.dim == 3][p.bo_gen];
    int v = k.load();
    if (v == 0)
    {
        v = 1 + max_cluster(cluster_kernel(p));
        k.store(v);
    }
    return v - 1;
}

static int groups_of(int n, int ls) { return div_up(n, 32 >> ls); }

// shared memory of the staged grid form on `grid` blocks, and whether that form serves them
static size_t staged_smem(const Problem &p, int grid, size_t real)
{
    return (size_t)div_up(p.bo_ng, grid) * p.bo_width * 32 * (p.dim * real + sizeof(int));
}
static bool staged_fits(const Problem &p, int grid, size_t real)
{
    return !p.bo_gen && div_up(p.bo_ng, grid) <= kStagedThreads / 32 && staged_smem(p, grid, real) <= kStagedSmem;
}

// Builds the layout once per problem.  The cluster form when the problem fits one cluster (the grid
// form's barriers alone cost more than a whole cluster iteration up to that size: 11,500 particles take
// 5.2 us in a cluster and 6.7 us on the grid), with as many lanes per row as keep a CTA within 8 warps
// of rows (725 particles at 8, 4, 2, 1 lanes: 3.2, 2.9, 2.9, 3.2 us; 4,096 in 3D at 2, 1: 5.9, 5.4 us);
// else lanes per row so that the grid's threads are used.  Elastic-damage and fatigue particles keep the assembled matrix: their load paths
// end in torn or unloaded states whose stresses are what the linear solves leave of their rounding.
cudaError_t setup_bond_op(Problem &p)
{
    p.bo_ok = false;
    if (p.max_bonds < 1 || p.max_bonds > kMaxBonds || p.nbonds >= ((int64_t)1 << 30) ||
        (p.desc.ptype != LPMGPU_ELASTIC && p.desc.ptype != LPMGPU_J2))
        return cudaSuccess;
    cudaError_t e;
    const int ncmax = cluster_limit(p);
    auto shape = [&p](int ls) {
        p.bo_ls = ls;
        p.bo_width = (p.max_bonds + (1 << ls) - 1) >> ls;
        p.bo_ng = groups_of(p.n, ls);
    };
    int lc = 3, lg = 0; // lanes per row of the cluster form and of the grid form
    while (lc > 0 && div_up(groups_of(p.n, lc), std::max(ncmax, 1)) > 8)
        --lc;
    // the grid form: lanes per row so that the staged form's threads are used, where it serves, else the
    // general one's
    auto lanes = [&p](int threads) {
        int l = 0;
        while (l < 2 && ((int64_t)p.n << (l + 1)) <= (int64_t)p.num_sms * threads)
            ++l;
        return l;
    };
    lg = lanes(kStagedThreads);
    shape(lg);
    if (p.bo_gen || !staged_fits(p, p.num_sms, sizeof(double)))
        lg = lanes(kBondThreads);
    shape(lc);
    const int G = div_up(p.bo_ng, std::max(ncmax, 1));
    p.bo_nc = (ncmax > 0 && G <= 31 && cluster_smem_of(p, G, G * (32 >> lc)) <= kClusterSmem) ? ncmax : 0;
    while (p.bo_nc > p.bo_ng)
        p.bo_nc /= 2;
    const bool grid_used = p.desc.precision != LPMGPU_MIXED || p.dim == 2; // solve_dim's rule
    if (p.bo_nc == 0)
        shape(lg);
    if (p.bo_nc == 0 && !grid_used)
        return cudaSuccess;
    // one allocation for all arrays, each on a 256-byte boundary, sized for either shape
    const size_t n = (size_t)p.n;
    const int rs = 4 * p.dim + p.dim * (p.dim + 1) / 2;
    const bool mixed = p.desc.precision == LPMGPU_MIXED && p.dim == 2;
    size_t ent = (size_t)p.bo_ng * p.bo_width * 32, ngr = (size_t)p.bo_ng;
    if (p.bo_nc > 0)
    {
        const size_t w = (p.max_bonds + (1 << lg) - 1) >> lg;
        ent = std::max(ent, (size_t)groups_of(p.n, lg) * w * 32);
        ngr = std::max(ngr, (size_t)groups_of(p.n, lg));
    }
    size_t at = 0;
    auto take = [&at](size_t bytes) {
        const size_t o = at;
        at = (at + bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_col = take(4 * ent), o_src = take(4 * ent), o_reach = take(8 * ngr + 4), o_mask = take(n),
                 o_c = take(8 * p.dim * ent), o_th = take(32 * n), o_tm = take(p.bo_gen ? 16 * ent : 0),
                 o_row = take(p.bo_gen ? 8 * rs * n : 0), o_c32 = take(mixed ? 4 * p.dim * ent : 0),
                 o_th32 = take(mixed ? 16 * n : 0), o_tm32 = take(mixed && p.bo_gen ? 8 * ent : 0),
                 o_row32 = take(mixed && p.bo_gen ? 4 * rs * n : 0);
    unsigned char *mem = nullptr;
    if ((e = dalloc(p, &mem, at)) != cudaSuccess)
        return e;
    p.bo_col = reinterpret_cast<int *>(mem + o_col);
    p.bo_src = reinterpret_cast<int *>(mem + o_src);
    p.bo_reach = reinterpret_cast<int *>(mem + o_reach);
    p.bo_mask = mem + o_mask;
    p.bo_c = reinterpret_cast<double *>(mem + o_c);
    p.bo_th = reinterpret_cast<double *>(mem + o_th);
    p.bo_tm = p.bo_gen ? reinterpret_cast<double *>(mem + o_tm) : nullptr;
    p.bo_row = p.bo_gen ? reinterpret_cast<double *>(mem + o_row) : nullptr;
    p.bo_c32 = mixed ? reinterpret_cast<float *>(mem + o_c32) : nullptr;
    p.bo_th32 = mixed ? reinterpret_cast<float *>(mem + o_th32) : nullptr;
    p.bo_tm32 = mixed && p.bo_gen ? reinterpret_cast<float *>(mem + o_tm32) : nullptr;
    p.bo_row32 = mixed && p.bo_gen ? reinterpret_cast<float *>(mem + o_row32) : nullptr;
    int *bad = reinterpret_cast<int *>(mem + o_reach + 8 * ngr); // zeroed with the rest
    auto fill = [&]() -> cudaError_t {
        k_bo_fill<<<div_up(p.bo_ng, 4), 128, 0, p.stream>>>(p.n, p.bo_ng, p.bo_ls, p.bo_width, p.bstart, p.nb0, p.bp2,
                                                            p.brev, p.bo_col, p.bo_src, p.bo_reach, bad);
        return cudaGetLastError();
    };
    if ((e = fill()) != cudaSuccess)
        return e;
    int hbad = 0;
    p.bo_reach_host.resize(2 * (size_t)p.bo_ng);
    if (p.bo_nc > 0 && (e = cudaMemcpyAsync(p.bo_reach_host.data(), p.bo_reach, sizeof(int) * p.bo_reach_host.size(),
                                            cudaMemcpyDeviceToHost, p.stream)) != cudaSuccess)
        return e;
    if ((e = cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, p.stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(p.stream)) != cudaSuccess)
        return e;
    if (p.bo_nc > 0 && !cluster_holds(p, p.bo_nc))
    { // the halos do not fit: the grid form
        p.bo_nc = 0;
        shape(lg);
        if ((e = fill()) != cudaSuccess)
            return e;
    }
    p.bo_ok = hbad == 0 && (p.bo_nc > 0 || grid_used);
    return cudaSuccess;
}

// Takes the bond form of the K that was just assembled: the state's cosines, coefficients and mask.
cudaError_t launch_bond_refresh(Problem &p, bool apply_bc)
{
    cudaError_t e;
    if ((e = cudaMemsetAsync(&p.scal->bond_flag, 0, sizeof(int), p.stream)) != cudaSuccess)
        return e;
    const int64_t ent = (int64_t)p.bo_ng * p.bo_width * 32;
    const int gp = div_up(ent, 256), gr = div_up(p.n, 128);
#define BO_REFRESH(D, GEN)                                                                                             \
    do                                                                                                                 \
    {                                                                                                                  \
        k_bo_pack<D, GEN><<<gp, 256, 0, p.stream>>>(ent, p.bo_src, p.brev, p.cs, p.Kn, p.Tv, p.bdamage, p.bo_c,        \
                                                    p.bo_c32, p.bo_tm, p.bo_tm32, &p.scal->bond_flag);                          \
        k_bo_rows<D, GEN><<<gr, 128, 0, p.stream>>>(p.n, apply_bc ? 1 : 0, p.bstart, p.nb0, p.cons, p.damage_visual,   \
                                                    p.cs, p.Kn, p.Tv, p.bdamage, p.cs_sum, p.bo_mask, p.bo_row,        \
                                                    p.bo_row32, &p.scal->bond_flag);                                            \
    } while (0)
    if (p.dim == 2 && p.bo_gen)
        BO_REFRESH(2, true);
    else if (p.dim == 2)
        BO_REFRESH(2, false);
    else if (p.bo_gen)
        BO_REFRESH(3, true);
    else
        BO_REFRESH(3, false);
#undef BO_REFRESH
    p.ctr.kernel_launches += 2;
    return cudaGetLastError();
}

int bond_flags_bad(const Problem &p)
{
    return p.bo_gen ? kBondUnsupported : (kBondUnsupported | kBondGeneral);
}

template <typename TV>
static void fill_args(const Problem &p, BondCG<TV> &s)
{
    constexpr bool f64 = sizeof(TV) == 8;
    s.n = p.n;
    s.ng = p.bo_ng;
    s.ls = p.bo_ls;
    s.width = p.bo_width;
    s.col = p.bo_col;
    if constexpr (f64)
    {
        s.c = p.bo_c;
        s.tm = p.bo_tm;
        s.row = p.bo_row;
        s.th = p.bo_th;
    }
    else
    {
        s.c = p.bo_c32;
        s.tm = p.bo_tm32;
        s.row = p.bo_row32;
        s.th = p.bo_th32;
    }
    s.mask = p.bo_mask;
    s.flag = &p.scal->bond_flag;
    s.reach = p.bo_reach;
    s.flag_bad = bond_flags_bad(p);
    const bool hex = p.cell.lattice == LPMGPU_HEXAGON2D; // k_bonds_fill's assignment
    s.Kn[0] = (TV)p.kntv[0];
    s.Kn[1] = (TV)(hex ? p.kntv[0] : p.kntv[1]);
    s.T[0] = s.T[1] = (TV)(hex ? p.kntv[1] : p.kntv[2]);
    const int64_t bytes = (int64_t)p.bo_ng * p.bo_width * 32 * (4 + (int64_t)sizeof(TV) * (p.dim + (p.bo_gen ? 2 : 0)));
    s.keep = bytes <= (int64_t)80 << 20;
    s.bar = p.barrier;
    s.part = p.partials;
    s.info = p.cg_info;
    s.wait_ns = p.wait_ns;
}

static cudaError_t clear_words(Problem &p)
{
    cudaError_t e = cudaMemsetAsync(p.barrier, 0, 2 * sizeof(unsigned), p.stream);
    return e != cudaSuccess ? e : cudaMemsetAsync(p.cg_info, 0, 4 * sizeof(int64_t), p.stream);
}

// CTAs of the cluster form under the handle's launch limit (cg_grid); 0 when it does not fit them
static int cluster_ctas(const Problem &p)
{
    int nc = p.bo_nc;
    while (nc > 0 && p.cg_grid > 0 && nc > p.cg_grid)
        nc /= 2;
    return nc > 0 && nc != p.bo_nc && !cluster_holds(p, nc) ? 0 : nc;
}

cudaError_t enqueue_bond_cluster(Problem &p, const double *b, double *x, double rtol, double atol, double abs_stop,
                                 int64_t maxit)
{
    cudaError_t e = clear_words(p);
    if (e != cudaSuccess)
        return e;
    BondCG<double> s;
    fill_args(p, s);
    s.rtol = rtol;
    s.atol = atol;
    s.abs_stop = abs_stop;
    s.maxit = maxit;
    s.b = b;
    s.x = x;
    s.r = s.pa = s.pb = nullptr;
    const int nc = cluster_ctas(p);
    int G = div_up(p.bo_ng, nc), slots = G * p.bo_width, held = held_rows(p, nc);
    p.cg_form = "cluster";
    void *args[] = {&s, &G, &slots, &held};
    if ((e = launch_cluster(cluster_kernel(p), nc, 32 * (G + 1), cluster_smem_of(p, G, held), args, p.stream)) != cudaSuccess)
        return e;
    p.ctr.kernel_launches++;
    p.ctr.cg_launches++;
    return cudaSuccess;
}

template <typename TV, int D, bool GEN>
static cudaError_t bond_grid(const Problem &p, int *grid)
{
    int occ = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_cg_bond<TV, D, GEN, false>, kBondThreads, 0);
    if (e != cudaSuccess)
        return e;
    *grid = std::max(1, std::min(p.num_sms * std::min(std::max(occ, 1), 1), p.bo_ng));
    return cudaSuccess;
}

template <typename TV, int D, bool GEN>
static cudaError_t launch_grid(Problem &p, BondCG<TV> &s)
{
    int grid = 0;
    cudaError_t e = bond_grid<TV, D, GEN>(p, &grid);
    if (e != cudaSuccess)
        return e;
    if (p.cg_grid > 0 && p.cg_grid < grid)
        grid = p.cg_grid;
    void *args[] = {&s};
    bool staged = false;
    p.cg_form = "general";
    if constexpr (!GEN)
        if (staged_fits(p, grid, sizeof(TV)))
        {
            staged = true;
            p.cg_form = "staged";
            if ((e = cudaFuncSetAttribute(k_cg_bond<TV, D, GEN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kStagedSmem)) != cudaSuccess)
                return e;
            e = cudaLaunchCooperativeKernel((const void *)k_cg_bond<TV, D, GEN, true>, dim3(grid), dim3(kStagedThreads), args,
                                            staged_smem(p, grid, sizeof(TV)), p.stream);
        }
    if (!staged)
        e = cudaLaunchCooperativeKernel((const void *)k_cg_bond<TV, D, GEN, false>, dim3(grid), dim3(kBondThreads), args, 0,
                                        p.stream);
    if (e != cudaSuccess)
        return e;
    p.ctr.kernel_launches++;
    p.ctr.cg_launches++;
    return cudaSuccess;
}

template <typename TV>
cudaError_t enqueue_bond_grid(Problem &p, const TV *b, TV *x, TV *r, TV *pa, TV *pb, double rtol, double atol,
                              double abs_stop, int64_t maxit)
{
    cudaError_t e = clear_words(p);
    if (e != cudaSuccess)
        return e;
    BondCG<TV> s;
    fill_args(p, s);
    s.rtol = rtol;
    s.atol = atol;
    s.abs_stop = abs_stop;
    s.maxit = maxit;
    s.b = b;
    s.x = x;
    s.r = r;
    s.pa = pa;
    s.pb = pb;
    if (p.dim == 2)
        return p.bo_gen ? launch_grid<TV, 2, true>(p, s) : launch_grid<TV, 2, false>(p, s);
    if constexpr (sizeof(TV) == 8)
        return p.bo_gen ? launch_grid<TV, 3, true>(p, s) : launch_grid<TV, 3, false>(p, s);
    return cudaErrorInvalidValue; // FP32 in 3D runs on the assembled matrix (solve_dim)
}
template cudaError_t enqueue_bond_grid<double>(Problem &, const double *, double *, double *, double *, double *, double,
                                               double, double, int64_t);
template cudaError_t enqueue_bond_grid<float>(Problem &, const float *, float *, float *, float *, float *, double, double,
                                              double, int64_t);

bool bond_cluster_fits(const Problem &p) { return p.bo_ok && p.bo_valid && cluster_ctas(p) > 0; }

// the default launch size of the problem's CG on the bond form: its cluster's CTAs, else the grid
template <typename TV>
cudaError_t bond_default_grid(const Problem &p, int *grid)
{
    if (p.bo_nc > 0)
    {
        *grid = p.bo_nc;
        return cudaSuccess;
    }
    if (p.dim == 2)
        return p.bo_gen ? bond_grid<TV, 2, true>(p, grid) : bond_grid<TV, 2, false>(p, grid);
    if constexpr (sizeof(TV) == 8)
        return p.bo_gen ? bond_grid<TV, 3, true>(p, grid) : bond_grid<TV, 3, false>(p, grid);
    return cudaErrorInvalidValue;
}
template cudaError_t bond_default_grid<double>(const Problem &, int *);
template cudaError_t bond_default_grid<float>(const Problem &, int *);

} // namespace lpm
