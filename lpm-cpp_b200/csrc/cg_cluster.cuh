// CGs of small systems inside one thread-block cluster (cg_cluster.cu).
#pragma once

#include "lpm_internal.cuh"

namespace lpm
{

constexpr int kCgDeclined = 8; // status bit: the launch solved nothing, the grid kernel is to be run

// k_cg's solve of a 2D FP64 system on the assembled matrix, the same bits.  sell_cluster_fits: the
// problem is small enough, and its launch size is the default one whose sums the kernel reproduces.
bool sell_cluster_fits(const Problem &p);
cudaError_t enqueue_sell_cluster(Problem &p, const double *b, double *x, double rtol, double atol, double abs_stop,
                                 int64_t maxit);

// the allocation-free CG of a caller's block-CSR matrix: launched when the vectors leave room for a
// matrix; the kernel declines (kCgDeclined in info[1]) when the matrix does not fit beside them
bool bsr_cluster_may_fit(int dim, int nrows);
cudaError_t enqueue_bsr_cluster(int dim, int nrows, const int *rowptr, const int *col, const double *val, const double *b,
                                double *x, double rtol, double atol, int64_t maxit, int64_t *info, cudaStream_t st);

} // namespace lpm
