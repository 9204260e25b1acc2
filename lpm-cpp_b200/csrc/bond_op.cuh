// The bond form of the stiffness product and the CG kernels that run on it (bond_op.cu).
//
// K of one assembly is the sum over bond layers of the terms of assembly_fast.cu.  Its product
// with a vector x needs no matrix: with c_a the cosines of bond a = i -> j (c of the opposite
// bond is -c_a), T and Kn the layer's coefficients and
//     d_a     = c_a . (x_i - x_j)                        one value per bond
//     theta_i = sum of d_a over i's bonds of the layer   one value per particle and layer
// the row of particle i is
//     (K x)_i = sum_a c_a [ T (theta_i + theta_j) + 2 Kn d_a ]
// and x . K x = sum_i T theta_i^2 + sum_a Kn d_a^2, which is known as soon as theta is.  The sum of
// 2 Kn c_a d_a is known then too (z), so the second pass needs only theta_j of the partners.
//
// With coefficients that differ from bond to bond (per-bond properties, continuous damage), with
// T_a = (1 - D_a) Tv_a, F_a = (1 - D_a)(2 Kn_a + Tv_a) equal for a bond and its opposite, S and U the
// layer's sums of c and T c, and G_i = sum c_a . x_j, H_i = sum 2 T_a c_a . x_j:
//     alpha_i = 3/4 S_i.x_i - 1/2 G_i,   beta_i = 1/4 (U_i.x_i - H_i)
//     (K x)_i = Self_i x_i + sum_a c_a [ T_a alpha_j + beta_j - T_a c_a.x_i + (T_a - F_a) c_a.x_j ]
//               - sum_layers (3/8 S_i H_i + 1/4 U_i G_i)
//     x . K x = sum_i x_i.Self_i x_i - sum_a (T_a (c_a.x_i)^2 - (T_a - F_a)(c_a.x_i)(c_a.x_j))
//               + sum_layers (-3/4 (S_i.x_i) H_i - 1/2 (U_i.x_i) G_i + 1/2 G_i H_i)
// These are the sums of assembly_fast.cu's closed form, taken path by path in another order.
//
// Layout.  Rows in particle order, in groups of 32 / S rows; S lanes share a row.  Group g holds
// the bond slots [g*width, (g + 1)*width); slot t of the row at lanes r*S .. r*S + S - 1 holds S of
// its bonds, one per lane.  Entry (t, lane): col = 2 * partner + layer at col[t*32 + lane], the
// cosines at c[(t*D + k)*32 + lane], T and T - F at tm[(2*t + k)*32 + lane].  A missing bond has
// c = 0 and its own row as partner.
#pragma once

#include <cstdint>

#include "lpm_internal.cuh"

namespace lpm
{

constexpr int kBondGeneral = 1;     // flag bit: some bond's coefficients are not its layer's
constexpr int kBondUnsupported = 2; // flag bit: K of this assembly has no bond form here
constexpr int kBondDeclined = 8;    // status bit of a CG launch: the flags rule this kernel out

template <typename TV>
struct BondCG
{
    int n, ng, ls, width; // rows, groups, log2 of the lanes per row, slots per group
    const int *col;
    const TV *c, *tm, *row;
    const unsigned char *mask; // bit k: component k is constrained
    const int *reach;          // per group: lowest and highest row its bonds touch (cluster form)
    const int *flag;
    int flag_bad;              // flag bits this kernel cannot run with
    TV T[2], Kn[2];
    int keep;                  // the bond arrays fit L2 beside the vectors
    double rtol, atol, abs_stop;
    int64_t maxit;
    unsigned *bar;
    double *part;
    int64_t *info;
    unsigned long long wait_ns;
    const TV *b;
    TV *x, *r, *pa, *pb, *th;
};

} // namespace lpm
