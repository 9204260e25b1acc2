"""The bond form of the stiffness product (lpm-cpp_b200/csrc/bond_op.cuh) against the assembled K.

CPU: the two formulas of the bond form, restated in numpy over the oracle's bonds, reproduce the
oracle's stiffness (Stiffness::calcStiffness2D/3D, include/stiffness.h:198-361) on every lattice,
uniform and with per-bond coefficients and damage.  Tolerance 1e-12 of |K||x|: a row sums at most
about 200 products of cosines and coefficients, each rounded a few times.

GPU: a linear solve on the bond form equals the solve on the assembled matrix (the handle in
exact-assembly mode) of the same state.  Both stop at a residual of 1e-12 of the right-hand side,
so the solutions differ by at most about that times the condition number's square root; the bar is
1e-9, that of the other linear-solve tests.  Sizes sit at the edges of the layout: below one group
of rows, one row more or less than full groups, the cluster form with and without a full last CTA,
and problems too large for one cluster."""
import numpy as np
import pytest

from _util import CFG, LPM, gpu_problem, hetero_plate, oracle_problem, rel

HEX, SQ, SC, FCC, BCC = (LPM.LatticeType.Hexagon2D, LPM.LatticeType.Square2D, LPM.LatticeType.SimpleCubic3D,
                         LPM.LatticeType.FCC3D, LPM.LatticeType.BCC3D)
TIGHT = dict(cg_rtol=1e-24, cg_atol=0.0)


def _block(lattice, size, ptype=LPM.ParticleType.Elastic):
    """A plate or cube of the lattice in a box of the given size: bottom held, top moved."""
    if lattice == HEX:
        return CFG.hex_plate(size=size, radius=0.1, steps=1, total_disp=0.001)
    if lattice == SQ:
        c = CFG.hex_plate(size=size, radius=0.1, steps=1, total_disp=0.001)
        c.lattice, c.xyz = LPM.LatticeType.Square2D, LPM.createPlateSQ2D(c.box, LPM.UnitCell(SQ, 0.1))
        y = c.xyz[:, 1]
        c.groups = {"top": np.nonzero(y > y.max() - 0.1)[0].astype(np.int32),
                    "bottom": np.nonzero(y < y.min() + 0.1)[0].astype(np.int32)}
        c.types = np.zeros(len(c.xyz), np.int32)
        return c
    return CFG.sc_cube(size=size, radius=0.2, steps=1, total_disp=0.001, lattice=lattice)


def _moved(case, seed=5):
    rng = np.random.default_rng(seed)
    u = rng.uniform(-1, 1, case.xyz.shape) * 2e-3 * case.radius
    if case.dim == 2:
        u[:, 2] = 0.0
    return case.xyz * (1 + 1e-3) + u


# ------------------------------------------------------------------------------------ formulas
def _dense_oracle_k(o, n, dim):
    o.assemble(False)
    Kp, IK, JK, K = o.export_csr()
    A = np.zeros((n * dim, n * dim))
    row = np.repeat(np.arange(n * dim), np.diff(IK))
    A[row, np.asarray(JK) - 1] = K
    return A + np.triu(A, 1).T


def _bond_product(o, xyz, kn, tv, dmg, x, uniform):
    """K x by bond_op.cuh's formulas; x of shape (n, dim)."""
    nb0, nb1, p2 = o.bonds()
    n, dim = x.shape
    nb = nb0 + nb1
    i = np.repeat(np.arange(n), nb)
    L = (np.arange(len(p2)) - np.repeat(np.cumsum(nb) - nb, nb) >= np.repeat(nb0, nb)).astype(int)
    d = xyz[i] - xyz[p2]
    c = (d / np.linalg.norm(d, axis=1)[:, None])[:, :dim]
    c[np.abs(dmg - 1) < 1e-6] = 0.0
    key = 2 * i + L

    def seg(v):
        out = np.zeros((2 * n,) + v.shape[1:])
        np.add.at(out, key, v)
        return out

    def rows(v):
        out = np.zeros((n,) + v.shape[1:])
        np.add.at(out, i, v)
        return out

    ci, cj = (c * x[i]).sum(1), (c * x[p2]).sum(1)
    kj = 2 * p2 + L
    if uniform:
        th = seg(ci - cj)
        y = rows(c * (tv * (th[key] + th[kj]) + 2 * kn * (ci - cj))[:, None])
        return y, (0.5 * tv * (th[key] + th[kj]) * (ci - cj)).sum() + (kn * (ci - cj) ** 2).sum()
    T, F = (1 - dmg) * tv, (1 - dmg) * (2 * kn + tv)
    S, U, G, H = seg(c), seg(T[:, None] * c), seg(cj), seg(2 * T * cj)
    xx = np.repeat(x, 2, axis=0)
    s, u = (S * xx).sum(1), (U * xx).sum(1)
    al, be = 0.75 * s - 0.5 * G, 0.25 * (u - H)
    selfb = rows(F[:, None, None] * c[:, :, None] * c[:, None, :] + T[:, None, None] * c[:, :, None] * S[key][:, None, :])
    selfb = np.triu(selfb) + np.transpose(np.triu(selfb, 1), (0, 2, 1))
    sx = np.einsum("nij,nj->ni", selfb, x)
    y = rows(c * (T * (al[kj] - ci) + be[kj] + (T - F) * cj)[:, None]) + sx
    y -= (0.375 * S * H[:, None] + 0.25 * U * G[:, None]).reshape(n, 2, dim).sum(1)
    e = (x * sx).sum() - (T * ci * ci - (T - F) * ci * cj).sum() + (-0.75 * s * H - 0.5 * u * G + 0.5 * G * H).sum()
    return y, e


@pytest.mark.parametrize("lattice,size", [(HEX, 1.2), (SQ, 1.1), (SC, 1.7), (FCC, 1.5), (BCC, 1.6)])
@pytest.mark.parametrize("uniform", [True, False])
def test_formulas_against_the_oracle(lattice, size, uniform):
    case = _block(lattice, size)
    o = oracle_problem(case)
    nb0, nb1, p2 = o.bonds()
    i = np.repeat(np.arange(case.n), nb0 + nb1)
    kn, tv = (v.copy() for v in o.bond_kntv())
    dmg = np.zeros(len(p2))
    rng = np.random.default_rng(2)
    pair = np.minimum(i, p2) * case.n + np.maximum(i, p2)
    _, inv = np.unique(pair, return_inverse=True)
    if uniform:  # broken bonds stay within the uniform form: their cosines are zero
        dmg = (rng.random(inv.max() + 1) < 0.05)[inv].astype(np.float64)
    else:
        f = rng.uniform(0.6, 1.4, (2, inv.max() + 1))
        kn, tv = kn * f[0][inv], tv * f[1][inv]
        dmg = (rng.random(inv.max() + 1) * (rng.random(inv.max() + 1) < 0.3))[inv]
        o.set_bond_kntv(kn, tv)
    o.set_bond_damage(dmg)
    xyz = _moved(case)
    o.set_xyz(xyz)
    o.update_geometry()
    o.update_force_state()
    K = _dense_oracle_k(o, case.n, case.dim)
    for seed in range(2):
        x = np.random.default_rng(seed).standard_normal((case.n, case.dim))
        y, e = _bond_product(o, xyz, kn, tv, dmg, x, uniform)
        ref = (K @ x.reshape(-1)).reshape(case.n, case.dim)
        scale = (np.abs(K) @ np.abs(x.reshape(-1))).max()
        assert np.abs(y - ref).max() <= 1e-12 * scale
        assert abs(e - (x * ref).sum()) <= 1e-12 * (np.abs(x.reshape(-1)) @ np.abs(K) @ np.abs(x.reshape(-1)))


# ------------------------------------------------------------------------------------ device
def _solve(case, exact, precision=0, apply_bc=True, grid=0):
    g = gpu_problem(case, precision=precision, **TIGHT)
    g.set_assembly_exact(exact)
    if grid:
        g.set_cg_grid(grid)
    g.apply_load_step(case.load_step(0))
    g.set_xyz(_moved(case))
    g.update_force_state()
    g.assemble(apply_bc)
    g.update_rr()
    x, st = g.solve_linear()
    r = g.residual()
    g.close()
    return x, r, st


def _same(case, precision=0, grid=0, tol=1e-9):
    xa, ra, sa = _solve(case, True, precision)
    xb, rb, sb = _solve(case, False, precision, grid=grid)
    assert np.array_equal(ra, rb)
    assert rel(xb, xa) <= tol, rel(xb, xa)
    assert sb["cg_maxit_hits"] == 0
    if precision == 0:
        assert abs(sb["cg_iters"] - sa["cg_iters"]) <= 0.05 * sa["cg_iters"] + 2
    else:
        assert sb["refinements"] >= 1


# 2.0 mm hex: 110 particles; 3D 1.2 mm: one or two groups of rows; 6 and 12 mm hex: 1,044 and 4,140
# particles in one cluster; 25 mm hex and the 8.4 mm cubes: too large for one cluster
SIZES = [(HEX, 0.8), (HEX, 1.0), (HEX, 2.0), (HEX, 6.1), (HEX, 12.0), (HEX, 25.0), (SQ, 0.7), (SQ, 8.3), (SC, 1.2),
         (SC, 3.3), (SC, 5.0), (SC, 8.4), (FCC, 1.2), (FCC, 3.5), (FCC, 7.0), (BCC, 1.4), (BCC, 4.0), (BCC, 8.4)]


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,size", SIZES)
def test_solve_matches_assembled(lattice, size):
    _same(_block(lattice, size))


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,size", [(HEX, 2.0), (HEX, 25.0), (SQ, 30.0), (SC, 3.3), (SC, 8.4), (BCC, 8.4)])
def test_mixed_solve_matches_assembled(lattice, size):
    _same(_block(lattice, size), precision=1, tol=1e-8)


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [1, 3, 8, 40])
@pytest.mark.parametrize("lattice,size", [(HEX, 6.1), (SC, 3.3)])
def test_forced_launch_sizes(lattice, size, grid):
    _same(_block(lattice, size), grid=grid)


def _with_props(case, seed, damage, one_sided=False):
    """Per-bond Kn/Tv (one factor per pair) and damage on a case's bonds."""
    nb0, nb1, p2 = CFG.bond_lists(case.xyz, LPM.UnitCell(case.lattice, case.radius))
    case.bonds = (nb0, nb1, p2)
    o = oracle_problem(case)
    kn, tv = o.bond_kntv()
    i = np.repeat(np.arange(case.n), nb0 + nb1)
    pair = np.minimum(i, p2) * np.int64(case.n) + np.maximum(i, p2)
    _, inv = np.unique(pair, return_inverse=True)
    rng = np.random.default_rng(seed)
    f = rng.uniform(0.7, 1.3, (2, inv.max() + 1))
    dmg = (damage * rng.random(inv.max() + 1) * (rng.random(inv.max() + 1) < 0.4))[inv]
    if one_sided:
        dmg = np.where((i < p2) & (rng.random(len(p2)) < 0.02), 1.0, dmg)
    case.bond_props = (kn * f[0][inv], tv * f[1][inv], dmg)
    return case


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,size", [(HEX, 0.8), (HEX, 4.0), (HEX, 14.0), (HEX, 25.0), (SC, 2.4), (SC, 8.4), (BCC, 3.0)])
@pytest.mark.parametrize("precision", [0, 1])
def test_per_bond_properties(lattice, size, precision):
    _same(_with_props(_block(lattice, size), 3, 0.6), precision=precision, tol=1e-9 if precision == 0 else 1e-8)


@pytest.mark.gpu
def test_states_without_a_bond_form_keep_the_assembled_matrix():
    """A bond broken in one direction only has no bond form: both modes solve the assembled K, which
    the fast and the exact kernel round differently (1e-12 of max|K|)."""
    case = _with_props(_block(HEX, 4.0), 4, 0.3, one_sided=True)
    _same(case)
    _same(case, precision=1, tol=1e-8)
    _same(hetero_plate())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_zero_right_hand_side_and_iteration_cap(precision):
    """b = 0 solves to zero in no iterations; a cap is reported as a cap, at every problem size."""
    for case in (_block(HEX, 2.0), _block(HEX, 25.0)):
        g = LPM.GpuProblem(case.assembly(), precision=LPM.Precision(precision), cg_maxit=3, **TIGHT)
        g.update_force_state()
        g.assemble(True)
        g.update_rr()
        r = g.residual()
        x, st = g.solve_linear()
        if not r.any():
            assert not x.any() and st["cg_iters"] == 0 and st["cg_maxit_hits"] == 0
        g.apply_load_step(case.load_step(0))
        g.update_force_state()
        g.assemble(True)
        g.update_rr()
        x, st = g.solve_linear()
        assert st["cg_maxit_hits"] >= 1 and st["cg_iters"] >= 3
        g.close()
