"""The assembled-matrix CG inside one cluster (lpm-cpp_b200/csrc/cg_cluster.cu) keeps the bits of the
grid kernel's solve: the same sums in the same order.

lpmgpu_set_cg_grid with the grid's default (one block per slice of 32 rows) asks for the grid kernel,
so both run on the same system; exact assembly keeps the bond form out of the way.  Sizes: less than
one slice, one slice and one row, a CTA without a slice, a slice more than a full share, the largest
that fits and the first that does not (which runs the grid kernel both times)."""
import numpy as np
import pytest

from _util import CFG, LPM, gpu_problem

pytestmark = pytest.mark.gpu


def _solve(case, grid):
    g = gpu_problem(case, cg_rtol=1e-24, cg_atol=0.0)
    g.set_assembly_exact(True)
    g.set_cg_grid(grid)
    g.apply_load_step(case.load_step(0))
    rng = np.random.default_rng(3)
    u = rng.uniform(-1, 1, case.xyz.shape) * 1e-4
    u[:, 2] = 0
    g.set_xyz(case.xyz + u)
    g.update_force_state()
    g.assemble(True)
    g.update_rr()
    x, st = g.solve_linear()
    g.close()
    return x, st


@pytest.mark.parametrize("size", [0.6, 1.0, 1.1, 1.9, 3.0, 4.4, 4.5, 6.0, 8.0, 8.3, 8.8])
def test_cluster_keeps_the_grid_kernels_bits(size):
    case = CFG.hex_plate(size=size, radius=0.1, steps=1, total_disp=0.001)
    xa, sa = _solve(case, 0)
    xb, sb = _solve(case, (case.n + 31) // 32)
    assert sa["cg_iters"] == sb["cg_iters"] and sa["cg_maxit_hits"] == sb["cg_maxit_hits"] == 0
    assert np.array_equal(xa, xb)


def test_square_lattice():
    c = CFG.hex_plate(size=7.0, radius=0.1, steps=1, total_disp=0.001)
    c.lattice, c.xyz = LPM.LatticeType.Square2D, LPM.createPlateSQ2D(c.box, LPM.UnitCell(LPM.LatticeType.Square2D, 0.1))
    y = c.xyz[:, 1]
    c.groups = {"top": np.nonzero(y > y.max() - 0.1)[0].astype(np.int32),
                "bottom": np.nonzero(y < y.min() + 0.1)[0].astype(np.int32)}
    c.types = np.zeros(c.n, np.int32)
    (xa, sa), (xb, sb) = _solve(c, 0), _solve(c, (c.n + 31) // 32)
    assert sa["cg_iters"] == sb["cg_iters"] and np.array_equal(xa, xb)


def test_cap_and_zero_right_hand_side():
    case = CFG.hex_plate(size=3.0, radius=0.1, steps=1, total_disp=0.001)
    out = []
    for grid in (0, (case.n + 31) // 32):
        g = LPM.GpuProblem(case.assembly(), cg_maxit=5, cg_rtol=1e-24, cg_atol=0.0)
        g.set_assembly_exact(True)
        g.set_cg_grid(grid)
        g.update_force_state()
        g.assemble(True)
        x0, s0 = g.solve_linear()
        g.apply_load_step(case.load_step(0))
        g.update_force_state()
        g.assemble(True)
        g.update_rr()
        x, st = g.solve_linear()
        out.append((x0, s0["cg_iters"], x, st["cg_iters"], st["cg_maxit_hits"]))
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert out[0][4] == 1
