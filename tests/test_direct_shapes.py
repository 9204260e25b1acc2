"""The band Cholesky solve (lpmgpu_solve_direct) at the edges of its blocks: fewer unknowns than one
32-column block, a ragged last block, bands narrower than a block, wide enough for several rows of
window tiles, and too wide for the substitution's shared-memory panels (half-bandwidth above 415).
Both solves of a system agree within 1e-9, the bar of the other linear-solve tests: the factor is
backward stable and the CG stops at a residual of 1e-12 of the right-hand side."""
import numpy as np
import pytest

from _util import CFG, LPM, gpu_problem, rel

pytestmark = pytest.mark.gpu


def _plate(nx, ny, lattice):
    r = 0.1
    j, i = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    if lattice == LPM.LatticeType.Hexagon2D:
        x, y = 2 * r * i + r * (j % 2), r * np.sqrt(3.0) * j
    else:
        x, y = 2 * r * i, 2 * r * j
    c = CFG.hex_plate(size=1.0, radius=r, steps=1, total_disp=0.001)
    c.lattice = lattice
    c.xyz = np.ascontiguousarray(np.stack([x, y, 0 * x], -1).reshape(-1, 3).astype(float))
    c.types = np.zeros(c.n, np.int32)
    c.groups = {"bottom": np.nonzero(c.xyz[:, 1] < 1e-9)[0].astype(np.int32),
                "top": np.nonzero(c.xyz[:, 1] > c.xyz[:, 1].max() - 1e-9)[0].astype(np.int32)}
    return c


HEX, SQ = LPM.LatticeType.Hexagon2D, LPM.LatticeType.Square2D
CASES = [(HEX, 3, 4), (HEX, 4, 4), (SQ, 4, 4), (SQ, 3, 11), (HEX, 2, 40), (HEX, 5, 33), (HEX, 12, 13), (SQ, 31, 33),
         (HEX, 52, 53), (HEX, 75, 75)]


@pytest.mark.parametrize("lattice,nx,ny", CASES)
def test_plates(lattice, nx, ny):
    _check(_plate(nx, ny, lattice))


@pytest.mark.parametrize("lattice", [LPM.LatticeType.SimpleCubic3D, LPM.LatticeType.BCC3D])
def test_cubes(lattice):
    _check(CFG.sc_cube(size=2.1, radius=0.2, steps=1, total_disp=0.001, lattice=lattice))


def _check(case):
    g = gpu_problem(case, cg_rtol=1e-24, cg_atol=0.0)
    g.apply_load_step(case.load_step(0))
    for scale in (1.0, 1.001):  # a second K: the factor is renewed
        g.set_xyz(case.xyz * scale)
        g.update_force_state()
        g.assemble(True)
        g.update_rr()
        xc, _ = g.solve_linear()
        xd, _ = g.solve_direct()
        if scale != 1.0:
            assert rel(xd, xc) <= 1e-9
    again, _ = g.solve_direct()  # the same factor
    assert np.array_equal(again, xd)
    g.close()
