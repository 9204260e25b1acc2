"""The CG whose blocks keep their share of the assembled matrix in shared memory (lpm-cpp_b200/csrc/cg.cu:
k_cg's RES form).

A solve on the assembled matrix equals the solve on the bond form.  The grid sets the slices per block: 1
to 4 (16 to 4 columns a warp: the resident form), 5 and 8 (no longer fits; the general form), with a
partial last slice and blocks of unequal slice counts.  FP64: both stop at a residual of 1e-12 of the
right-hand side, and the bar is 1e-9; mixed: 1e-8, that of the other mixed solves."""
import pytest

from _util import LPM, rel
from test_bond_form import _block, _solve

L = LPM.LatticeType


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(0, 1e-9), (1, 1e-8)])
@pytest.mark.parametrize("lattice,size", [(L.Hexagon2D, 12.0), (L.Square2D, 14.3)])
@pytest.mark.parametrize("per_block", [1, 2, 3, 4, 5, 8])
def test_resident_solve(lattice, size, per_block, precision, tol):
    case = _block(lattice, size)
    slices = -(-case.n // 32)
    grid = -(-slices // per_block)
    xa, _, _ = _solve(case, False)
    xb, _, st = _solve(case, True, precision=precision, grid=grid)
    assert st["cg_maxit_hits"] == 0
    assert rel(xb, xa) <= tol, rel(xb, xa)
