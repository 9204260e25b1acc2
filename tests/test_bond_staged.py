"""The grid form of the bond CG with its bonds in shared memory (lpm-cpp_b200/csrc/bond_op.cu: k_cg_bond's
ST form) at the edges of its rule.

A solve on the bond form equals the solve on the assembled matrix.  The grid sets the groups per block: the
default, 16 (a group for every warp of the staged form), 17 (no longer one each: the general form), blocks
of unequal counts.  The 13.2 mm cube at the default grid takes the largest share that is staged, the 14 mm
one is just too large.  Tolerances as in test_bond_form.py: 1e-9, mixed 1e-8."""
import pytest

from _util import LPM
from test_bond_form import _block, _same

L = LPM.LatticeType


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("lattice,size", [(L.Hexagon2D, 25.0), (L.Square2D, 25.0), (L.SimpleCubic3D, 8.4), (L.FCC3D, 7.0)])
@pytest.mark.parametrize("per_block", [0, 16, 17])
def test_groups_per_block(lattice, size, per_block, precision):
    case = _block(lattice, size)
    lanes = 4 if case.n * 4 <= 148 * 512 else 2 if case.n * 2 <= 148 * 512 else 1
    groups = -(-case.n * lanes // 32)
    _same(case, precision=precision, grid=-(-groups // per_block) if per_block else 0, tol=1e-8 if precision else 1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("size", [13.2, 14.0])
def test_largest_share(size):
    _same(_block(L.SimpleCubic3D, size))
