"""The FP32 CG that streams its matrix through shared memory (lpm-cpp_b200/csrc/cg.cu: k_cg_stream), which
serves 3D solves whose blocks all hold more than half a slice per warp.

A mixed-precision solve on the assembled matrix equals the FP64 solve of the same state; both stop at a
residual of 1e-12 of the right-hand side and the bar is 1e-8, that of the other mixed solves.  The grid
sets the slices per block: 16 (the general kernel, just below the rule), 17 (the smallest), a warp's
second slice only in some warps, all slices in one block.  The 8.4 mm cubes end in a partial slice and
have rows of every length modulo the chunk of three block columns."""
import pytest

from _util import LPM, rel
from test_bond_form import _block, _solve

L = LPM.LatticeType


@pytest.mark.gpu
@pytest.mark.parametrize("lattice", [L.SimpleCubic3D, L.FCC3D, L.BCC3D])
@pytest.mark.parametrize("per_block", [16, 17, 32, 33, 40, 10**6])
def test_streamed_mixed_solve(lattice, per_block):
    case = _block(lattice, 8.4)
    slices = -(-case.n // 32)
    grid = max(1, slices // per_block)
    assert per_block > slices or slices // grid >= per_block
    xa, _, _ = _solve(case, True)
    xb, _, st = _solve(case, True, precision=1, grid=grid)
    assert st["cg_maxit_hits"] == 0 and st["refinements"] >= 1
    assert rel(xb, xa) <= 1e-8, rel(xb, xa)
