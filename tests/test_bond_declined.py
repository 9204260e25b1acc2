"""A K without a bond form costs one look at it, not one per solve.

Bonds broken in one direction only have no bond form (test_bond_form.py checks the solutions): the first
solve with such a K launches the bond CG, which declines, and the CG on the assembled matrix; later solves
with the same K launch the latter alone, until the next assembly."""
import pytest

from _util import LPM
from test_bond_form import TIGHT, _block, _with_props

L = LPM.LatticeType


@pytest.mark.gpu
@pytest.mark.parametrize("size", [4.0, 25.0])
def test_one_look_per_assembly(size):
    case = _with_props(_block(L.Hexagon2D, size), 4, 0.3, one_sided=True)
    g = LPM.GpuProblem(case.assembly(), **TIGHT)
    g.apply_load_step(case.load_step(0))
    g.update_force_state()
    launches = [g.counters()["cg_launches"]]
    for _ in range(2):
        g.assemble(True)
        g.update_rr()
        for _ in range(3):
            g.solve_linear()
            launches.append(g.counters()["cg_launches"])
    assert [b - a for a, b in zip(launches, launches[1:])] == [2, 1, 1, 2, 1, 1]
    g.close()
