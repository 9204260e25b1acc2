"""The caller's iteration cap in mixed precision (lpmgpu_desc.cg_maxit) holds for each inner solve.

A refinement goes on from an inner solve that reached the cap, so a cap of 50 iterations still ends at the
tolerance.  Problems small enough for one cluster first solve in FP64 at once; one that reaches the cap
there must go the same way.  Both stop at a residual of 1e-12 of the right-hand side; the bar is 1e-8, that
of the other mixed solves, and 1e-6 for a batch's mixed members, which must also take the Newton iterations
and sum up the reactions that they do alone."""
import numpy as np
import pytest

from _util import LPM, rel
from test_bond_form import TIGHT, _block, _moved

pytestmark = pytest.mark.gpu
L = LPM.LatticeType


@pytest.mark.parametrize("lattice,size", [(L.Hexagon2D, 2.0), (L.Hexagon2D, 6.0), (L.Square2D, 8.3),
                                          (L.SimpleCubic3D, 2.4), (L.FCC3D, 3.0)])
def test_capped_solve_refines(lattice, size):
    case = _block(lattice, size)
    out = []
    for precision, cap in ((0, 0), (1, 50), (1, 0)):
        g = LPM.GpuProblem(case.assembly(), precision=LPM.Precision(precision), cg_maxit=cap, **TIGHT)
        g.apply_load_step(case.load_step(0))
        g.set_xyz(_moved(case))
        g.update_force_state()
        g.assemble(True)
        g.update_rr()
        out.append(g.solve_linear())
        g.close()
    (x, _), (xc, sc), (xu, su) = out
    assert su["cg_maxit_hits"] == 0 and su["refinements"] == 1  # not capped: in FP64 at once
    assert sc["cg_maxit_hits"] >= 1 and sc["refinements"] >= 2
    assert rel(xc, x) <= 1e-8 and rel(xu, x) <= 1e-8


@pytest.mark.parametrize("tangent", [False, True])
def test_capped_batch_members(tangent):
    cases = [_block(L.Hexagon2D, 4.0), _block(L.Hexagon2D, 6.0), _block(L.SimpleCubic3D, 2.4)]

    def problem(case, precision, cap):
        return LPM.GpuProblem(case.assembly(), precision=LPM.Precision(precision), cg_maxit=cap, tol_iter=1e-9,
                              tangent=tangent, **TIGHT)

    batch = LPM.Batch()
    handles = [problem(c, 1, 50) for c in cases]
    mids = [batch.add(g, [c.load_step(0)]) for g, c in zip(handles, cases)]
    batch.run()
    for case, g, mid in zip(cases, handles, mids):
        alone, free = problem(case, 1, 50), problem(case, 0, 0)
        ok, st = alone.solve_load_step(case.load_step(0))
        assert ok
        ok, s0 = free.solve_load_step(case.load_step(0))
        assert ok
        info = batch.member(mid)
        assert info["state"] == 1 and info["total"]["cg_maxit_hits"] >= 1
        assert info["total"]["newton_solves"] == st["newton_solves"] == s0["newton_solves"]
        assert abs(info["total"]["reaction_norm"] - s0["reaction_norm"]) <= 1e-6 * s0["reaction_norm"]
        u = free.state(("xyz",))["xyz"] - case.xyz
        for h in (g, alone):
            assert rel(h.state(("xyz",))["xyz"] - case.xyz, u) <= 1e-6
            h.close()
        free.close()
    batch.close()
