"""The pivot that the direct solve reports for a stiffness that is not positive definite
(lpm-cpp_b200/csrc/direct.cu; PARDISO's error -4 has no such detail).

All bonds of one particle get a negative stiffness (per-bond properties), so its diagonal block is
negative and elimination fails at the latest there.  The particle is the first, a middle or the last one
in the reordered system: a pivot of the first 32-column block, of a later one, of the ragged last one.
The expected pivot is the first one that is not positive in a plain elimination of the exported matrix in
the order of lpmgpu_band_order; it and the pivots before it lie at least 1e-6 of the largest diagonal
entry away from zero, far more than rounding.  The handle stays usable: the CG reports as before, and a
direct solve reports the same pivot again."""
import re

import numpy as np
import pytest

from _util import LPM, gpu_problem, oracle_problem
from test_bond_form import _block
from test_direct_host import _rcm

L = LPM.LatticeType
NOT_SPD = 12


def _negative(case, place):
    """The case with the bonds of the particle at `place` (0 to 1) of the order turned negative."""
    o = oracle_problem(case)
    nb0, nb1, p2 = o.bonds()
    nconn, _, conns = o.conns()
    st, rank, _ = _rcm(np.concatenate([[0], np.cumsum(nconn)]), conns)
    assert st == 0
    bc = np.unique(np.concatenate([case.groups[k] for k in ("top", "bottom")]))
    free = np.setdiff1d(np.arange(case.n), bc)
    at = free[np.argsort(rank[free])[int(round(place * (len(free) - 1)))]]
    owner = np.repeat(np.arange(case.n), nb0 + nb1)
    sign = np.where((owner == at) | (p2 == at), -1.0, 1.0)
    kn, tv = o.bond_kntv()
    case.bonds = (nb0, nb1, p2)
    case.bond_props = (kn * sign, tv * sign, np.zeros(len(p2)))
    return case, rank


def _first_bad_pivot(IK, JK, K, n, dim, rank):
    N = n * dim
    A = np.zeros((N, N))
    A[np.repeat(np.arange(N), np.diff(IK)), np.asarray(JK) - 1] = K
    A = A + np.triu(A, 1).T
    order = np.argsort((dim * rank[:, None] + np.arange(dim)).reshape(-1))
    A = A[np.ix_(order, order)]
    margin = 1e-6 * np.abs(A.diagonal()).max()
    for j in range(N):
        assert abs(A[j, j]) > margin, (j, A[j, j])
        if A[j, j] < 0:
            return j + 1
        A[j + 1:, j + 1:] -= np.outer(A[j + 1:, j], A[j, j + 1:]) / A[j, j]
    return 0


CASES = [(L.Hexagon2D, 2.0, 0.0), (L.Hexagon2D, 2.0, 0.5), (L.Hexagon2D, 2.0, 1.0), (L.SimpleCubic3D, 2.1, 0.5)]


@pytest.mark.parametrize("lattice,size,place", CASES)
def test_the_cases_fail_where_they_are_meant_to(lattice, size, place):
    case, rank = _negative(_block(lattice, size), place)
    o = oracle_problem(case)
    o.update_geometry()
    o.update_force_state()
    o.apply_bc([(case.groups[g], {"x": 0, "y": 1, "z": 2}[f], v) for g, f, v in case.steps[0][0]], [])
    o.assemble(True)
    _, IK, JK, K = o.export_csr()
    bad = _first_bad_pivot(IK, JK, K, case.n, case.dim, rank)
    block, last = (bad - 1) // 32, (case.n * case.dim - 1) // 32
    assert bad > 0 and (case.n * case.dim) % 32 != 0
    assert {0.0: block == 0, 0.5: 0 < block < last, 1.0: block == last}[place], (bad, block, last)


@pytest.mark.gpu
@pytest.mark.parametrize("lattice,size,place", CASES)
def test_reported_pivot(lattice, size, place):
    case, rank = _negative(_block(lattice, size), place)
    g = gpu_problem(case)
    g.apply_load_step(case.load_step(0))
    g.update_force_state()
    g.assemble(True)
    g.update_rr()
    _, IK, JK, K = g.export_csr()
    want = _first_bad_pivot(np.asarray(IK), JK, K, g.n, g.dim, rank)
    for _ in range(2):
        with pytest.raises(LPM.LpmGpuError) as ex:
            g.solve_direct()
        assert ex.value.status == NOT_SPD
        assert int(re.search(r"pivot (\d+)", str(ex.value)).group(1)) == want
    g.close()
