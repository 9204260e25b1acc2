"""Row order of the sliced-ELL layout in 3D (lpm-cpp_b200/csrc/topology.cu: rows sorted by connection
count within windows of 1,024 rows).

The solve on the assembled matrix, which reads that layout, equals the solve on the bond form, which does
not.  Sizes sit at the window's edges: one window less a row, full, with one row more, two windows, and a
last window of a slice and a row.  Both stop at a residual of 1e-12 of the right-hand side; the bar is
1e-9, that of the other linear-solve tests."""
import numpy as np
import pytest

from _util import CFG, LPM
from test_bond_form import _same


@pytest.mark.gpu
@pytest.mark.parametrize("lattice", [LPM.LatticeType.SimpleCubic3D, LPM.LatticeType.FCC3D, LPM.LatticeType.BCC3D])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 2048, 2081])
def test_assembled_solve_at_window_edges(lattice, n):
    c = CFG.sc_cube(size=6.0, radius=0.2, steps=1, total_disp=0.001, lattice=lattice)
    assert c.n > n
    c.xyz, c.types = np.ascontiguousarray(c.xyz[:n]), c.types[:n]
    z = c.xyz[:, 2]
    for name, sel in (("top", z > z.max() - 0.05), ("bottom", z < z.min() + 0.05)):
        if name in c.groups:
            c.groups[name] = np.nonzero(sel)[0].astype(np.int32)
    c.groups = {k: v[v < n] for k, v in c.groups.items()}
    _same(c)
