"""Which form of the CG a linear solve runs, on both sides of each rule of the dispatch.

The log of a child process (LPMGPU_LOG, one line per CG launch) names the operator, the precision and the
form.  Sizes and launch sizes are those that the tests of the single forms take for their edges, so that
each of them is known to run the kernel it is about: one cluster or the grid, bonds in shared memory or
not, the assembled matrix in shared memory, streamed or neither."""
import os
import subprocess
import sys

import pytest

from _util import LPM, ROOT
from test_bond_form import _block, _same

# lattice, size, exact assembly, precision, groups or slices per block (0: the default grid) -> the form
FORMS = [
    ("Hexagon2D", 20.0, 0, 0, 0, "bond fp64 cluster/2d"),
    ("Hexagon2D", 25.0, 0, 0, 0, "bond fp64 staged/2d"),
    ("Hexagon2D", 25.0, 0, 0, 16, "bond fp64 staged/2d"),
    ("Hexagon2D", 25.0, 0, 0, 17, "bond fp64 general/2d"),
    ("Hexagon2D", 25.0, 0, 1, 16, "bond fp32 staged/2d"),
    ("Hexagon2D", 25.0, 0, 1, 17, "bond fp32 general/2d"),
    ("Square2D", 25.0, 0, 0, 0, "bond fp64 cluster/2d"),
    ("Square2D", 29.0, 0, 0, 16, "bond fp64 staged/2d"),
    ("Square2D", 29.0, 0, 1, 16, "bond fp32 staged/2d"),
    ("Square2D", 29.0, 0, 0, 17, "bond fp64 general/2d"),
    ("Square2D", 29.0, 0, 1, 17, "bond fp32 general/2d"),
    ("SimpleCubic3D", 5.6, 0, 0, 0, "bond fp64 cluster/3d"),
    ("SimpleCubic3D", 13.2, 0, 0, 0, "bond fp64 staged/3d"),
    ("SimpleCubic3D", 14.0, 0, 0, 0, "bond fp64 general/3d"),
    ("SimpleCubic3D", 8.4, 0, 1, 0, "assembled fp32 general/3d"),
    ("SimpleCubic3D", 8.4, 0, 1, 17, "assembled fp32 streamed/3d"),
    ("SimpleCubic3D", 8.4, 0, 1, 16, "assembled fp32 general/3d"),
    ("Hexagon2D", 8.3, 1, 0, 0, "assembled fp64 cluster/2d"),
    ("Hexagon2D", 12.0, 1, 0, 4, "assembled fp64 resident/2d"),
    ("Hexagon2D", 12.0, 1, 0, 5, "assembled fp64 general/2d"),
    ("Hexagon2D", 12.0, 1, 1, 4, "assembled fp32 resident/2d"),
]

CHILD = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
from _util import LPM
from test_bond_form import TIGHT, _block, _moved
for name, size, exact, precision, per_block, form in {forms!r}:
    case = _block(LPM.LatticeType[name], size)
    threads = 1 if exact or (precision and case.dim == 3) else 148 * 512
    lanes = 1 if threads == 1 else 4 if case.n * 4 <= threads else 2 if case.n * 2 <= threads else 1
    units = -(-case.n * lanes // 32)
    streamed = precision and case.dim == 3
    grid = 0 if per_block == 0 else units // per_block if streamed else -(-units // per_block)
    g = LPM.GpuProblem(case.assembly(), precision=LPM.Precision(precision), **TIGHT)
    g.set_assembly_exact(bool(exact))
    g.set_cg_grid(grid)
    g.apply_load_step(case.load_step(0))
    g.set_xyz(_moved(case))
    g.update_force_state()
    g.assemble(True)
    g.update_rr()
    print("==", file=sys.stderr, flush=True)
    g.solve_linear()
    g.close()
"""


@pytest.mark.gpu
def test_forms_of_the_dispatch():
    code = CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"), forms=FORMS)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600,
                       env={**os.environ, "LPMGPU_LOG": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
    seen = r.stderr.split("==\n")[1:]
    assert len(seen) == len(FORMS)
    wrong = []
    for want, log in zip(FORMS, seen):
        launches = [line for line in log.splitlines() if line.startswith("lpmgpu cg launch")]
        if not launches or not all(f": {want[-1]} " in line for line in launches):
            wrong.append((want, launches[:2]))
    assert not wrong


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("per_block", [0, 16, 17])
def test_square_plate_on_the_grid(per_block, precision):
    """The staged form and its neighbour on a square plate that one cluster does not hold (21,025 particles);
    tolerances as in test_bond_staged.py."""
    case = _block(LPM.LatticeType.Square2D, 29.0)
    groups = -(-case.n * 2 // 32)
    _same(case, precision=precision, grid=-(-groups // per_block) if per_block else 0, tol=1e-8 if precision else 1e-9)
