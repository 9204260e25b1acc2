"""The autotuner times what the default solve runs (lpmgpu_autotune).

A small 2D problem on the assembled matrix solves in one cluster at the default launch size and on the
grid at any other.  The log of a child process (LPMGPU_LOG, one line per CG launch) names the form of each
timed launch: the default's two launches, which come first, must be the cluster's, and the other
candidates' the grid's."""
import os
import subprocess
import sys

import pytest

from _util import ROOT

CHILD = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
from _util import LPM
from test_bond_form import TIGHT, _block
case = _block(LPM.LatticeType.Hexagon2D, 6.0)
g = LPM.GpuProblem(case.assembly(), **TIGHT)
g.set_assembly_exact(True)
g.apply_load_step(case.load_step(0))
g.update_force_state()
res = g.autotune(iterations=20)
print(len(res["candidates"]), res["candidates"][0] == res["grid_default"] == -(-case.n // 32))
g.close()
"""


@pytest.mark.gpu
def test_default_candidate_runs_in_the_cluster():
    code = CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LPMGPU_LOG": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
    count, default = r.stdout.split()
    forms = ["cluster" in line for line in r.stderr.splitlines() if line.startswith("lpmgpu cg launch")]
    assert default == "True" and len(forms) == 2 * int(count) >= 4
    assert forms == [True] * 2 + [False] * (len(forms) - 2), r.stderr
