"""A host program that ends the device's context once its handles are gone (cudaDeviceReset) and creates
problems again: memory that the library keeps between problems must not outlive the context.

Child processes, since the reset takes the whole process's CUDA state with it: a load step, the reset by
way of the driver (what cudaDeviceReset does), the same load step, twice over, with the same result."""
import os
import subprocess
import sys

import pytest

from _util import ROOT

CHILD = """
import ctypes as C, importlib, sys
sys.path[:0] = [{root!r}, {tests!r}]
from _util import CFG, gpu_problem
drv = C.CDLL("libcuda.so.1")
first = None
for round in range(3):
    for size in (3.0, 4.0):
        case = CFG.hex_plate(size=size, radius=0.1, steps=1, total_disp=0.001)
        g = gpu_problem(case)
        ok, _ = g.solve_load_step(case.load_step(0))
        assert ok
        xyz = g.state()["xyz"].tobytes()
        g.close()
    first = first or xyz
    assert xyz == first
    assert drv.cuDevicePrimaryCtxReset_v2(0) == 0
print("ok")
"""


@pytest.mark.gpu
def test_problems_after_a_reset():
    code = CHILD.format(root=ROOT, tests=os.path.join(ROOT, "tests"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), (r.returncode, r.stdout[-500:], r.stderr[-2000:])
