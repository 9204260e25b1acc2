"""Handles of different sizes on different host threads at once (lpmgpu.h: one thread per handle).

Elastic plates on the assembled matrix, which a launch keeps in the shared memory of 20 blocks with 147 KB
each or of 18 blocks with 74 KB (the resident form of k_cg; the six launches fit the GPU side by side).
Each thread solves over and over, one CG iteration a solve so that the launches follow one another closely:
every solve must succeed, with the bits of the handle's first one."""
import threading

import numpy as np
import pytest

from _util import LPM
from test_bond_form import TIGHT, _block, _moved

pytestmark = pytest.mark.gpu


def test_two_sizes_on_six_threads():
    handles = []
    for size, per_block in ((8.0, 3), (4.4, 1)) * 3:
        case = _block(LPM.LatticeType.Hexagon2D, size)
        slices = -(-case.n // 32)
        g = LPM.GpuProblem(case.assembly(), cg_maxit=1, **TIGHT)
        g.set_assembly_exact(True)
        g.set_cg_grid(-(-slices // per_block))
        g.apply_load_step(case.load_step(0))
        g.set_xyz(_moved(case))
        g.update_force_state()
        g.assemble(True)
        g.update_rr()
        handles.append((g, g.solve_linear()[0]))
    errors = []
    start = threading.Barrier(len(handles))

    def work(g, want):
        try:
            start.wait()
            for _ in range(4000):
                x, _ = g.solve_linear()
            assert np.array_equal(x, want)
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=h) for h in handles]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, _ in handles:
        g.close()
