"""The time limits of the device-side waits, form by form.

Each form of the linear solve runs with a limit of 1 ns, which its first exchange, grid sum or copy
outlasts, and must report LPMGPU_ERR_TIMEOUT; with the default limit back, the same handle must give the
bits of a handle that never failed.  The forms: the bond CG in one cluster, staged and general on the
grid; the assembled CG in one cluster, resident, general (FP64 and FP32) and streamed; the direct solve's
factorisation and substitution.  No fault, trap or endless loop is involved: a wait that passes its limit
ends the kernel."""
import numpy as np
import pytest

from _util import LPM
from test_bond_form import TIGHT, _block, _moved

L = LPM.LatticeType
# lattice, size, exact assembly, precision, slices per block (0: the default grid)
FORMS = {
    "bond_cluster_2d": (L.Hexagon2D, 4.0, False, 0, 0),
    "bond_cluster_3d": (L.SimpleCubic3D, 2.4, False, 0, 0),
    "bond_staged": (L.Hexagon2D, 25.0, False, 0, 0),
    "bond_general": (L.SimpleCubic3D, 14.4, False, 0, 0),
    "assembled_cluster": (L.Hexagon2D, 4.0, True, 0, 0),
    "assembled_resident": (L.Hexagon2D, 14.3, True, 0, 0),
    "assembled_general": (L.SimpleCubic3D, 8.4, True, 0, 0),
    "assembled_fp32": (L.SimpleCubic3D, 8.4, True, 1, 0),
    "assembled_streamed": (L.SimpleCubic3D, 8.4, True, 1, 17),
}


def _system(case, exact, precision, grid):
    g = LPM.GpuProblem(case.assembly(), precision=LPM.Precision(precision), **TIGHT)
    g.set_assembly_exact(exact)
    g.set_cg_grid(grid)
    g.apply_load_step(case.load_step(0))
    g.set_xyz(_moved(case))
    g.update_force_state()
    g.assemble(True)
    g.update_rr()
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("form", list(FORMS))
def test_limit_is_reported_and_the_handle_recovers(form):
    lattice, size, exact, precision, per_block = FORMS[form]
    case = _block(lattice, size)
    grid = max(1, case.n // 32 // per_block) if per_block else 0
    ref = _system(case, exact, precision, grid)
    want, _ = ref.solve_linear()
    ref.close()
    g = _system(case, exact, precision, grid)
    g.set_wait_limit_ns(1)
    for _ in range(3):
        with pytest.raises(LPM.LpmGpuError) as ex:
            g.solve_linear()
        assert ex.value.status == LPM.ERR_TIMEOUT, str(ex.value)
    g.set_wait_limit_ns(0)
    got, st = g.solve_linear()
    assert st["cg_iters"] > 0 and np.array_equal(got, want)
    g.close()


@pytest.mark.gpu
def test_direct_solve():
    """The factorisation's grid barriers, then the copies of the substitution on a factor that exists."""
    case = _block(L.Hexagon2D, 6.0)
    ref = _system(case, False, 0, 0)
    want, _ = ref.solve_direct()
    ref.close()
    g = _system(case, False, 0, 0)
    for _ in range(2):  # without a factor, then with one
        g.set_wait_limit_ns(1)
        for _ in range(2):
            with pytest.raises(LPM.LpmGpuError) as ex:
                g.solve_direct()
            assert ex.value.status == LPM.ERR_TIMEOUT, str(ex.value)
        g.set_wait_limit_ns(0)
        got, _ = g.solve_direct()
        assert np.array_equal(got, want)
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("ns", [1, 300, 600, 1000, 1500, 2000, 3000])
def test_batch_member(ns):
    """A batch member whose cluster solve times out, at once or on the way, is left between two Newton
    iterations: without the unfinished increment that the update behind the solve would add.  The states
    there may be are those of the same iterations driven one by one."""
    case = _block(L.Hexagon2D, 6.0)
    ref = LPM.GpuProblem(case.assembly(), **TIGHT)
    ref.apply_load_step(case.load_step(0))
    ref.assemble(True)
    states = [ref.state(("xyz",))["xyz"]]
    for _ in range(8):
        ref.update_force_state()
        ref.update_rr()
        u = np.zeros_like(case.xyz)
        u[:, :case.dim] = ref.solve_linear()[0].reshape(case.n, case.dim)
        states.append(states[-1] + u)
        ref.set_xyz(states[-1])
    ref.close()
    for _ in range(5):
        g = LPM.GpuProblem(case.assembly(), **TIGHT)
        g.set_wait_limit_ns(ns)
        batch = LPM.Batch()
        mid = batch.add(g, [case.load_step(0)])
        batch.run()
        info = batch.member(mid)
        assert info["state"] in (1, 2) and (ns > 1 or info["state"] == 2)
        if info["state"] == 2:
            assert info["status"] == LPM.ERR_TIMEOUT
            xyz = g.state(("xyz",))["xyz"]
            assert any(np.array_equal(xyz, s) for s in states)
        batch.close()
        g.close()
