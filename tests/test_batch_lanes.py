"""The batched CG itself (lpm-cpp_b200/csrc/batch.cu: k_cg_batch, k_cg_batch_sr).

Members whose K has a bond form that fits one cluster solve there, side by side, and small members all do.
Here every handle is in exact-assembly mode, whose K is solved as assembled, so the members wait in their
lanes for the batched launches.  The cases, twins and tolerances are test_batch.py's: FP64 members with one
and three lanes, mixed members with each FP32 kernel and with the tuner, paused and resumed solves, members
that join a running batch, tangent mode.

That the launches were shared shows in their number: a lane's members solve together, so a batch of several
members takes fewer launches than its members have solves (without a limit on a launch's iterations)."""
import pytest

import test_batch as TB
from _util import LPM, gpu_problem

pytestmark = pytest.mark.gpu


@pytest.fixture
def lanes(monkeypatch):
    """Exact-assembly handles in test_batch's tests; the statistics and members of its batches."""
    seen = []

    def exact(*args, **kw):
        g = gpu_problem(*args, **kw)
        g.set_assembly_exact(True)
        return g

    class Batch(LPM.Batch):
        def add(self, g, steps):
            mid = super().add(g, steps)
            self.mids = getattr(self, "mids", []) + [mid]
            return mid

        def remove(self, mid):
            self.removed = True
            super().remove(mid)

        def close(self):
            if not getattr(self, "removed", False):
                seen.append((self.stats(), [self.member(m) for m in self.mids]))
            super().close()

    monkeypatch.setattr(TB, "gpu_problem", exact)
    monkeypatch.setattr(TB.LPM, "Batch", Batch)
    return seen


def _shared(seen):
    (stats, members), = seen
    solves = sum(m["total"]["newton_solves"] for m in members)
    assert 0 < stats["cg_launches"] < solves, (stats["cg_launches"], solves)


@pytest.mark.parametrize("count", [1, 3])
def test_fp64_members(lanes, count):
    TB.test_batch_fp64_members_match_alone(count)
    _shared(lanes)


@pytest.mark.parametrize("count,kernel", [(1, None), (2, None), (1, "0"), (1, "1"), (1, "2"), (1, "3")])
def test_mixed_members(lanes, count, kernel, monkeypatch):
    TB.test_batch_mixed_members_match_fp64_alone(count, kernel, monkeypatch)
    if count == 1:
        _shared(lanes)


@pytest.mark.parametrize("precision,tol", [(0, TB.FP64_TOL), (1, TB.MIXED_TOL)])
def test_paused_solves(lanes, precision, tol, monkeypatch):
    TB.test_batch_paused_solves_resume(precision, tol, monkeypatch)
    (stats, members), = lanes
    # 7 iterations a launch: a member alone needs at least its iterations / 7 launches
    assert stats["cg_launches"] * 7 >= max(m["total"]["cg_iters"] for m in members)


@pytest.mark.parametrize("count", [1, 2])
def test_joining_members(lanes, count):
    TB.test_batch_members_join_while_others_run(count)


@pytest.mark.parametrize("precision,tol", [(0, TB.FP64_TOL), (1, TB.MIXED_TOL)])
def test_tangent_members(lanes, precision, tol):
    TB.test_batch_tangent_members_match_alone(precision, tol)
    _shared(lanes)
