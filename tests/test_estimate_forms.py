"""The admission estimate (lpmgpu_estimate_bytes) counts the bond form of K where a problem has one.

Host arithmetic, no device: elastic and J2 particles have the form, elastic-damage and fatigue particles do
not, and 3D mixed precision only up to the size that one cluster may hold.  A request without it must not be
refused for memory that it does not take.  On the device: the estimate is no less than what the problem
holds, for every kind."""
import ctypes as C

import pytest

from _util import CFG, LPM, gpu_problem, hetero_plate
from test_bond_form import _block

P, L = LPM.ParticleType, LPM.LatticeType
# per lattice: bonds and dimensions as the estimate takes them
SHAPE = {L.Square2D: (8, 2), L.Hexagon2D: (12, 2), L.SimpleCubic3D: (18, 3), L.FCC3D: (18, 3), L.BCC3D: (14, 3)}


def _estimate(lattice, n, ptype, precision, per_bond=False):
    d = LPM.Desc()
    d.lattice, d.n, d.ptype, d.precision, d.radius = int(lattice), n, int(ptype), precision, 0.1
    one = (C.c_double * 1)(1.0)
    if per_bond:
        d.bond_kn = C.cast(one, C.POINTER(C.c_double))
    out = C.c_int64()
    assert LPM.lib().lpmgpu_estimate_bytes(C.byref(d), C.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("per_bond", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("lattice", list(SHAPE))
def test_form_is_counted_where_it_exists(lattice, precision, per_bond):
    nb, dim = SHAPE[lattice]
    rows = 4 * dim + dim * (dim + 1) // 2
    for n in (1000, 15872, 15873, 400000):
        base = _estimate(lattice, n, P.ElasticDamage, precision, per_bond)
        assert base == _estimate(lattice, n, P.FatigueHCF, precision, per_bond)
        form = (nb + 8) * (8 + 8 * dim + 16 * per_bond) + 36 + 8 * rows * per_bond
        if precision and dim == 2:
            form += (nb + 8) * (4 * dim + 8 * per_bond) + 16 + 4 * rows * per_bond
        if precision and dim == 3 and n > 15872:
            form = 0
        for ptype in (P.Elastic, P.J2Plasticity):
            assert _estimate(lattice, n, ptype, precision, per_bond) - base == n * form


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", ["hex", "hex_large", "square", "sc", "fcc", "bcc_large", "hetero", "edamage"])
def test_estimate_covers_the_problem(which, precision):
    case = {"hex": lambda: _block(L.Hexagon2D, 6.0), "hex_large": lambda: _block(L.Hexagon2D, 25.0),
            "square": lambda: _block(L.Square2D, 8.3), "sc": lambda: _block(L.SimpleCubic3D, 4.4),
            "fcc": lambda: _block(L.FCC3D, 7.0), "bcc_large": lambda: _block(L.BCC3D, 12.0),
            "hetero": lambda: hetero_plate(size=4.0), "edamage": lambda: CFG.edamage_plate()}[which]()
    g = gpu_problem(case, precision=precision)
    held = g.sizes["device_bytes"]
    g.close()
    d, keep = LPM._pack_desc(case.assembly(), precision=LPM.Precision(precision))
    est = C.c_int64()
    assert LPM.lib().lpmgpu_estimate_bytes(C.byref(d), C.byref(est)) == 0
    assert est.value >= held > 0
