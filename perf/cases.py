"""Workloads of the implicit quasi-static step, timed through the public entry points.

Every case is what a user's program does with this library, at a size that such a program has:

* ``newton``   one Newton iteration of a caller-driven loop on a deformed specimen: positions in,
               force state, stiffness, residual, linear solve, displacement increment out
* ``force``    the force state of a deformed specimen, with particle forces and stresses out (what an
               explicit or post-processing program calls per step)
* ``direct``   the Newton iteration with the band Cholesky solve (``SolverMode::PARDISO``'s role)
* ``noalloc``  the allocation-free CG on a block-CSR system that the caller holds on the device
* ``run``      a whole run from coordinates to final fields: problem set-up and every load step
* ``batch``    many notched plates of uneven size, set up and carried through their load paths
* ``fatigue``  a fatigue specimen: set-up, one static step, load cycles, final fields

The lattices are generated here, in the order of the reference's generators, so that inputs and the
64-bit values of ``exact`` do not depend on the library's own generators.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

LPM = importlib.import_module("lpm-cpp_b200.lpm")
CFG = importlib.import_module("lpm-cpp_b200.configs")

RADIUS = {"hex": 0.1, "sq": 0.1, "sc": 0.2, "fcc": 0.2, "bcc": 0.2}
LATTICE = {"sq": LPM.LatticeType.Square2D, "hex": LPM.LatticeType.Hexagon2D, "sc": LPM.LatticeType.SimpleCubic3D,
           "fcc": LPM.LatticeType.FCC3D, "bcc": LPM.LatticeType.BCC3D}
DIM = {"hex": 2, "sq": 2, "sc": 3, "fcc": 3, "bcc": 3}
PER_CELL = {"hex": 1, "sq": 1, "sc": 1, "fcc": 4, "bcc": 2}
BONDS = {"hex": 12, "sq": 8, "sc": 18, "fcc": 18, "bcc": 14}
CONNS = {"hex": 31, "sq": 17, "sc": 61, "fcc": 61, "bcc": 41}
# The stopping test of the linear solves: the squared-norm test at the level the parity tests of
# this repository use, so that a displacement increment is good to many digits.
TIGHT = {"cg_rtol": 1e-24, "cg_atol": 0.0}


# ------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest specimen of an interactive study: launch and barrier latency count
        {"name": "newton_hex_small", "kind": "newton", "lattice": "hex", "nx": 25, "ny": 29, "nz": 1, "mixed": False},
        # the 20 x 20 mm hexagonal plate of the isotropic-elasticity example
        {"name": "newton_hex_plate", "kind": "newton", "lattice": "hex", "nx": 100, "ny": 115, "nz": 1, "mixed": False},
        # the 20 mm simple-cubic cube of the benchmark (127,500 particles)
        {"name": "newton_sc_cube", "kind": "newton", "lattice": "sc", "nx": 51, "ny": 50, "nz": 50, "mixed": False},
        # near the top of the serving stream's range, mixed precision, odd sizes
        {"name": "newton_bcc_mixed", "kind": "newton", "lattice": "bcc", "nx": 61, "ny": 59, "nz": 57, "mixed": True},
        # forces and stresses of a mid-size cube
        {"name": "force_sc", "kind": "force", "lattice": "sc", "nx": 41, "ny": 40, "nz": 39},
        # the direct solve of the 10 x 10 mm plate
        {"name": "direct_hex", "kind": "direct", "lattice": "hex", "nx": 50, "ny": 58, "nz": 1},
        # a plugin that owns all device memory: a small plate and a 10 mm cube
        {"name": "noalloc_hex", "kind": "noalloc", "lattice": "hex", "nx": 31, "ny": 35, "nz": 1},
        {"name": "noalloc_sc", "kind": "noalloc", "lattice": "sc", "nx": 25, "ny": 25, "nz": 25},
        # single-crystal J2 bar, stiffness re-assembled before every Newton solve
        {"name": "run_fcc_tangent", "kind": "run", "model": "fcc_j2", "size": 5.0, "steps": 2, "mixed": False},
        # nonlocal elastic damage on a plate
        {"name": "run_hex_edamage", "kind": "run", "model": "edamage", "size": 8.0, "steps": 2, "mixed": False},
        # notched plates of uneven size in one batch, mixed precision
        {"name": "batch_plates", "kind": "batch", "count": 12, "side_max": 14.0, "steps": 3, "mixed": True},
        # the 25 mm high-cycle-fatigue plate: one static step and one load cycle of four steps
        {"name": "fatigue_plate", "kind": "fatigue", "size": 25.0, "cycles": 1},
    ]


def draw(rng):
    kind = rng.choice(["newton"] * 5 + ["force"] * 2 + ["direct", "noalloc", "noalloc", "run", "batch", "fatigue"])

    def cells(lattice, lo, hi):
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        d = DIM[lattice]
        side = (n / PER_CELL[lattice]) ** (1.0 / d)
        dims = [max(4, int(round(side * rng.uniform(0.85, 1.18)))) for _ in range(d)]
        return dict(zip(("nx", "ny", "nz"), dims + [1] * (3 - d)))

    if kind in ("newton", "force"):
        lattice = rng.choice(["hex", "sq", "sc", "fcc", "bcc"])
        c = {"kind": kind, "lattice": lattice, **cells(lattice, 500, 40000 if DIM[lattice] == 2 else 250000)}
        if kind == "newton":
            c["mixed"] = rng.random() < 0.5
        return c
    if kind == "direct":
        return {"kind": kind, "lattice": rng.choice(["hex", "sq"]), **cells("hex", 300, 4000)}
    if kind == "noalloc":
        lattice = rng.choice(["hex", "sq", "sc", "fcc", "bcc"])
        return {"kind": kind, "lattice": lattice, **cells(lattice, 300, 12000)}
    if kind == "run":
        model = rng.choice(["fcc_j2", "edamage", "elastic"])
        size = {"fcc_j2": rng.uniform(2.0, 5.0), "edamage": rng.uniform(2.0, 8.0), "elastic": rng.uniform(3.0, 10.0)}
        return {"kind": kind, "model": model, "size": round(size[model], 2), "steps": rng.randint(1, 2),
                "mixed": rng.random() < 0.3 and model == "elastic"}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 12), "side_max": round(rng.uniform(6.0, 14.0), 1),
                "steps": rng.randint(1, 3), "mixed": rng.random() < 0.5}
    return {"kind": kind, "size": round(rng.uniform(3.0, 25.0), 1), "cycles": 1}


# ------------------------------------------------------------------------------------ inputs
def _sites(lattice, nx, ny, nz):
    """Integer lattice coordinates (z slowest, x fastest) and the length of one unit along each axis."""
    r = RADIUS[lattice]
    if lattice == "hex":
        j, i = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
        ij = np.stack([2 * i + j % 2, j, 0 * i], -1).reshape(-1, 3)
        return ij, np.array([r, r * math.sqrt(3.0), 0.0])
    if lattice in ("sq", "sc"):
        k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        return np.stack([i, j, k], -1).reshape(-1, 3), np.array([2 * r, 2 * r, 2 * r if lattice == "sc" else 0.0])
    k, j, i = np.meshgrid(np.arange(2 * nz), np.arange(2 * ny), np.arange(2 * nx), indexing="ij")
    p = np.stack([i, j, k], -1).reshape(-1, 3)
    if lattice == "fcc":
        return p[(p.sum(1) % 2) == 0], np.full(3, 2 * r / math.sqrt(2.0))
    return p[((p[:, 0] % 2) == (p[:, 1] % 2)) & ((p[:, 1] % 2) == (p[:, 2] % 2))], np.full(3, 2 * r / math.sqrt(3.0))


def _specimen(case, seed):
    """Coordinates of a specimen, its deformed coordinates, constraints and material, from the seed."""
    lat, d = case["lattice"], DIM[case["lattice"]]
    rng = np.random.default_rng([seed, 17])
    sites, unit = _sites(lat, case["nx"], case["ny"], case["nz"])
    xyz = np.ascontiguousarray(sites * unit)
    E, mu, strain = float(rng.uniform(50e3, 250e3)), float(rng.uniform(0.2, 0.35)), float(rng.uniform(0.5e-3, 1.5e-3))
    up = d - 1  # the loading axis
    ext = xyz.max(0) + (xyz.max(0) == 0)
    grad = np.full(d, -mu * strain)
    grad[up] = strain
    now = xyz.copy()
    now[:, :d] += xyz[:, :d] * grad
    wave = rng.uniform(-1, 1, (4, d))
    phase = rng.uniform(0, 2 * math.pi, (4, d))
    for m in range(4):
        arg = (xyz[:, :d] / ext[:d] * rng.integers(1, 4, d)).sum(1, keepdims=True) * math.pi
        now[:, :d] += 0.01 * strain * ext[up] * wave[m] * np.sin(arg + phase[m])
    lo, hi = xyz[:, up] < 1e-9, xyz[:, up] > xyz[:, up].max() - 1e-9
    now[hi, up] += 0.1 * strain * ext[up]
    bottom, top = np.nonzero(lo)[0].astype(np.int32), np.nonzero(hi)[0].astype(np.int32)
    if d == 2:  # bottom edge fixed, top edge moved
        fixed = [(bottom, "x"), (bottom, "y"), (top, "y")]
    else:  # bottom face held in z with two corners pinned, top face moved
        b = xyz[bottom]
        c0 = bottom[np.lexsort((b[:, 1], b[:, 0]))[:1]]
        c1 = bottom[np.lexsort((b[:, 1], -b[:, 0]))[:1]]
        fixed = [(bottom, "z"), (c0, "x"), (c0, "y"), (c1, "y"), (top, "z")]
    return {"xyz": xyz, "now": now, "fixed": fixed, "E": E, "mu": mu, "sites": sites}


def _problem(case, s, precision):
    lat = case["lattice"]
    box = [float(v) for k in range(3) for v in (s["xyz"][:, k].min(), s["xyz"][:, k].max())]
    a = LPM.Assembly(s["xyz"], box, LPM.UnitCell(LATTICE[lat], RADIUS[lat]), LPM.ParticleType.Elastic)
    a.setParticleProperty(0.0, DIM[lat] == 2, s["E"], s["mu"], 1.0)
    p = LPM.GpuProblem(a, max_iter=30, tol_iter=1e-9, precision=precision, **TIGHT)
    hold = LPM.LoadStep([LPM.DispBC(g, LPM.LoadMode.Relative, f, 0.0) for g, f in s["fixed"]], [])
    p.apply_load_step(hold)
    return p


def _prepare_run(case, seed):
    """The specimen of a whole run: a configuration of the package with the seed's material."""
    rng = np.random.default_rng([seed, 23])
    scale = float(rng.uniform(0.8, 1.25))
    if case["model"] == "fcc_j2":
        c = CFG.fcc_bar(size=(case["size"], case["size"], 2 * case["size"]), radius=0.18, E=110e3 * scale, steps=50,
                        j2=(60.0 * 3.06 * float(rng.uniform(0.9, 1.1)), 0.0, 500.0, 0.0), tol_iter=1e-9)
    elif case["model"] == "edamage":
        c = CFG.edamage_plate(size=case["size"], E=69e3 * scale, steps=4, total_disp=0.008 * case["size"] / 2.4)
    else:
        c = CFG.sc_cube(size=case["size"], E=2e5 * scale, mu=float(rng.uniform(0.2, 0.3)), steps=20, tol_iter=1e-9)
    return {"case": c, "opt": dict(undamaged_pt_type=c.undamaged_type, max_iter=c.max_iter, tol_iter=c.tol_iter,
                                   tangent=case["model"] == "fcc_j2", **TIGHT)}


def prepare(case, seed):
    kind = case["kind"]
    precision = LPM.Precision.MIXED if case.get("mixed") else LPM.Precision.FP64
    if kind in ("newton", "force", "direct"):
        s = _specimen(case, seed)
        return {"kind": kind, "p": _problem(case, s, precision), "now": s["now"]}
    if kind == "noalloc":
        s = _specimen(case, seed)
        rowptr, col, val, b = _bsr(case, s)
        i32 = dict(dtype=torch.int32, device="cuda")
        return {"kind": kind, "dim": DIM[case["lattice"]], "n": len(s["xyz"]), "rowptr": rowptr.to(**i32),
                "col": col.to(**i32), "val": val.cuda(), "b": b.cuda(), "x": torch.zeros_like(b, device="cuda")}
    if kind == "run":
        return {"kind": kind, "steps": case["steps"], "precision": precision, **_prepare_run(case, seed)}
    if kind == "batch":
        cases = CFG.batched_notched_plates(count=case["count"], steps=case["steps"], side=(4.0, case["side_max"]),
                                           opening=0.3, tol_iter=1e-8)
        rng = np.random.default_rng([seed, 31])
        for c in cases:  # the geometry of the workload; stiffness, strength and opening from the seed
            tough = float(rng.uniform(0.8, 1.2))
            c.material.E *= float(rng.uniform(0.8, 1.25))
            c.material.critical_bstrain *= tough
            c.steps = [([(g, f, v * tough) for g, f, v in disp], force) for disp, force in c.steps]
        return {"kind": kind, "cases": cases, "precision": precision}
    rng = np.random.default_rng([seed, 29])
    c = CFG.fatigue_plate(size=case["size"], E=69e3 * float(rng.uniform(0.8, 1.25)), cycles=2 * case["cycles"],
                          amplitude=0.004 * case["size"] / 2.4)
    fat = c.meta["fatigue"]
    groups = [c.groups[g] for g in fat["groups"]]
    cycles = [LPM.generateLoadCycle(LPM.FatigueLoadType.LoadUniaxialDisp, fat["spectrum"], k, fat["n_interval"], groups)
              for k in range(case["cycles"])]
    return {"kind": kind, "case": c, "cycles": cycles, "dndt": 2.0}


# ------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "newton":
        p = state["p"]
        p.set_xyz(state["now"])
        p.update_force_state()
        p.assemble(True)
        p.update_rr()
        disp, _ = p.solve_linear()
        return {"disp": disp, "residual": p.residual()}
    if kind == "force":
        p = state["p"]
        p.set_xyz(state["now"])
        p.update_force_state()
        return p.state(("pin", "stress"))
    if kind == "direct":
        p = state["p"]
        p.set_xyz(state["now"])
        p.update_force_state()
        p.assemble(True)
        p.update_rr()
        disp, _ = p.solve_direct()
        return {"disp": disp, "residual": p.residual()}
    if kind == "noalloc":
        ptr = [ctypes.c_void_p(state[k].data_ptr()) for k in ("rowptr", "col", "val", "b", "x")]
        it = ctypes.c_int64(0)
        status = LPM.lib().lpmgpu_cg_bsr_noalloc(state["dim"], state["n"], *ptr, TIGHT["cg_rtol"], TIGHT["cg_atol"], 0,
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                                 ctypes.byref(it))
        if status != LPM.OK:
            raise LPM.LpmGpuError(status, "lpmgpu_cg_bsr_noalloc")
        return state["x"]
    if kind == "run":
        c = state["case"]
        p = LPM.GpuProblem(c.assembly(), precision=state["precision"], **state["opt"])
        for s in range(state["steps"]):
            ok, _ = p.solve_load_step(c.load_step(s))
            if not ok:
                raise RuntimeError("load step did not converge")
        out = p.state(("xyz", "pin", "stress", "state_var"))
        p.close()
        return out
    if kind == "batch":
        problems = [LPM.GpuProblem(c.assembly(), undamaged_pt_type=c.undamaged_type, max_iter=c.max_iter,
                                   tol_iter=c.tol_iter, precision=state["precision"], **TIGHT) for c in state["cases"]]
        batch = LPM.Batch()
        for p, c in zip(problems, state["cases"]):
            batch.add(p, [c.load_step(s) for s in range(len(c.steps))])
        batch.run()
        out = [p.state(("xyz",))["xyz"] for p in problems]
        batch.close()
        for p in problems:
            p.close()
        return out
    c = state["case"]
    p = LPM.GpuProblem(c.assembly(), undamaged_pt_type=c.undamaged_type, max_iter=c.max_iter, tol_iter=c.tol_iter,
                       **TIGHT)
    p.fatigue_static_step(c.load_step(0))
    for steps in state["cycles"]:
        p.fatigue_cycle(steps, state["dndt"])
    out = p.state(("xyz", "stress", "damage", "state_var"))
    p.close()
    return out


# ------------------------------------------------------------------------------------ work
def _particles(case):
    kind = case["kind"]
    if "nx" in case:
        return PER_CELL[case["lattice"]] * case["nx"] * case["ny"] * case["nz"]
    if kind == "run":
        return {"fcc_j2": 2 * case["size"] ** 3 / (8 * 0.18 ** 3 / math.sqrt(2.0)),
                "edamage": 29 * case["size"] ** 2, "elastic": (case["size"] / 0.4) ** 3}[case["model"]]
    if kind == "batch":
        lo, hi = 4.0, case["side_max"]
        return case["count"] * 29 * (hi * hi - lo * lo) / (2 * math.log(hi / lo))
    return 29 * case["size"] ** 2


def work(case):
    """What one pass cannot do without: positions in and fields out once, the bond list once per force
    state, and per CG iteration the arithmetic of the bond-wise stiffness product (about 14 operations
    per bond and dimension) plus the vector updates.  The iteration counts follow the specimen's length in
    particles (an unpreconditioned CG needs a multiple of it); for the caller's block-CSR matrix the
    arithmetic is the matrix's own."""
    kind, n = case["kind"], _particles(case)
    lat = case.get("lattice") or {"fcc_j2": "fcc", "elastic": "sc"}.get(case.get("model"), "hex")
    d, nb = DIM[lat], BONDS[lat]
    side = n ** (1.0 / d) if kind != "batch" else (n / case["count"]) ** 0.5
    iters = (26.0 if d == 2 else 24.0) * side
    state = n * (nb * 4 + nb * 8 + 60)
    if kind == "force":
        return {"bytes": state + n * 72, "flops": n * nb * 60}
    if kind == "noalloc":
        nnz = n * CONNS[lat] * d * d
        return {"bytes": nnz * 8 + n * (CONNS[lat] * 4 + 16 * d), "flops": iters * (2 * nnz + 10 * n * d)}
    solve = iters * n * (14 * nb * d + 10 * d)
    if kind == "direct":
        band = 2 * math.sqrt(n) * d + d
        return {"bytes": state + n * 16 * d, "flops": n * d * (band * band + 4 * band)}
    solves = {"newton": 1, "run": 3 * case.get("steps", 1), "batch": 8 * case.get("steps", 1), "fatigue": 10}[kind]
    return {"bytes": state + n * 16 * d, "flops": solves * (solve + n * nb * 60)}


# ------------------------------------------------------------------------------------ 64-bit values
def _kntv(lat, E, mu):
    """Bond coefficients Kn, Tv per layer of the isotropic elastic particle (plane stress in 2D)."""
    r, s2, s3 = RADIUS[lat], math.sqrt(2.0), math.sqrt(3.0)
    if DIM[lat] == 2:
        Ce = np.array([E / (1 - mu * mu), mu * E / (1 - mu * mu), E / 2 / (1 + mu)])
    else:
        Ce = np.array([E * (1 - mu), E * mu, E * (1 - 2 * mu) / 2]) / ((1 + mu) * (1 - 2 * mu))
    m = {"sq": [[.5, -.5, 0], [0, 0, .5], [0, 1 / 12, -1 / 12]],
         "hex": [[s3 / 12, -s3 / 12, 0], [-s3 / 144, s3 / 48, 0], [0, 0, 1]],
         "sc": [[1, -1, -1], [0, 0, 1], [0, 1 / 18, -1 / 18]],
         "fcc": [[0, 0, s2], [s2 / 4, -s2 / 4, -s2 / 4], [0, s2 / 24, -s2 / 24]],
         "bcc": [[0, 0, s3], [1 / s3, -1 / s3, 0], [0, s3 / 14, s3 / 14]]}[lat]
    k = (np.array(m) @ Ce) * (1.0 if DIM[lat] == 2 else r)
    return ([k[0], k[0]], [k[1], k[1]]) if lat == "hex" else ([k[0], k[1]], [k[2], k[2]])


_AX = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
_DIAG = [(1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1)]
_HALF = {"hex": ([(2, 0, 0), (1, 1, 0), (-1, 1, 0)], [(3, 1, 0), (-3, 1, 0), (0, 2, 0)]),
         "sq": ([(1, 0, 0), (0, 1, 0)], [(1, 1, 0), (1, -1, 0)]),
         "sc": (_AX, _DIAG), "fcc": (_DIAG, [(2, 0, 0), (0, 2, 0), (0, 0, 2)]),
         "bcc": ([(1, 1, 1), (1, 1, -1), (1, -1, 1), (-1, 1, 1)], [(2, 0, 0), (0, 2, 0), (0, 0, 2)])}


class _Model:
    """The linear-elastic lattice of a deformed specimen in 64-bit torch: bonds, forces and the
    bond-wise product with the stiffness of the current state."""

    def __init__(self, case, s, device):
        lat = case["lattice"]
        self.d = DIM[lat]
        sites = s["sites"] + 4
        table = np.full(sites.max(0) + 5, -1, np.int64)
        table[tuple(sites.T)] = np.arange(len(sites))
        kn, tv = _kntv(lat, s["E"], s["mu"])
        f64 = dict(dtype=torch.float64, device=device)
        x0, x = torch.as_tensor(s["xyz"]).to(**f64), torch.as_tensor(s["now"]).to(**f64)
        self.n, self.layers = len(sites), []
        for L in (0, 1):
            i, j = [], []
            for o in _HALF[lat][L]:
                for sign in (1, -1):
                    k = table[tuple((sites + sign * np.array(o)).T)]
                    i.append(np.nonzero(k >= 0)[0])
                    j.append(k[k >= 0])
            i, j = (torch.as_tensor(np.concatenate(v)).to(device) for v in (i, j))
            dx = x[i] - x[j]
            dis = dx.norm(dim=1)
            dl = dis - (x0[i] - x0[j]).norm(dim=1)
            self.layers.append((i, j, dx / dis[:, None], dis, dl, float(kn[L]), float(tv[L])))
        held = torch.zeros(self.n, 3, dtype=torch.bool, device=device)
        for ids, axis in s["fixed"]:
            held[torch.as_tensor(ids.astype(np.int64)).to(device), "xyz".index(axis)] = True
        self.free = (~held[:, :self.d]).to(torch.float64)

    def _sum(self, i, v):
        return torch.zeros((self.n,) + tuple(v.shape[1:]), dtype=v.dtype, device=v.device).index_add_(0, i, v)

    def forces(self, r, nneigh, pvol):
        pin = stress = 0
        count = sum(self._sum(b[0], torch.ones_like(b[3])) for b in self.layers)
        for i, j, c, dis, dl, kn, tv in self.layers:
            th = self._sum(i, dl)
            f = 2 * kn * dl + tv * (th[i] + th[j])  # half the sum of the two directed bonds' forces
            pin = pin + self._sum(i, c * f[:, None])
            w = (0.5 * dis * f / (pvol * count[i] / nneigh))[:, None]
            cc = torch.stack([c[:, 0] ** 2, c[:, 1] ** 2, c[:, 2] ** 2, c[:, 1] * c[:, 2], c[:, 0] * c[:, 2],
                              c[:, 0] * c[:, 1]], 1)
            stress = stress + self._sum(i, w * cc)
        return pin, stress

    def product(self, u):
        """K u for u of shape (n, d), constrained rows and columns left out."""
        u = u * self.free
        out = 0
        for i, j, c, dis, dl, kn, tv in self.layers:
            c = c[:, :self.d]
            e = (c * (u[i] - u[j])).sum(1)
            th = self._sum(i, e)
            out = out + self._sum(i, c * (tv * (th[i] + th[j]) + 2 * kn * e)[:, None])
        return out * self.free

    def solve(self, b):
        x, r = torch.zeros_like(b), b.clone()
        p, rr = r.clone(), (r * r).sum()
        stop = float(rr) * 1e-30
        for it in range(20 * self.n):
            q = self.product(p)
            a = rr / (p * q).sum()
            x += a * p
            r -= a * q
            rn = (r * r).sum()
            if it % 25 == 0 and float(rn) <= stop:
                break
            p = r + (rn / rr) * p
            rr = rn
        return x


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _bsr(case, s):
    """The specimen's stiffness as a block-CSR matrix with the constraints eliminated (unit-scaled
    diagonal), and the residual: what the plugin of the ``noalloc`` cases holds."""
    m = _Model(case, s, _device())
    d, n = m.d, m.n
    keys, blocks = [], []

    def add(i, j, v):
        keys.append(i * n + j)
        blocks.append(v.reshape(-1, d * d))

    for i, j, c, dis, dl, kn, tv in m.layers:
        c = c[:, :d]
        cc = c[:, :, None] * c[:, None, :]
        add(i, i, 2 * kn * cc)
        add(i, j, -2 * kn * cc)
        # theta_k = S_k . u_k - sum_b c_b . u_j(b): its outer product over particle k and its neighbours
        S = m._sum(i, c)
        order = torch.argsort(i, stable=True)
        io, jo, co = i[order], j[order], c[order]
        cnt = torch.bincount(io, minlength=n)
        start = torch.cumsum(cnt, 0) - cnt
        width = int(cnt.max())
        ids = torch.full((n, width + 1), -1, dtype=torch.int64, device=i.device)
        g = torch.zeros(n, width + 1, d, dtype=torch.float64, device=i.device)
        ids[:, 0] = torch.arange(n, device=i.device)
        g[:, 0] = S
        slot = torch.arange(len(io), device=i.device) - start[io] + 1
        ids[io, slot] = jo
        g[io, slot] = -co
        for a in range(width + 1):
            for b in range(width + 1):
                ok = (ids[:, a] >= 0) & (ids[:, b] >= 0)
                add(ids[ok, a], ids[ok, b], tv * g[ok, a, :, None] * g[ok, b, None, :])
    key, inv = torch.unique(torch.cat(keys), return_inverse=True)
    val = torch.zeros(len(key), d * d, dtype=torch.float64, device=key.device).index_add_(0, inv, torch.cat(blocks))
    row, col = key // n, key % n
    val = (val.reshape(-1, d, d) * m.free[row][:, :, None] * m.free[col][:, None, :])
    diag = torch.diagonal(val[row == col], dim1=1, dim2=2)
    norm = float(diag.norm())
    val[row == col] += torch.diag_embed((1 - m.free) * norm)
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=key.device)
    rowptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    pin, _ = m.forces(RADIUS[case["lattice"]], 1.0, 1.0)
    return rowptr, col, val.reshape(-1).contiguous(), (-pin[:, :d] * m.free).reshape(-1).contiguous()


def exact(case, seed):
    if "nx" not in case:  # whole runs: plasticity, damage and fatigue paths have no closed 64-bit value
        return None
    s = _specimen(case, seed)
    m = _Model(case, s, _device())
    lat, r = case["lattice"], RADIUS[case["lattice"]]
    pvol = {"sq": 4 * r * r, "hex": 2 * math.sqrt(3.0) * r * r, "sc": 8 * r ** 3, "fcc": 4 * math.sqrt(2.0) * r ** 3,
            "bcc": 32 * math.sqrt(3.0) / 9 * r ** 3}[lat]
    pin, stress = m.forces(r, BONDS[lat], pvol)
    if case["kind"] == "force":
        return {"pin": pin, "stress": stress}
    res = -pin[:, :m.d] * m.free
    x = m.solve(res).reshape(-1)
    return x if case["kind"] == "noalloc" else {"disp": x, "residual": res.reshape(-1)}
