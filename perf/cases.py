"""Performance cases of the solver step, through the entry points that programs call.

Each case is one pass of a real use: a schedule period (or a page's frames) of one of the solvers
plus the readout that a host takes after it, from the state the pass before left.

  sp        ``Context(flavor="solver.py")``: one 100-step schedule period, then the energies
  new       ``Context(flavor="new")``: 20 imaginary-time steps (five V-cycles), then the energies
  evaluate  ``autograd.EnergyModel``: one energy-and-force evaluation of a geometry step -- moved
            nuclei, warm-started iterations, energy, adjoint forces through them
  batch     ``Batch``: 20 steps of many uneven instances, energies and forces of all
  mj        ``Context(flavor="molecule.js")``: one frame of the page, energies and forces
  lobpcg    the same page's LOBPCG frames
  mf        ``MolFast``: one drawn frame (steps, forces, nuclear move) and its fields
  rb        ``RealqmRb``: the steps between two readouts, energies and fields
  shells    ``AtomShells``: physics steps, energies and fields

Geometries, seeds of the electron domains and starting fields come from the case's seed.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from realmolecule_b200 import Context, _lib as L, configs
from realmolecule_b200.autograd import EnergyModel
from realmolecule_b200.batch import Batch
from realmolecule_b200.mol_fast import MolFast
from realmolecule_b200.realqm_rb import RealqmRb
from realmolecule_b200.shells import AtomShells

DENSE = 27.2  # edge in bohr of the cube that holds 100 waters at 1 g/cm^3


def listed():
    return [
        # the benchmark's headline workload: glycine in the reference's all-electron idiom
        {"name": "sp_glycine128", "kind": "sp", "NN": 128, "h": 0.2, "waters": 0},
        # the reference's large jobs: a few hundred atoms on a 300^3 grid (bandwidth-bound)
        {"name": "sp_255atoms_300", "kind": "sp", "NN": 300, "h": 0.2, "waters": 85},
        # the smallest: one water in plain FP64
        {"name": "new_water64_fp64", "kind": "new", "NN": 64, "h": 0.25, "waters": 1, "precision": "fp64"},
        # one molecule in mixed precision
        {"name": "new_glycine128_mixed", "kind": "new", "NN": 128, "h": 0.2, "waters": 0, "precision": "mixed"},
        # one step of a FIRE relaxation of 100 waters: 200 iterations forward and back
        {"name": "evaluate_water100_192", "kind": "evaluate", "NN": 192, "h": 0.2, "waters": 100, "iters": 200},
        # one step of the dynamics of 1000 waters: 50 iterations forward and back
        {"name": "evaluate_water1000_320", "kind": "evaluate", "NN": 320, "h": 0.2, "waters": 1000, "iters": 50},
        # throughput: 96 uneven water clusters stepped together
        {"name": "batch_clusters96", "kind": "batch", "n": 96, "precision": "mixed"},
        # a molecule.js page: water with its per-electron Poisson, a 50-step frame
        {"name": "mj_water64", "kind": "mj", "NN": 64, "screen": 16.0, "frames": 1, "steps": 50, "sic": 1},
        # the same page under its 'L' solver
        {"name": "lobpcg_water64", "kind": "lobpcg", "NN": 64, "screen": 16.0, "frames": 5, "steps": 10, "sic": 0},
        # mol_fast.js's CH4 page, a whole drawn frame
        {"name": "mf_ch4_200", "kind": "mf", "NN": 200, "screen": 12.0, "hydrogens": 4, "steps": 500},
        # realqm_rb.js's H2 page
        {"name": "rb_h2_100", "kind": "rb", "NN": 100, "screen": 8.0, "nuclei": 2, "ne": 1, "steps": 100},
        # atom.js's He page: two half-space shells with the multigrid Poisson solve
        {"name": "shells_he_100", "kind": "shells", "NN": 100, "shells": 2, "split": True, "poisson": "multigrid",
         "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _waters_that_fit(NN, h):
    return max(1, int(100 * max(0.0, (NN * h - 8.0) / DENSE) ** 3))


def _mg_grid(rng, lo, hi):
    """An NN that halves down to a coarsest level of 6..11 intervals."""
    while True:
        NN = rng.choice((6, 7, 8, 9, 10, 11)) << rng.randint(2, 5)
        if lo <= NN <= hi:
            return NN


def draw(rng):
    kind = rng.choice(("sp", "new", "evaluate", "batch", "mj", "lobpcg", "mf", "rb", "shells"))
    c = {"kind": kind}
    if kind == "sp":
        NN = 2 * _log(rng, 12, 150)
        h = rng.choice((0.2, 0.25, 0.3))
        c.update(NN=NN, h=h, waters=rng.randint(1, min(85, _waters_that_fit(NN, h))))
    elif kind == "new":
        NN = _mg_grid(rng, 32, 192)
        h = rng.choice((0.2, 0.25))
        c.update(NN=NN, h=h, waters=rng.randint(1, min(100, _waters_that_fit(NN, h))),
                 precision=rng.choice(("mixed", "fp64")))
    elif kind == "evaluate":
        NN = _mg_grid(rng, 40, 192)
        c.update(NN=NN, h=0.2, waters=rng.randint(1, min(100, _waters_that_fit(NN, 0.2))), iters=_log(rng, 10, 200))
    elif kind == "batch":
        c.update(n=_log(rng, 2, 96), precision=rng.choice(("mixed", "mixed", "fp64")))
        if c["precision"] == "fp64":
            c["n"] = min(c["n"], 40)
    elif kind == "mj":
        c.update(NN=2 * rng.randint(16, 50), screen=rng.choice((12.0, 16.0)), frames=1, steps=rng.choice((10, 25, 50)),
                 sic=rng.randint(0, 1))
    elif kind == "lobpcg":
        c.update(NN=2 * rng.randint(16, 50), screen=rng.choice((12.0, 16.0)), frames=rng.randint(2, 5), steps=10,
                 sic=rng.randint(0, 1))
    elif kind == "mf":
        c.update(NN=2 * _log(rng, 16, 100), screen=12.0, hydrogens=rng.randint(1, 4), steps=rng.choice((50, 120, 500)))
    elif kind == "rb":
        nuclei, ne = rng.randint(2, 3), rng.randint(1, 2)
        c.update(NN=_log(rng, 24, 150), screen=8.0, nuclei=nuclei, ne=ne, steps=_log(rng, 10, 100))
    else:
        c.update(NN=2 * _log(rng, 10, 50), shells=rng.randint(1, 4), split=False,
                 poisson=rng.choice(("multigrid", "multigrid", "simultaneous")), steps=_log(rng, 2, 10))
        if c["shells"] == 2:
            c["split"] = bool(rng.randint(0, 1))
    return c


# ---- geometries ---------------------------------------------------------------------------
def _water_cube(n, rng):
    """n rigid waters of random orientation at 1 g/cm^3: the cells of a cubic lattice, jittered."""
    m = int(math.ceil(n ** (1 / 3) - 1e-9))
    edge = DENSE * (n / 100.0) ** (1 / 3)
    s = edge / m
    cells = np.array([(a, b, c) for a in range(m) for b in range(m) for c in range(m)], np.float64)
    cells = cells[rng.permutation(len(cells))[:n]]
    O = (cells + 0.5) * s - edge / 2 + rng.uniform(-0.08, 0.08, (n, 3)) * s
    xyz = np.concatenate([configs.water_bohr(configs.random_rotation(rng)) + o for o in O])
    return ["O", "H", "H"] * n, xyz - xyz.mean(0)


def _geometry(c, seed):
    rng = np.random.default_rng(seed)
    if c["waters"]:
        el, xyz = _water_cube(c["waters"], rng)
    else:
        el, xyz = configs.glycine_bohr()
        xyz = (xyz - xyz.mean(0)) @ configs.random_rotation(rng).T
    g = configs.Geometry("", el, xyz, c["NN"], c["h"])
    g.seeds, g.seed_owner = configs.electron_seeds(el, xyz, rng)
    return g


def _moved(g, seed):
    """The positions a geometry step evaluates: nuclei moved by a few hundredths of a bohr."""
    return g.xyz + np.random.default_rng(seed + 1).normal(0.0, 0.02, g.xyz.shape)


def _cluster_geometries(c, seed):
    """Water clusters of 1-12 molecules, O-O at least 2.7 angstrom apart inside a sphere, on grids that
    hold the sphere and 6 bohr; the counts and grids belong to the case, the places to the seed."""
    counts = np.random.default_rng(c["n"]).integers(1, 13, c["n"])
    rng = np.random.default_rng(seed)
    out = []
    for n in map(int, counts):
        radius = 2.0 * configs.ANG * n ** (1 / 3) + 1.0
        el, xyz = configs.water_box(n, radius, 2.7, rng, sphere=True)
        NN = 64 if n == 1 else min(128, int(math.ceil((2 * radius + 12.0) / 0.25 / 16) * 16))
        g = configs.Geometry("", el, xyz, NN, 0.25)
        g.seeds, g.seed_owner = configs.electron_seeds(el, xyz, rng)
        out.append(g)
    return out


def _mj_atoms(c, seed):
    """Water in the page's idiom (an O core of 0.4 bohr), randomly turned, on whole grid points."""
    rng = np.random.default_rng(seed)
    h, mid = c["screen"] / c["NN"], c["NN"] // 2
    xyz = configs.water_bohr(configs.random_rotation(rng)) / h
    return [{"i": mid + int(round(p[0])), "j": mid + int(round(p[1])), "k": mid + int(round(p[2])), "Z": z, "Z_nuc": z,
             "rc": 0.4 if z == 6 else 0.0} for p, z in zip(xyz, (6, 1, 1))]


def _mf_page(c, seed):
    """The CH4 page with its first hydrogens, the molecule turned at random."""
    rng = np.random.default_rng(seed)
    N, h = c["NN"], c["screen"] / c["NN"]
    s2, s6 = math.sqrt(2), math.sqrt(6)
    d = np.array([(1, 0, 0), (-1 / 3, 2 * s2 / 3, 0), (-1 / 3, -s2 / 3, s6 / 3), (-1 / 3, -s2 / 3, -s6 / 3)])
    pos = N / 2 + 2.054 / h * (d @ configs.random_rotation(rng).T)[:c["hydrogens"]]
    nuc = [{"i": N / 2, "j": N / 2, "k": N / 2, "Z": 4, "rc": 0.5}]
    nuc += [{"i": float(p[0]), "j": float(p[1]), "k": float(p[2]), "Z": 1, "rc": 0.0} for p in pos]
    return {"nuclei": nuc, "NN": N, "screen": c["screen"], "norm_targets": [4] + [1] * c["hydrogens"],
            "steps_per_frame": c["steps"], "max_steps": 1 << 30, "dynamics": True}


def _rb_nuclei(c, seed):
    """Hydrogen-like nuclei 1.4 bohr apart along i (three: a bent chain), off the grid points."""
    rng = np.random.default_rng(seed)
    h, mid = c["screen"] / c["NN"], c["NN"] // 2
    place = [(-0.7, 0.0, 0.0), (0.7, 0.0, 0.0), (0.0, 1.2, 0.0)][:c["nuclei"]]
    off = rng.uniform(-0.4, 0.4, (len(place), 3))
    return [{"i": mid + p[0] / h + float(o[0]), "j": mid + p[1] / h + float(o[1]), "k": mid + p[2] / h + float(o[2]),
             "Z": c["ne"], "rc": 0, "ne": c["ne"]} for p, o in zip(place, off)]


def _shell_list(c):
    if c["split"]:
        return [{"ne": 1, "Rmax": 5.0, "Zeff": 2, "split": "halfspace", "halfIndex": q, "fixedW": True} for q in (0, 1)]
    r = (1.0, 2.0, 3.0, 5.0)
    return [{"ne": 1, "Rmax": 5.0 if q == c["shells"] - 1 else r[q], "Zeff": 2.0 / (q + 1)} for q in range(c["shells"])]


# ---- device views and kept host buffers ------------------------------------------------------
class _Device:
    """A context's device buffer, for torch (no copy); a tensor made from it keeps the context."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _views(state, names):
    """The context's live fields as torch tensors (made once per buffer)."""
    ctx = state["ctx"]
    inf = ctx.info()
    real = "<f8" if inf.precision == L.PREC_FP64 else "<f4"
    types = {"psi": real, "P": real, "label": "<i4", "W": "<f4"}
    out = {}
    for q in names:
        ptr = getattr(inf, q)
        if (ptr, q) not in state["views"]:
            S = inf.S
            state["views"][ptr, q] = torch.as_tensor(_Device(ctx, ptr, (S, S, S), types[q]), device="cuda")
        out[q] = state["views"][ptr, q]
    return out


def _host_buffers(n, S3):
    """Pinned buffers a host keeps for the fields it reads back (U, W, P of every electron)."""
    return torch.empty((n, 3, S3), dtype=torch.float32, pin_memory=True)


def _read_fields(download, handle, buf):
    for m in range(buf.shape[0]):
        st = download(handle, m, *(ctypes.c_void_p(buf[m, q].data_ptr()) for q in range(3)))
        if st:
            raise RuntimeError(f"field download failed: {st}")
    return buf


# ---- prepare and run -----------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "sp":
        g = _geometry(c, seed)
        ctx = Context(g.NN, g.screen, configs.to_reference_atoms(g), flavor="solver.py")
        ctx.initialize()
        return {"kind": kind, "ctx": ctx, "views": {}}
    if kind == "new":
        g = _geometry(c, seed)
        ctx = Context(g.NN, g.screen, configs.to_domain_atoms(g), flavor="new", precision=c["precision"], label_until=1)
        ctx.initialize()
        return {"kind": kind, "ctx": ctx, "views": {}}
    if kind == "evaluate":
        g = _geometry(c, seed)
        off = (g.NN // 2) * g.h
        model = EnergyModel(g.NN, g.h, g.charges, g.xyz + off, g.seeds + off, precision="mixed", tol=None,
                            warm_steps=c["iters"], label_until=1)
        return {"kind": kind, "model": model, "ctx": model.ctx, "x": _moved(g, seed) + off, "views": {}}
    if kind == "batch":
        inst = [{"NN": g.NN, "screen": g.screen, "atoms": configs.to_domain_atoms(g)}
                for g in _cluster_geometries(c, seed)]
        b = Batch(inst, precision=c["precision"], label_until=1)
        b.initialize()
        return {"kind": kind, "batch": b}
    if kind in ("mj", "lobpcg"):
        ctx = Context(c["NN"], c["screen"], _mj_atoms(c, seed), flavor="molecule.js", steps_per_frame=c["steps"],
                      sic=c["sic"], lobpcg=1 if kind == "lobpcg" else 0)
        ctx.initialize()
        return {"kind": kind, "ctx": ctx, "views": {}, "n": c["frames"] * (1 if kind == "lobpcg" else c["steps"])}
    if kind == "mf":
        mf = MolFast(**_mf_page(c, seed))
        return {"kind": kind, "mf": mf, "buf": _host_buffers(mf.n, mf.S3)}
    if kind == "rb":
        nuc = _rb_nuclei(c, seed)
        rb = RealqmRb(nuc, NN=c["NN"], screen=c["screen"], max_steps=1 << 30)
        return {"kind": kind, "rb": rb, "n": c["steps"], "buf": _host_buffers(rb.nelec, rb.S3)}
    # atom.js: the page's initial state with the amplitudes of a run some steps on (a few per cent off)
    sh = AtomShells(c["NN"], 5.0, 2.0, _shell_list(c), d=0.15, poisson=c["poisson"])
    rng = np.random.default_rng(seed)
    for m in range(sh.n_shells):
        U = sh.fields(m)["U"]
        sh.set_fields(m, U=U * (1.0 + 0.03 * rng.uniform(-1.0, 1.0, U.shape)).astype(np.float32))
    return {"kind": kind, "sh": sh, "n": c["steps"], "buf": _host_buffers(sh.n_shells, sh.S3)}


def run(state):
    kind = state["kind"]
    if kind == "sp":
        state["ctx"].step(100)
        e = state["ctx"].energy()
        return {"energy": e, **_views(state, ("psi", "P", "label"))}
    if kind == "new":
        state["ctx"].step(20)
        e = state["ctx"].energy()
        return {"energy": e, **_views(state, ("psi", "P", "label"))}
    if kind == "evaluate":
        E, F, _ = state["model"].evaluate(state["x"])
        return {"E": E, "F": F, **_views(state, ("psi", "P"))}
    if kind == "batch":
        b = state["batch"]
        b.step(20)
        return {"energy": b.energy(), "F": np.concatenate(b.forces())}
    if kind in ("mj", "lobpcg"):
        ctx = state["ctx"]
        if kind == "lobpcg":
            ctx.initialize()  # the page's 'L' run is a fresh start: its frames are the first ones
        ctx.step(state["n"])
        e = ctx.energy()
        F = ctx.forces(L.FORCE_GRADP)
        return {"energy": e, "F": F, **_views(state, ("psi", "P", "label", "W"))}
    if kind == "mf":
        mf = state["mf"]
        out = mf.frame()
        _read_fields(mf.lib.rq_mf_download, mf.s, state["buf"])
        return {"energies": {k: out[k] for k in ("E", "E_T", "E_eK", "E_ee")}, "norms": out["norms"],
                "force": [list(f) for f in mf.nuc_force], "fields": state["buf"]}
    if kind == "rb":
        rb = state["rb"]
        rb.doSteps(state["n"])
        e = rb.computeEnergy()
        _read_fields(rb.lib.rq_rb_download, rb.s, state["buf"])
        return {"energies": [e["E_T"], e["E_eK"], e["E_ee"]], "fields": state["buf"]}
    sh = state["sh"]
    e = sh.step(state["n"])
    _read_fields(sh.lib.rq_shells_download, sh.s, state["buf"])
    return {"energies": [e["E_T"], e["E_eK"], e["E_ee"]], "fields": state["buf"]}


# ---- what a pass cannot do without -------------------------------------------------------------
def _mg_bytes(n, es):
    """One V(1,1): the right-hand side and P read, P written, per level (coarser ones 1/8 each)."""
    return 3 * es * n * 8 / 7


def work(case):
    """Per step, each field the step needs read once and each field it changes written once (the
    steps depend on one another and the fields of the larger grids exceed the caches); operations
    of the stencils by count."""
    c, kind = case, case["kind"]
    if kind == "sp":  # psi, label, K, P -> psi, P every step; one 7-point update and one sweep
        n = (c["NN"] - 1) ** 3
        return {"bytes": 100 * 24.0 * n, "flops": 100 * 30.0 * n}
    if kind in ("new", "evaluate"):
        n = (c["NN"] - 1) ** 3
        es = 8 if c.get("precision") == "fp64" else 4
        step = 4 * es + 1 + _mg_bytes(1, es) / 4
        if kind == "new":
            return {"bytes": 20 * step * n, "flops": 20 * 30.0 * n}
        # forward as above with psi kept; backward: adjoint psi, psi, K, P -> adjoint psi, and dE/dK
        back = 5 * es + 1 + 2 * _mg_bytes(1, es) / 4
        return {"bytes": c["iters"] * (step + es + back) * n + 16.0 * n, "flops": c["iters"] * 90.0 * n}
    if kind == "batch":
        es = 8 if c["precision"] == "fp64" else 4
        n = sum((g.NN - 1) ** 3 for g in _cluster_geometries(c, 0))
        return {"bytes": 20 * (4 * es + 4 + _mg_bytes(1, es) / 4) * n + 5.0 * es * n, "flops": 20 * 30.0 * n}
    if kind == "mj":
        # per step: psi, label, K, Pother -> psi; the Poisson potentials (one each of the three
        # electrons, or the total) read and written; per level-set pass: label, psi, W -> W, label
        n = (c["NN"] - 1) ** 3
        return {"bytes": c["steps"] * (20.0 + (24 if c["sic"] else 8) + 20.0) * n, "flops": c["steps"] * 60.0 * n}
    if kind == "lobpcg":
        # per domain and iteration the vectors X, W, P and H applied to them, read and written, on
        # that domain's third of the cells; then the level-set passes
        n = (c["NN"] - 1) ** 3
        return {"bytes": c["frames"] * (10 * 60.0 + c["steps"] * 20.0) * n, "flops": c["frames"] * 10 * 100.0 * n}
    if kind == "mf":
        n = (c["NN"] - 1) ** 3
        ne = 1 + c["hydrogens"]
        return {"bytes": c["steps"] * (24.0 * ne + 4) * n, "flops": c["steps"] * 100.0 * ne * n}
    if kind == "rb":
        n = (c["NN"] - 1) ** 3
        ne = c["nuclei"] * c["ne"]
        return {"bytes": c["steps"] * (24.0 * ne + 4) * n, "flops": c["steps"] * 90.0 * ne * n}
    n = (c["NN"] - 1) ** 3
    sweeps = 8 + 20 / 8 if c["poisson"] == "multigrid" else 1
    return {"bytes": c["steps"] * c["shells"] * 32.0 * n, "flops": c["steps"] * c["shells"] * (60 + 9 * sweeps) * n}


# ---- the same in 64 bits ---------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _axes(S, h, dev):
    x = torch.arange(S, dtype=torch.float64, device=dev) * h
    return x.view(-1, 1, 1), x.view(1, -1, 1), x.view(1, 1, -1)


def _in(a):
    return a[1:-1, 1:-1, 1:-1]


def _shifts(a):
    """The six neighbours of the interior points: +i, -i, +j, -j, +k, -k."""
    return (a[2:, 1:-1, 1:-1], a[:-2, 1:-1, 1:-1], a[1:-1, 2:, 1:-1], a[1:-1, :-2, 1:-1], a[1:-1, 1:-1, 2:],
            a[1:-1, 1:-1, :-2])


def _sum6(a):
    p = _shifts(a)
    return p[0] + p[1] + p[2] + p[3] + p[4] + p[5]


def _domain_sum(v, lab, n):
    return torch.zeros(n, dtype=torch.float64, device=v.device).index_add_(0, lab.reshape(-1), v.reshape(-1))


class _Field:
    """The solver.py and new flavours restated: psi, P, label, K on an S^3 grid."""

    def __init__(self, NN, h, rows):
        self.NN, self.S, self.h = NN, NN + 1, h
        self.rows = rows
        self.dev = _dev()
        self.Z = torch.tensor([r["Z"] for r in rows], dtype=torch.float64, device=self.dev)
        self.psi = torch.zeros((self.S,) * 3, dtype=torch.float64, device=self.dev)
        self.P = torch.zeros_like(self.psi)
        self.K = torch.zeros_like(self.psi)
        self.label = torch.zeros((self.S,) * 3, dtype=torch.int64, device=self.dev)

    def same(self):
        """Where the six neighbours carry the point's label."""
        c = _in(self.label)
        return [q == c for q in _shifts(self.label)]

    def update(self, same, half_dv, dt):
        c = _in(self.psi)
        lap = -6.0 * c
        for q, s in zip(_shifts(self.psi), same):
            lap = lap + torch.where(s, q, c)
        new = torch.zeros_like(self.psi)
        _in(new)[...] = c + half_dv * lap + dt * (_in(self.K) - 2.0 * _in(self.P)) * c
        self.psi = new

    def normalise(self):
        n = _domain_sum(self.psi ** 2 * self.h ** 3, self.label, len(self.rows))
        s = torch.where((self.Z > 0) & (n > 0), torch.sqrt(self.Z / n.clamp(min=1e-300)), torch.ones_like(n))
        self.psi = self.psi * s[self.label]

    def kinetic(self, faces):
        """h/2 times the squared forward differences to neighbours of the same label, per point."""
        u, l = _in(self.psi), _in(self.label)
        t = torch.zeros_like(u)
        sh, lh = _shifts(self.psi), _shifts(self.label)
        for q in (0, 2, 4):
            t = t + torch.where(lh[q] == l, (sh[q] - u) ** 2, torch.zeros_like(u))
        if faces:  # the edge to the Dirichlet face below the first layer
            for q, a in ((1, 0), (3, 1), (5, 2)):
                first = [slice(None)] * 3
                first[a] = slice(0, 1)
                first = tuple(first)
                t[first] += torch.where(lh[q][first] == l[first], u[first] ** 2, torch.zeros_like(u[first]))
        return 0.5 * t * self.h


def _pair_energy(xyz, Z, soft2):
    e = 0.0
    for a in range(len(Z)):
        d = xyz[a + 1:] - xyz[a]
        e += float(np.sum(Z[a] * Z[a + 1:] / np.sqrt((d * d).sum(1) + soft2)))
    return e


def _exact_sp(c, seed):
    g = _geometry(c, seed)
    rows = configs.to_reference_atoms(g)
    f = _Field(c["NN"], g.screen / c["NN"], rows)
    h, dev = f.h, f.dev
    pos = np.array([[r["i"], r["j"], r["k"]] for r in rows], np.float32).astype(np.float64) * h
    zs = [r["Z"] for r in rows]
    x, y, z = _axes(f.S, h, dev)
    best = torch.zeros_like(f.psi)
    for n, (p, Z) in enumerate(zip(pos, zs)):
        r = torch.sqrt((x - p[0]) ** 2 + (y - p[1]) ** 2 + (z - p[2]) ** 2 + h * h)
        _in(f.K).add_(_in(Z / r))
        u = Z * Z * 0.5641895835 * torch.exp(-Z * r)
        win = torch.zeros_like(f.label, dtype=torch.bool)
        _in(win)[...] = _in(u > best)
        best = torch.where(win, u, best)
        f.label = torch.where(win, torch.full_like(f.label, n), f.label)
    f.psi = best
    f.normalise()

    def sweep():
        new = torch.zeros_like(f.P)
        _in(new)[...] = (_sum6(f.P) + 2.0 * math.pi * _in(f.psi) ** 2 * h * h) / 6.0
        f.P = new

    for _ in range(200):
        sweep()
    n = len(rows)
    dv = 0.005 if n > 500 else 0.01 if n > 200 else 0.02 if n > 100 else 0.03 if n > 30 else 0.12
    same = f.same()
    for s in range(1, 101):
        if s % 2 == 0:
            sweep()
            sweep()
        f.update(same, 0.5 * dv, dv * h * h)
        if s % 20 == 0:
            f.normalise()
    # the label step of step 100: a cell with two foreign neighbours goes to the strongest atom
    foreign = sum((~q).to(torch.int64) for q in same)
    top = torch.full_like(f.psi, -1.0)
    who = f.label.clone()
    mine = torch.zeros_like(f.psi)
    for q, (p, Z) in enumerate(zip(pos, zs)):
        sc = Z / torch.sqrt((x - p[0]) ** 2 + (y - p[1]) ** 2 + (z - p[2]) ** 2 + h * h)
        mine = torch.where(f.label == q, sc, mine)
        win = sc > top
        top = torch.where(win, sc, top)
        who = torch.where(win, torch.full_like(who, q), who)
    _in(f.label)[...] = torch.where((foreign >= 2) & (_in(top) > 1.1 * _in(mine)), _in(who), _in(f.label))
    rho = _in(f.psi) ** 2 * h ** 3
    T, EK, EE = (float(v.sum()) for v in (f.kinetic(False), -_in(f.K) * rho, _in(f.P) * rho))
    KK = _pair_energy(pos, np.array(zs), h * h)
    return {"energy": np.array([T + EK + EE + KK, T, EK, EE, KK, 0, 0, 0]), "psi": f.psi, "P": f.P, "label": None}


def _gaussian_potential(f, pos, Z, sigma):
    x, y, z = _axes(f.S, f.h, f.dev)
    K = torch.zeros_like(f.psi)
    for p, q in zip(pos, Z):
        r = torch.sqrt((x - p[0]) ** 2 + (y - p[1]) ** 2 + (z - p[2]) ** 2)
        v = torch.where(r < 1e-12, torch.full_like(r, math.sqrt(2 / math.pi) / sigma),
                        torch.erf(r / (math.sqrt(2) * sigma)) / r.clamp(min=1e-12))
        _in(K).add_(_in(v), alpha=float(q))
    return K


def _nearest(f, seeds, first):
    """Nearest electron seed (f32 distances, as the labels are whole numbers) and its distance."""
    S, dev = f.S, f.dev
    hf = np.float32(f.h)
    x = torch.from_numpy(np.arange(S, dtype=np.float32) * hf).to(dev)
    best = torch.full((S, S, S), 3.4e38, dtype=torch.float32, device=dev)
    lab = torch.zeros((S, S, S), dtype=torch.int64, device=dev)
    for q, s in enumerate(np.asarray(seeds, np.float64).astype(np.float32)):
        d = [(x - float(s[a])) ** 2 for a in range(3)]
        d2 = (d[0].view(-1, 1, 1) + d[1].view(1, -1, 1)) + d[2].view(1, 1, -1)
        win = d2 < best
        best = torch.where(win, d2, best)
        lab.masked_fill_(win, first + q)
    return lab, best.double()


def _vcycle(P, fr, h, NN):
    """One V(1,1): red-black sweeps, full weighting, trilinear correction, 16 coarsest sweeps."""
    n = torch.arange(1, NN, device=P.device)
    par = (n.view(-1, 1, 1) + n.view(1, -1, 1) + n.view(1, 1, -1)) & 1

    def sweep():
        for color in (0, 1):
            v = (_sum6(P) + h * h * _in(fr)) / 6.0
            _in(P)[...] = torch.where(par == color, v, _in(P))

    if NN % 2 or NN // 2 < 6:  # the coarsest level
        for _ in range(16):
            sweep()
        return P
    sweep()
    r = torch.zeros_like(P)
    _in(r)[...] = _in(fr) + (_sum6(P) - 6.0 * _in(P)) / (h * h)
    for a in range(3):  # full weighting, one axis at a time
        m = r.shape[a]
        lo, mid, hi = (r.index_select(a, torch.arange(q, m - 3 + q, 2, device=P.device)) for q in (1, 2, 3))
        r = 0.25 * lo + 0.5 * mid + 0.25 * hi
        pad = [0, 0, 0, 0, 0, 0]
        pad[2 * (2 - a)] = pad[2 * (2 - a) + 1] = 1
        r = torch.nn.functional.pad(r, pad)
    e = _vcycle(torch.zeros_like(r), r, 2 * h, NN // 2)
    for a in range(3):  # trilinear
        m = e.shape[a]
        shape = list(e.shape)
        shape[a] = 2 * m - 1
        fine = torch.empty(shape, dtype=e.dtype, device=e.device)
        even = tuple(slice(0, None, 2) if q == a else slice(None) for q in range(3))
        odd = tuple(slice(1, None, 2) if q == a else slice(None) for q in range(3))
        fine[even] = e
        fine[odd] = 0.5 * (e.narrow(a, 0, m - 1) + e.narrow(a, 1, m - 1))
        e = fine
    _in(P).add_(_in(e))
    sweep()
    return P


def _new_state(NN, h, rows):
    f = _Field(NN, h, rows)
    f.pos = np.array([[r["i"], r["j"], r["k"]] for r in rows if r["Z_nuc"] > 0]) * h
    f.q = np.array([r["Z_nuc"] for r in rows if r["Z_nuc"] > 0])
    seeds = np.array([[r["i"], r["j"], r["k"]] for r in rows if r["Z"] > 0]) * h
    f.K = _gaussian_potential(f, f.pos, f.q, h)
    f.label, d2 = _nearest(f, seeds, len(f.q))
    _in(f.psi)[...] = _in(torch.exp(-torch.sqrt(d2)))
    f.normalise()
    for _ in range(10):
        _vcycle(f.P, 2.0 * math.pi * f.psi ** 2, h, NN)
    return f


def _new_steps(f, done, n):
    same = f.same()
    for s in range(done + 1, done + n + 1):
        if s % 4 == 0:
            _vcycle(f.P, 2.0 * math.pi * f.psi ** 2, f.h, f.NN)
        f.update(same, 0.1, 0.2 * f.h * f.h)
        if (s + 1) % 4 == 0:
            f.normalise()
    f.normalise()


def _new_energy(f):
    """The readout: per-domain terms and the P-stationary Hartree energy."""
    h3 = f.h ** 3
    rho = _in(f.psi) ** 2 * h3
    AP = (6.0 * _in(f.P) - _sum6(f.P)) / (f.h * f.h)
    T, EK = float(f.kinetic(True).sum()), float((-_in(f.K) * rho).sum())
    EE = float(2.0 * (_in(f.P) * rho).sum() - h3 / (2.0 * math.pi) * (_in(f.P) * AP).sum())
    KK = _pair_energy(f.pos, f.q, 0.0)
    return np.array([T + EK + EE + KK, T, EK, EE, KK, 0, 0, 0])


def _hf_forces(f):
    """Hellmann-Feynman forces of the Gaussian nuclei plus their repulsion, per entry."""
    x, y, z = _axes(f.S, f.h, f.dev)
    rho, sig = f.psi ** 2, f.h
    F = np.zeros((len(f.rows), 3))
    for n, (p, q) in enumerate(zip(f.pos, f.q)):
        d = (x - p[0], y - p[1], z - p[2])
        r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2).clamp(min=1e-12)
        dk = math.sqrt(2 / math.pi) / sig * torch.exp(-r * r / (2 * sig * sig)) / r - \
            torch.erf(r / (math.sqrt(2) * sig)) / (r * r)
        w = -f.h ** 3 * rho * dk / r
        F[n] = [q * float((w * t).sum()) for t in d]
        e = p - np.delete(f.pos, n, 0)
        F[n] += (q * np.delete(f.q, n)[:, None] * e / ((e * e).sum(1) ** 1.5)[:, None]).sum(0)
    return F


def _exact_rb(c, seed):
    """realqm_rb.js: nuclei with one electron each, red and black passes of front, amplitude and
    potential, normalisation on every fifth step."""
    NN, h, dev = c["NN"], c["screen"] / c["NN"], _dev()
    S, n = NN + 1, c["nuclei"]
    nuc = [[float(np.float32(a[q])) for q in "ijk"] + [float(a["Z"])] for a in _rb_nuclei(c, seed)]
    ax = torch.arange(S, dtype=torch.float64, device=dev)
    d2 = [h * h * ((ax - a[0]).view(-1, 1, 1) ** 2 + (ax - a[1]).view(1, -1, 1) ** 2 + (ax - a[2]).view(1, 1, -1) ** 2)
          for a in nuc]
    K = torch.zeros((S, S, S), dtype=torch.float64, device=dev)
    U, W, P = ([torch.zeros_like(K) for _ in range(n)] for _ in range(3))
    for m, a in enumerate(nuc):
        soft = torch.sqrt(d2[m] + 1.2 * h * h)
        _in(K).add_(_in(a[3] / soft))
        own = torch.sqrt(d2[m]) < 3.0
        for b in range(n):
            if b != m:
                own = own & ~(d2[m] > d2[b])
        _in(W[m])[...] = _in(own.double())
        _in(U[m])[...] = _in(torch.where(own, torch.exp(-0.5 * a[3] * soft), torch.zeros_like(soft)))
        _in(P[m])[...] = _in(0.5 / soft)
    i = torch.arange(1, NN, device=dev)
    par = (i.view(-1, 1, 1) + i.view(1, -1, 1) + i.view(1, 1, -1)) & 1
    dt, half_d = 0.1 * h * h, 0.05
    for s in range(c["steps"]):
        u0 = [_in(u).clone() for u in U]
        rho = sum(u * u for u in u0)
        rival = [torch.stack([u0[q] for q in range(n) if q != m]).amax(0) for m in range(n)]
        for color in (0, 1):
            on = par == color
            for m in range(n):
                u, w, p = _in(U[m]).clone(), _in(W[m]), _in(P[m])
                cc = 0.1 * (u - rival[m])
                ws, us, ps = _shifts(W[m]), _shifts(U[m]), _shifts(P[m])
                lap = sum(ws) - 6.0 * w
                grad = torch.sqrt(sum(((ws[q] - ws[q + 1]) / h) ** 2 for q in (0, 2, 4)))
                w2 = w + 0.5 * dt * cc.abs() * lap / (h * h) + 10.0 * dt * cc * grad
                wl = sum((us[q] - u) * (ws[q] + w2) * 0.5 for q in range(6))
                new = u + half_d * wl + dt * (_in(K) - 2.0 * p) * u * w2
                lapP = sum(ps) - 6.0 * p
                pn = p + dt * (lapP / (h * h) + 2.0 * math.pi * (rho - new * new).clamp(min=0.0))
                for a, v in ((W[m], w2), (U[m], new), (P[m], pn)):
                    _in(a)[...] = torch.where(on, v, _in(a))
        if s % 5 == 0:
            for m in range(n):
                norm = float((_in(U[m]) ** 2).sum()) * h ** 3
                if norm > 0:
                    _in(U[m]).mul_(math.sqrt(1.0 / norm))
    T = EK = EE = 0.0
    for m in range(n):
        u, w = _in(U[m]), _in(W[m])
        us, ws = _shifts(U[m]), _shifts(W[m])
        for q in (0, 2, 4):
            T += 0.5 * h * float(torch.where((w > 0.1) & (ws[q] > 0.1), (us[q] - u) ** 2, torch.zeros_like(u)).sum())
        EK -= float((_in(K) * u * u).sum()) * h ** 3
        EE += float((_in(P[m]) * u * u).sum()) * h ** 3
    fields = torch.stack([torch.stack([a[m].reshape(-1) for a in (U, W, P)]) for m in range(n)])
    return {"energies": [T, EK, EE], "fields": fields}


def exact(case, seed):
    """The pass restated in 64 bits.  The adjoint forces have no value here (a reverse sweep through
    hundreds of steps), the labels are whole numbers, and the pages of molecule.js, mol_fast.js and
    atom.js are defined by the f32 stores, tree sums and fixed-point sums of their in-place passes."""
    c, kind = case, case["kind"]
    if kind == "sp":
        return _exact_sp(c, seed) if (c["NN"] ** 3) * max(10, 3 * c["waters"]) < 8e9 else None
    if kind == "new":
        g = _geometry(c, seed)
        if g.NN ** 3 * len(g.seeds) > 8e9:
            return None
        f = _new_state(g.NN, g.h, configs.to_domain_atoms(g))
        _new_steps(f, 0, 20)
        return {"energy": _new_energy(f), "psi": f.psi, "P": f.P, "label": None}
    if kind == "evaluate":
        g = _geometry(c, seed)
        if g.NN ** 3 * len(g.seeds) > 8e9:
            return None
        f = _new_state(g.NN, g.h, configs.to_domain_atoms(g))
        _new_steps(f, 0, 1)
        f.pos = _moved(g, seed) + (g.NN // 2) * g.h
        f.K = _gaussian_potential(f, f.pos, f.q, g.h)
        _new_steps(f, 1, c["iters"])
        return {"E": float(_new_energy(f)[0]), "F": None, "psi": f.psi, "P": f.P}
    if kind == "batch":
        if c["n"] > 48:
            return None
        E, F = [], []
        for g in _cluster_geometries(c, seed):
            f = _new_state(g.NN, g.h, configs.to_domain_atoms(g))
            _new_steps(f, 0, 20)
            E.append(_new_energy(f))
            F.append(_hf_forces(f))
        return {"energy": np.stack(E), "F": np.concatenate(F)}
    if kind == "rb" and c["ne"] == 1:
        return _exact_rb(c, seed)
    return None
