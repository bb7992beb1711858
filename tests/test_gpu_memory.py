"""Device memory: what a solver object holds, in fields of its grid, and steps with less of it than they would like.

A field is S^3 elements; the counts are those of the buffers each solver cannot do without (two psi, two P, K, ...),
plus the multigrid levels (1/7 of a field each).  Allocations are rounded up to 2 MB, and small ones share blocks."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BLOCK = 2 << 20


def held(make):
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    obj = make()
    torch.cuda.synchronize()
    return obj, free0 - torch.cuda.mem_get_info()[0]


ROWS = [{"i": 100, "j": 100, "k": 100, "Z": 2.0, "Z_nuc": 2.0}, {"i": 110, "j": 100, "k": 100, "Z": 1.0, "Z_nuc": 1.0},
        {"i": 90, "j": 95, "k": 100, "Z": 1.0, "Z_nuc": 1.0}]


@pytest.mark.parametrize("flavor,kw,per_point,blocks", [
    # blocks: the fields, three coarse levels, small ones
    # psi, psi', P, P', K, W, labels twice, the FP64 K, the label mask, P and f of the coarse levels
    ("new", {}, 4 * 5 + 4 + 8 + 8 + 1 + 2 * 4 / 7, 20), ("new", dict(precision="fp64"), 8 * 5 + 4 + 8 + 1 + 2 * 8 / 7, 20),
    ("solver.py", {}, 4 * 7 + 8, 13),  # psi, psi', P, P', K, W, the trial state; labels twice
    # psi, psi', P, P', K, W, trial state, rho, Pother, residual, two self-potentials, P_m; labels twice; coarse grid
    ("molecule.js", dict(sic=1), 4 * (12 + len(ROWS)) + 8 + 4 * 3 / 8, 25)])
def test_context(flavor, kw, per_point, blocks):
    from realmolecule_b200 import Context
    NN = 320
    ctx, got = held(lambda: Context(NN, 32.0, ROWS, flavor=flavor, **kw))
    ctx.close()
    assert got <= per_point * (NN + 1) ** 3 + blocks * BLOCK, got / (NN + 1) ** 3


def test_adjoint_window():
    """5 steps (psi), 4 P, lambda and dE/dP twice, dE/df, dE/dK in FP64, four fields of the coarse levels, and the
    finest residual's adjoint."""
    from realmolecule_b200 import Context
    NN = 320
    ctx = Context(NN, 32.0, ROWS, flavor="new")
    _, got = held(lambda: ctx.set_adjoint_window(5))
    ctx.close()
    assert got <= (4 * (5 + 4 + 2 + 2 + 1 + 1) + 8 + 4 * 4 / 7) * (NN + 1) ** 3 + 25 * BLOCK, got / (NN + 1) ** 3


def test_batch():
    """psi, psi', P, P', K in both precisions (a mixed batch keeps a set to be promoted into), the coarse levels with a
    residual each, labels twice, W, the label mask."""
    from realmolecule_b200.batch import Batch
    NN = 320
    b, got = held(lambda: Batch([{"NN": NN, "screen": 32.0, "atoms": ROWS}], precision="mixed"))
    b.close()
    assert got <= (12 * 5 + 8 + 4 + 1 + 3 * 12 / 7) * (NN + 1) ** 3 + 45 * BLOCK, got / (NN + 1) ** 3


@pytest.mark.parametrize("room", [6.6, 4.0, 1.6])
def test_shells_with_little_memory(room):
    """Six shells whose Poisson buffers (a field and a quarter each) do not all fit: solved a few at a time, the same
    fields bit for bit and the same energies."""
    from realmolecule_b200.shells import AtomShells
    NN, n = 200, 6
    shells = [{"ne": 1, "Rmax": 0.6 + 0.5 * q if q < n - 1 else 5.0, "Zeff": 2.0 / (q + 1)} for q in range(n)]
    make = lambda: AtomShells(NN, 6.0, 6.0, shells, d=0.1)
    field = 4 * (NN + 1) ** 3
    out = []
    for short in (False, True):
        if short:
            free = torch.cuda.mem_get_info()[0]
            ballast = torch.empty(free - int((3 * n + 1 + room) * field), dtype=torch.uint8, device="cuda")
        sh = make()
        r = sh.step(2)
        out.append((r, [sh.fields(m) for m in range(n)], sh.kernel_launches))
        sh.close()
        if short:
            del ballast
            torch.cuda.empty_cache()
    assert out[1][2] > out[0][2]
    for a, b in zip(out[0][1], out[1][1]):
        for k in ("U", "W", "P"):
            np.testing.assert_allclose(a[k], b[k], rtol=2.4e-7, atol=0)  # the FP64 norm's order: the scale's last bit
    np.testing.assert_allclose([out[0][0][k] for k in ("E", "E_T", "E_eK", "E_ee")],
                               [out[1][0][k] for k in ("E", "E_T", "E_eK", "E_ee")], rtol=1e-9)
