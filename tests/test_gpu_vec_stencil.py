"""The 16-byte-vector stencil passes at the sizes where their groups can go wrong: rows of every alignment
(S = 1 and 3 mod 4), the smallest grids, planes of one block and of several, one and several planes per
block.  Against the oracle's restatement: the solver.py schedule is f32 arithmetic in the reference's
order, so psi and P after one step are the oracle's bit for bit; the label step is integer work."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


def atoms_for(NN, n, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(0.15 * NN, 0.85 * NN, (n, 3))
    return [{"i": float(a), "j": float(b), "k": float(c), "Z": float(rng.integers(1, 9)), "rc": 0.0} for a, b, c in p]


@pytest.mark.parametrize("NN", [8, 10, 14, 16, 30, 32, 62, 64, 66, 126, 200])
def test_solverpy_steps_bit_exact(NN):
    from realmolecule_b200 import Context
    atoms = atoms_for(NN, 5, NN)
    ref = orc.SolverPyDriver({"gridN": NN, "screen": 0.25 * NN, "atoms": atoms}, kernels="oracle")
    rng = np.random.default_rng(1)
    S = NN + 1
    inner = np.zeros((S, S, S), bool)
    inner[1:-1, 1:-1, 1:-1] = True
    ctx = Context(NN, 0.25 * NN, atoms, flavor="solver.py")
    ctx.initialize()
    ref.initialize(bootstrap=0)
    ref.K[:] = ctx.download_K()
    ref.U[:] = np.where(inner, rng.uniform(0.0, 0.5, inner.shape), 0).astype(np.float32).ravel()
    ref.P[:] = np.where(inner, rng.uniform(0.0, 2.0, inner.shape), 0).astype(np.float32).ravel()
    ref.P[:] *= np.float32(10.0) ** rng.integers(-44, 1, ref.P.shape).astype(np.float32)  # to the subnormals
    ref.label[:] = rng.integers(0, 5, ref.label.shape) // 2  # neighbours equal and different in every mix
    ctx.upload(psi=ref.U, label=ref.label, P=ref.P)
    for _ in range(5):  # both fused forms, no normalisation
        ref.steps_done += 1
        ref.step(ref.steps_done)
    ctx.step(5)
    st = ctx.download(psi=True, label=True, P=True)
    assert np.array_equal(st["psi"].view(np.uint32), ref.U.view(np.uint32))
    assert np.array_equal(st["P"].view(np.uint32), ref.P.view(np.uint32))
    ctx.close()


@pytest.mark.parametrize("NN,n", [(8, 65), (22, 90), (46, 300)])
def test_binned_label_step_from_any_labels(NN, n):
    from realmolecule_b200 import Context
    atoms = atoms_for(NN, n, NN)
    ref = orc.SolverPyDriver({"gridN": NN, "screen": 0.3 * NN, "atoms": atoms}, kernels="oracle")
    ctx = Context(NN, 0.3 * NN, atoms, flavor="solver.py", label_interval=1)
    ctx.initialize()
    lab = np.random.default_rng(2).integers(0, n, ref.label.shape).astype(np.int32)
    ref.label[:] = lab
    ctx.upload(label=lab)
    ctx.step(1)
    ref.boundary()
    got = ctx.download(psi=False, label=True)["label"].reshape((NN + 1,) * 3)
    want = ref.label.reshape((NN + 1,) * 3)
    assert np.array_equal(got[1:-1, 1:-1, 1:-1], want[1:-1, 1:-1, 1:-1])
    ctx.close()
