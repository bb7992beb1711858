"""The atom.js per-shell solver (rq_shells_*) on the GPU against the oracle's sequential
restatement of atom.js (oracle.AtomShellsDriver).

The GPU runs the reference's in-place lexicographic sweeps as hyperplane wavefronts, so each
cell sees exactly the neighbour values the sequential loop sees and every f32 store is the
same.  Only the FP64 sums (the per-shell normalisation and the energies) are summed in another
order: the scale of a normalisation can then differ in its last bit, which moves a rare f32
store by one ulp.  Bars: the initial state bit-exact; after the steps >= 99.9 % of the values of
every field bit-equal and all within 1e-5 relative; energies within 1e-9 relative.
"""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu

HE = [{"ne": 1, "Rmax": 5.0, "Zeff": 2, "split": "halfspace", "halfIndex": 0, "fixedW": True},
      {"ne": 1, "Rmax": 5.0, "Zeff": 2, "split": "halfspace", "halfIndex": 1, "fixedW": True}]
RADIAL = [{"ne": 1, "Rmax": 1.0, "Zeff": 2}, {"ne": 1, "Rmax": 5.0, "Zeff": 1}]
THREE = [{"ne": 2, "Rmax": 1.2, "Zeff": 3}, {"ne": 1, "Rmax": 3.0, "Zeff": 1.5},
         {"ne": 1, "Rmax": 0.0, "Zeff": 1, "outerHalf": True}]

CASES = [("he_halfspace", 32, 5.0, 2, HE, 0.15, "multigrid", 4),
         ("radial_fronts", 40, 10.0, 2, RADIAL, 0.1, "multigrid", 4),
         ("three_simultaneous", 36, 9.0, 3, THREE, 0.1, "simultaneous", 6)]


def pair(case):
    from realmolecule_b200.shells import AtomShells
    _, NN, scr, Z, shells, d, mode, _ = case
    ref = orc.AtomShellsDriver(NN, scr, Z, shells, d=d, poisson=mode)
    ref.initialize()
    gpu = AtomShells(NN, scr, Z, shells, d=d, poisson=mode)
    return ref, gpu


def fields_of(ref, m):
    S3 = ref.S3
    return {"U": ref.U[m * S3:(m + 1) * S3], "W": ref.W[m * S3:(m + 1) * S3], "P": ref.P[m * S3:(m + 1) * S3]}


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_initial_state_bit_exact(case):
    ref, gpu = pair(case)
    for m in range(gpu.n_shells):
        g, r = gpu.fields(m), fields_of(ref, m)
        for k in ("U", "W", "P"):
            assert np.array_equal(g[k].view(np.uint32), r[k].view(np.uint32)), (m, k)
    gpu.close()


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_steps_match_the_sequential_sweep(case):
    ref, gpu = pair(case)
    nsteps = case[-1]
    for _ in range(nsteps):
        E4, ps = ref.step()
    res = gpu.step(nsteps)
    for m in range(gpu.n_shells):
        g, r = gpu.fields(m), fields_of(ref, m)
        for k in ("U", "W", "P"):
            same = (g[k].view(np.uint32) == r[k].view(np.uint32)).mean()
            assert same >= 0.999, (m, k, same)
            np.testing.assert_allclose(g[k], r[k], rtol=1e-5, atol=1e-7 * np.abs(r[k]).max())
    for key, v in zip(("E", "E_T", "E_eK", "E_ee"), E4):
        assert abs(res[key] - v) <= 1e-9 * max(1.0, abs(v)), (key, res[key], v)
    np.testing.assert_allclose(np.array(res["nrm_m"]), ps[:, 3], rtol=1e-9)
    assert gpu.kernel_launches > 0
    gpu.close()


def radial(n):
    return [{"ne": 1, "Rmax": 0.6 + 0.5 * q if q < n - 1 else 5.0, "Zeff": 2.0 / (q + 1), "fixedW": q % 3 == 2}
            for q in range(n)]


# Interiors of one partial block, a block and one cell, two blocks and one, and whole blocks, of both
# block edges (16: up to two shells; 8: more shells, and the coarse smoother)
@pytest.mark.parametrize("mode", ["multigrid", "simultaneous"])
@pytest.mark.parametrize("n_shells", [1, 2, 3, 8])
@pytest.mark.parametrize("NN", [8, 10, 18, 34, 48])
def test_block_edges_match_the_sequential_sweep(NN, n_shells, mode):
    ref, gpu = pair(("", NN, 6.0, 2, radial(n_shells), 0.1, mode, 1))
    E4, ps = ref.step()
    res = gpu.step(1)
    for m in range(n_shells):
        g, r = gpu.fields(m), fields_of(ref, m)
        for k in ("W", "P"):  # no sum enters these in the first step
            assert np.array_equal(g[k].view(np.uint32), r[k].view(np.uint32)), (m, k)
        np.testing.assert_allclose(g["U"], r["U"], rtol=2.4e-7, atol=0)  # the scale's last bit, then one rounding
    for key, v in zip(("E", "E_T", "E_eK", "E_ee"), E4):
        assert abs(res[key] - v) <= 1e-9 * max(1.0, abs(v)), (key, res[key], v)
    np.testing.assert_allclose(np.array(res["nrm_m"]), ps[:, 3], rtol=1e-9)
    gpu.close()
