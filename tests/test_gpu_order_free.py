"""The per-domain sums that scale fp32 fields (the norms, the readout's weights, the reverse sweep's <psi, lambda>)
do not depend on the order in which the blocks of a launch finish."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(NN, waters, seed, **kw):
    from realmolecule_b200 import configs
    from realmolecule_b200.autograd import EnergyModel
    rng = np.random.default_rng(seed)
    el, xyz = configs.water_box(waters, NN * 0.1 - 5.0, 2.7, rng, sphere=True)
    g = configs.Geometry("", el, xyz, NN, 0.2)
    seeds, _ = configs.electron_seeds(el, xyz, rng)
    off = NN // 2 * 0.2
    m = EnergyModel(NN, 0.2, g.charges, xyz + off, seeds + off, tol=None, label_until=1, **kw)
    return m, xyz + off + rng.normal(0.0, 0.02, xyz.shape)


@pytest.mark.parametrize("NN,waters,precision", [(128, 12, "mixed"), (80, 2, "mixed"), (64, 1, "fp64")])
def test_two_evaluations_agree(NN, waters, precision):
    """Fresh models, two evaluations each: psi and P bit for bit, and with them every rounding of the reverse sweep, so
    that the forces differ by their own last FP64 sums only (about 1e5 terms in any order: 1e5 2^-53 ~ 1e-11)."""
    runs = []
    for _ in range(3):
        m, x = _model(NN, waters, 5, precision=precision, warm_steps=24)
        got = []
        for _ in range(2):
            E, F, _ = m.evaluate(x)
            s = m.ctx.download(psi=True, label=False, P=True)
            got.append((E, F, s["psi"], s["P"]))
        runs.append(got)
        m.ctx.close()
    for other in runs[1:]:
        for (E, F, psi, P), (E1, F1, psi1, P1) in zip(runs[0], other):
            assert np.array_equal(psi, psi1) and np.array_equal(P, P1)
            assert E == E1
            assert np.abs(F - F1).max() <= 1e-11 * np.abs(F).max()


def test_domain_sums_match_numpy():
    """The readout's norm of every domain against numpy's sum of the downloaded state: n 2^-53 of it."""
    m, x = _model(80, 2, 7, precision="mixed", warm_steps=8)
    m.evaluate(x)
    _, pd = m.ctx.energy(per_domain=True)
    s = m.ctx.download(psi=True, label=True)
    u2 = s["psi"].astype(np.float64) ** 2 * 0.2 ** 3
    want = np.bincount(s["label"], weights=u2, minlength=m.ctx.n_atoms)
    assert np.abs(pd[:, 0] - want).max() <= 81 ** 3 * 2.0 ** -53 * want.max()
    m.ctx.close()
