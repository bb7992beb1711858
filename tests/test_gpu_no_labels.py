"""A context whose state comes by upload without labels, and which was never initialised, steps as one domain: its
labels are 0 from the allocation, and so is what the kernels derive from them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flavor,opts,steps", [("solver.py", dict(poisson_interval=2), 5), ("new", dict(label_until=1), 6),
                                               ("new", dict(label_until=1, precision="fp64"), 6)])
@pytest.mark.parametrize("NN", [16, 22])
def test_upload_without_labels(flavor, opts, steps, NN):
    from realmolecule_b200 import Context
    rng = np.random.default_rng(3)
    S = NN + 1
    x = np.zeros((S, S, S))
    x[1:-1, 1:-1, 1:-1] = rng.uniform(0.2, 1.0, (NN - 1,) * 3)
    P = np.zeros_like(x)
    P[1:-1, 1:-1, 1:-1] = rng.uniform(0.0, 0.3, (NN - 1,) * 3)
    rows = [{"i": NN / 2, "j": NN / 2, "k": NN / 2, "Z": 1.0, "Z_nuc": 1.0}]
    out = []
    for label in (None, np.zeros(S ** 3, np.int32)):
        ctx = Context(NN, 8.0, rows, flavor=flavor, **opts)
        ctx.set_atoms(rows)  # the nuclear potential, which initialize() would have made
        ctx.upload(psi=x, P=P, label=label)
        ctx.step(steps)
        out.append(ctx.download(psi=True, label=False, P=True))
        ctx.close()
    assert np.abs(out[0]["psi"]).max() >= 8.0 ** -1.5  # the mean amplitude of one electron in the box
    for f in ("psi", "P"):
        assert np.array_equal(out[0][f], out[1][f])
