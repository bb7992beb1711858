"""molecule.js's direct per-electron Poisson with one launch's worth of domains, one more, and the fewest, bit for bit
against the C restatement."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NN", [8, 18])
@pytest.mark.parametrize("domains", [2, 4, 5])
@pytest.mark.parametrize("opts,steps", [(dict(steps_per_frame=3), 4), (dict(steps_per_frame=2, lobpcg=True), 2)])
def test_domains_per_launch(NN, domains, opts, steps):
    from realmolecule_b200 import Context
    c = NN // 2
    at = [(c, c, c, 2, 0.3), (c + 1, c + 1, c, 1, 0.0), (c - 1, c, c - 1, 1, 0.0), (c, c - 2, c + 1, 1, 0.0), (c + 2, c, c - 1, 1, 0.0)]
    rows = [{"i": i, "j": j, "k": k, "Z": z, "Z_nuc": z, "rc": rc} for i, j, k, z, rc in at[:domains]]
    ref = orc.MoleculeJsDriver(NN, NN * 0.25, rows, sic=True, **opts)
    ref.initialize()
    ctx = Context(NN, NN * 0.25, rows, flavor="molecule.js", sic=1, **{k: int(v) for k, v in opts.items()})
    ctx.initialize()
    ctx.upload(psi=ref.U, label=ref.label.astype(np.int32))
    for _ in range(steps):
        ref.step()
    ctx.step(steps)
    st = ctx.download(psi=True, label=True, W=True, P=True)
    ctx.close()
    assert np.array_equal(st["psi"].view(np.uint32), ref.U.view(np.uint32))
    assert np.array_equal(st["label"] & 0x3FFFFFFF, ref.label.astype(np.int32))
    assert np.array_equal(st["W"].view(np.uint32), ref.W.view(np.uint32))
    assert np.array_equal(st["P"].view(np.uint32), ref.P.view(np.uint32))
