"""The small levels of a V(1,1) cycle in one block, forward and transposed, in tails of two, three and four levels
(the default hierarchies end in two; mg_levels gives longer ones), against the FP64 oracle: 1e-12 of the largest
value forward after a few steps, 1e-9 for the reverse sweep, as for the level-by-level kernels."""
import numpy as np
import pytest

import nm_adjoint as adj
import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NN,levels,steps", [(24, None, 9), (32, None, 9), (48, None, 5), (56, None, 5), (24, 4, 8), (32, 4, 8),
                                             (32, 5, 8), (64, 6, 5)])
def test_tail_matches_the_oracle(NN, levels, steps):
    from realmolecule_b200 import Context
    h = 7.2 / NN
    N2, d = NN / 2, 1.4 / 2 / h
    rows = [{"i": N2 - d, "j": N2, "k": N2 + 0.2, "Z": 0.0, "Z_nuc": 1.0},
            {"i": N2 + d, "j": N2 + 0.3, "k": N2, "Z": 0.0, "Z_nuc": 1.0},
            {"i": N2 - d + 0.05, "j": N2, "k": N2, "Z": 1.0, "Z_nuc": 0.0},
            {"i": N2 + d - 0.05, "j": N2, "k": N2, "Z": 1.0, "Z_nuc": 0.0}]
    drv = orc.NewMethodDriver(NN, NN * h, rows, label_until=1, poisson_interval=2, levels=levels)
    drv.initialize()
    ctx = Context(NN, NN * h, rows, flavor="new", precision="fp64", label_until=1, poisson_interval=2, mg_levels=levels)
    ctx.initialize()
    assert ctx.info().mg_levels == drv.levels
    ctx.upload(psi=drv.U, label=drv.label, P=drv.P)
    ctx.set_adjoint_window(steps)
    ctx.step(steps)
    F, g = ctx.adjoint(forces=True, potential=True)
    st = ctx.download(psi=True, label=False, P=True)
    ctx.close()
    _, Fo, go = adj.gradient(drv, steps)
    assert np.abs(st["psi"] - drv.U).max() <= 1e-12 * np.abs(drv.U).max()
    assert np.abs(st["P"] - drv.P).max() <= 1e-12 * np.abs(drv.P).max()
    Fo, go = np.asarray(Fo), np.asarray(go)
    assert np.abs(F - Fo).max() <= 1e-9 * np.abs(Fo).max()
    assert np.abs(g - go.ravel()).max() <= 1e-9 * np.abs(go).max()
