"""Hierarchies down to levels of two and one intervals (mg_levels), whose small levels run as kernels (two sweeps on a
side), alone and in a batch, against the FP64 oracle: 1e-12 of the largest value; fp32 fields against the FP64 ones
at their resolution."""
import numpy as np
import pytest

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NN,levels", [(16, 4), (16, 5), (32, 5), (32, 6), (24, 4)])
def test_deep_hierarchies(NN, levels):
    from realmolecule_b200 import Context
    from realmolecule_b200.batch import Batch
    h = 7.2 / NN
    c = NN / 2
    rows = [{"i": c, "j": c, "k": c + 0.2, "Z": 0.0, "Z_nuc": 2.0}, {"i": c - 0.6, "j": c, "k": c, "Z": 1.0, "Z_nuc": 0.0},
            {"i": c + 0.6, "j": c, "k": c, "Z": 1.0, "Z_nuc": 0.0}]
    kw = dict(label_until=1, poisson_interval=2, mg_levels=levels)
    drv = orc.NewMethodDriver(NN, NN * h, rows, label_until=1, poisson_interval=2, levels=levels, pre=2)
    drv.initialize()
    for _ in range(6):
        drv.step()
    drv.state()
    got = {}
    for prec in ("fp64", "mixed"):
        ctx = Context(NN, NN * h, rows, flavor="new", precision=prec, mg_pre=2, **kw)
        ctx.initialize()
        ctx.step(6)
        got[prec] = ctx.download(psi=True, label=False, P=True)
        if NN >> (levels - 1) > 1:
            b = Batch([{"NN": NN, "screen": NN * h, "atoms": rows}], precision=prec, mg_pre=2, **kw)
            b.initialize()
            b.step(6)
            assert np.abs(b.energy()[0] - ctx.energy()).max() <= (1e-11 if prec == "fp64" else 1e-4)
            b.close()
        ctx.close()
    assert np.abs(got["fp64"]["P"] - drv.P).max() <= 1e-12 * np.abs(drv.P).max()
    assert np.abs(got["fp64"]["psi"] - drv.U).max() <= 1e-12 * np.abs(drv.U).max()
    assert np.abs(got["mixed"]["P"] - drv.P).max() <= 1e-5 * np.abs(drv.P).max()
