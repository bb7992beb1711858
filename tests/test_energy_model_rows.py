"""EnergyModel's atom table takes and refuses the shapes that its rows did one by one."""
import numpy as np
import pytest

from realmolecule_b200.autograd import EnergyModel


def _model(n_nuc, seeds):
    m = EnergyModel.__new__(EnergyModel)
    m.h, m.n_nuc, m.charges, m.seeds = 0.2, n_nuc, np.full(n_nuc, 2.0), np.asarray(seeds, np.float64)
    return m


@pytest.mark.parametrize("pos,seeds", [(np.ones((2, 1)), np.ones((3, 3))), (np.ones((2, 2)), np.ones((3, 3))), (np.ones(2), []),
                                       (np.ones((2, 3)), np.ones((3, 1))), (np.ones((2, 3)), np.ones((3, 2))),
                                       (np.ones((2, 3)), np.ones(3))])
def test_rows_without_three_coordinates_are_refused(pos, seeds):
    with pytest.raises(IndexError):
        _model(2, seeds)._rows(pos)


@pytest.mark.parametrize("pos,seeds,n", [(np.ones((2, 3)), np.ones((3, 3)), 5), (np.ones((2, 5)), np.ones((3, 4)), 5),
                                         (np.ones((4, 3)), [], 2), (np.ones((1, 3)), [], 1), (np.ones((0, 3)), [], 0)])
def test_rows_taken(pos, seeds, n):
    assert len(_model(2, seeds)._rows(pos)) == n
