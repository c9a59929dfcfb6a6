"""Pairs with shifts along no, one, two or three cell axes, in cells with and
without zero components: the list against the oracle's, bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reps", [(6, 6, 6), (9, 2, 1), (1, 7, 2), (1, 1, 1)])
@pytest.mark.parametrize("shear", [
    np.zeros((3, 3)),
    np.array([[0, 0, 0], [-0.3, 0, 0], [0, 0, 0]]),
    np.array([[0, 0.2, 0], [0, 0, -0.25], [0.1, 0, 0]]),
])
def test_list_bit_exact(reps, shear):
    import flare_gb300 as fg
    r = np.random.Generator(np.random.PCG64(sum(reps)))
    grid = np.stack(np.meshgrid(*map(np.arange, reps), indexing="ij"), -1)
    frac = (grid.reshape(-1, 3) + r.uniform(0.0, 0.2, size=(grid.size // 3, 3)))
    unit = 2.5 * (np.eye(3) + shear)
    cell = unit * np.asarray(reps)[:, None]
    pos = frac @ unit
    sp = np.zeros(len(pos), int)
    o = oracle.Structure(cell, sp, pos, 4.0, [])
    a = fg.Structure(cell, sp, pos, 4.0, []).neighbor_arrays()
    np.testing.assert_array_equal(a["neighbor_count"], o.neighbor_count)
    np.testing.assert_array_equal(a["structure_indices"], o.structure_indices)
    np.testing.assert_array_equal(a["shifts"], o.shifts)
    np.testing.assert_array_equal(a["relative_positions"], o.relative_positions)
