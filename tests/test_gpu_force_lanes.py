"""FP64 forces and stress with neighbour counts around the sixteen lanes that
share an atom's pairs, against the oracle on the same weights."""
import numpy as np
import pytest

import oracle
from test_gpu_fp64_stage import weighted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33])
def test_neighbour_counts_around_the_lanes(n):
    import flare_gb300 as fg
    ogp, gp, calc, args = weighted((9, 5), 3, 2, 2, seed=n)
    r = np.random.Generator(np.random.PCG64(n))
    u = r.normal(size=(n + 1, 3))
    u *= (1.9 * r.uniform(0.2, 1.0, size=(n + 1, 1)) ** (1 / 3)
          / np.linalg.norm(u, axis=1)[:, None])
    # n + 1 atoms within reach of one another, and one atom alone
    pos = np.concatenate([u + 10.0, [[25.0, 25.0, 25.0]]])
    cell, sp = np.eye(3) * 35.0, r.integers(2, size=n + 2)
    st = oracle.Structure(cell, sp, pos, 4.0, [oracle.B2Settings(*args)])
    ogp.predict_local_uncertainties(st)
    m = st.mean_efs
    g = gp.predict_batch([fg.Structure(cell, sp, pos, 4.0, [calc])],
                         precision="fp64")
    f = m[1:-6].reshape(-1, 3)
    # as in the FP64 stage's own tests
    assert np.abs(g["forces"] - f).max() <= 1e-11 * max(1.0, np.abs(f).max())
    assert np.abs(g["stress"][0] - m[-6:]).max() <= \
        1e-11 * max(1.0, np.abs(m[-6:]).max())
    assert not g["forces"][-1].any()
