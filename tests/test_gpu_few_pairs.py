"""k_b2_dervs takes four pairs a block while four centres' A and gradients fit
in 48 kB, else one (launch_b2_dervs).  A structure has an even number of
pairs, so a last block has four or two: both, alone and after a full block, and
the one-pair form, against the FP64 oracle."""
import numpy as np
import pytest

import oracle
from test_gpu_stored_gradients import cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dimers", [1, 2, 3, 4])
@pytest.mark.parametrize("nmax,lmax", [
    (3, 2),     # 4 pairs: 1.1 kB each
    (8, 4),     # 4 pairs: 8.0 kB each
    (12, 5),    # 1 pair: 17.8 kB each, run-time l_max
])
def test_pair_counts(dimers, nmax, lmax):
    import flare_gb300 as fg
    rc = 4.0
    args = ("chebyshev", "quadratic", [0.0, rc], [], [2, nmax, lmax])
    calc = fg.B2(*args)
    cd = cluster((7, 5), calc.n_descriptors, seed=dimers)
    r = np.random.Generator(np.random.PCG64(10 * dimers + nmax))
    at = np.repeat(np.arange(dimers), 2)[:, None] * [11.0, 0.0, 0.0]
    pos = at + r.uniform(0.0, 2.0, size=(2 * dimers, 3))
    cell, sp = np.eye(3) * 50.0, np.tile([0, 1], dimers)
    g = fg.Structure(cell, sp, pos, rc, [calc])
    assert g.n_neighbors == 2 * dimers
    o = oracle.Structure(cell, sp, pos, rc, [oracle.B2Settings(*args)])
    K0 = oracle.NormalizedDotProduct(1.5, 2).envs_struc(cd, o.descriptors[0])
    K1 = fg.NormalizedDotProduct(1.5, 2).envs_struc(cd, g)
    # columns are sums over all pairs of products with n_d-term dots
    assert np.abs(K1 - K0).max() <= 1e-11 * np.abs(K0).max()
