"""Descriptors evaluated half a chunk (32 pairs) at a time, at neighbour counts
around the half (32) and the whole chunk (64): FP64 against the oracle, and the
double-float ones through the energy of a mixed-precision prediction."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 96, 97, 130])
def test_neighbour_counts_around_the_halves(n):
    import flare_gb300 as fg
    r = np.random.Generator(np.random.PCG64(n))
    # n + 1 atoms within reach of one another, one atom alone, and a pair
    # whose distance is beyond the cutoff
    u = r.normal(size=(n + 1, 3))
    u *= (2.4 * r.uniform(size=(n + 1, 1)) ** (1 / 3)
          / np.linalg.norm(u, axis=1)[:, None])
    pos = np.concatenate([u + 10.0, [[30.0, 30.0, 30.0]]])
    cell, sp = np.eye(3) * 40.0, np.zeros(n + 2, int)
    args = ("chebyshev", "quadratic", [0.0, 5.0], [], [1, 10, 6])
    o = oracle.Structure(cell, sp, pos, 5.0, [oracle.B2Settings(*args)],
                         compute_dervs=False)
    calc = fg.B2(*args)
    st = fg.Structure(cell, sp, pos, 5.0, [calc])
    assert st.n_neighbors == n * (n + 1)
    B, norm = st.b2_values()
    ob = o.descriptors[0].atom_B2
    np.testing.assert_allclose(B.cpu().numpy(), ob, rtol=1e-11,
                               atol=1e-12 * np.abs(ob).max())
    np.testing.assert_allclose(norm.cpu().numpy(), o.descriptors[0].atom_norms,
                               rtol=1e-12)
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = 1, calc.n_descriptors
    dv.descriptors = [r.normal(size=(7, calc.n_descriptors)) + 1.0]
    dv.descriptor_norms = [np.linalg.norm(dv.descriptors[0], axis=1)]
    dv.n_clusters_by_type = [7]
    gp = fg.SparseGP([fg.NormalizedDotProduct(1.5, 2)], 0.1, 0.1, 0.1)
    gp.set_weights([fg.ClusterDescriptor.from_values(dv)], r.normal(size=7),
                   np.eye(7) * 0.1, [calc])
    a = gp.predict_batch([st], precision="fp64")
    b = gp.predict_batch([st], precision="mixed")
    assert abs(a["energy"][0] - b["energy"][0]) <= 1e-6 * (n + 2)
