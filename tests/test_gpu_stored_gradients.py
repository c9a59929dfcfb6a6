"""The stored-gradient kernels (envs_struc, envs_envs) at the edges of their
blocks: a last block of fewer than eight pairs, descriptors whose pair basis
takes two pairs a block, sparse counts around 32, 48 and 128, species without
sparse rows, powers 1, 2 and 3; against the FP64 oracle."""
import numpy as np
import pytest

import oracle
from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def cluster(counts, n_d, seed):
    import flare_gb300 as fg
    r = np.random.Generator(np.random.PCG64(seed))
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = len(counts), n_d
    dv.descriptors = [r.normal(size=(n, n_d)) + 0.5 for n in counts]
    dv.descriptor_norms = [np.linalg.norm(d, axis=1) for d in dv.descriptors]
    dv.n_clusters_by_type = list(counts)
    return fg.ClusterDescriptor.from_values(dv)


@pytest.mark.parametrize("atoms,counts,nmax,lmax,power", [
    (3, (1, 2), 3, 2, 2),
    (41, (31, 33), 3, 2, 2),
    (70, (0, 49), 4, 3, 1),
    (60, (129, 16), 3, 1, 3),
    (12, (5, 4), 12, 9, 2),       # two pairs a block, runtime l_max
])
def test_envs_struc_block_edges(atoms, counts, nmax, lmax, power):
    import flare_gb300 as fg
    rc = 4.0
    args = ("chebyshev", "quadratic", [0.0, rc], [], [2, nmax, lmax])
    calc = fg.B2(*args)
    cd = cluster(counts, calc.n_descriptors, seed=atoms)
    cell, sp, pos = syn.random_alloy(atoms, density=0.05, dmin=1.6,
                                     seed=300 + atoms)
    sp[:2] = (0, 1)
    o = oracle.Structure(cell, sp, pos, rc, [oracle.B2Settings(*args)])
    K0 = oracle.NormalizedDotProduct(1.5, power).envs_struc(cd,
                                                            o.descriptors[0])
    K1 = fg.NormalizedDotProduct(1.5, power).envs_struc(
        cd, fg.Structure(cell, sp, pos, rc, [calc]))
    # columns are sums over up to all pairs of products with n_d-term dots
    assert K1.shape == K0.shape
    assert np.abs(K1 - K0).max() <= 1e-11 * np.abs(K0).max()


@pytest.mark.parametrize("n1,n2,n_d,power", [
    (1, 1, 10, 2), (33, 127, 144, 2), (48, 49, 680, 1), (129, 32, 1500, 3)])
def test_envs_envs_block_edges(n1, n2, n_d, power):
    import flare_gb300 as fg
    a, b = cluster((n1, 0), n_d, seed=n1), cluster((n2, 3), n_d, seed=n2 + 7)
    K0 = oracle.NormalizedDotProduct(2.0, power).envs_envs(a, b)
    K1 = fg.NormalizedDotProduct(2.0, power).envs_envs(a, b)
    # |k| <= sigma^2 and each dot product rounds by at most n_d ulp
    assert np.abs(K1 - K0).max() <= 4 * power * n_d * 4.0 * 2.3e-16
