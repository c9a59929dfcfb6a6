"""One-block scans and species permutation and the chunked structure sums on
both sides of the sizes where they give way to the many-block forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(n, seed):
    """n atoms of 2 species on a jittered cubic grid, spacing 2.6 A."""
    r = np.random.Generator(np.random.PCG64(seed))
    k = int(np.ceil(n ** (1 / 3) - 1e-9))
    site = np.arange(n)
    grid = np.stack(np.unravel_index(site, (k, k, k)), 1)
    pos = grid * 2.6 + r.uniform(-0.2, 0.2, size=(n, 3))
    return np.eye(3) * 2.6 * k, r.integers(2, size=n), pos


@pytest.mark.parametrize("n", [1, 1023, 1025, 2048, 2049, 8192, 8193, 20001])
def test_sizes_around_the_one_block_forms(n):
    """A structure alone and after another of 700 atoms in one batch: the same
    bits, and the energies add up to the per-atom sum of the same model."""
    import flare_gb300 as fg
    calc = fg.B2("chebyshev", "quadratic", [0.0, 3.5], [], [2, 3, 2])
    r = np.random.Generator(np.random.PCG64(1))
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = 2, calc.n_descriptors
    dv.descriptors = [r.normal(size=(m, calc.n_descriptors)) + 1.0
                      for m in (5, 3)]
    dv.descriptor_norms = [np.linalg.norm(d, axis=1) for d in dv.descriptors]
    dv.n_clusters_by_type = [5, 3]
    gp = fg.SparseGP([fg.NormalizedDotProduct(1.5, 2)], 0.1, 0.1, 0.1)
    alpha = r.normal(size=8)
    gp.set_weights([fg.ClusterDescriptor.from_values(dv)], alpha,
                   np.eye(8) * 0.1, [calc])
    cell, sp, pos = lattice(n, n)
    one = fg.Structure(cell, sp, pos, 3.5, [calc])
    for prec in ("fp64", "mixed"):
        a = gp.predict_batch([one], precision=prec)
        b = gp.predict_batch([fg.Structure(*lattice(700, 9), 3.5, [calc]), one],
                             precision=prec)
        assert a["energy"][0] == b["energy"][1]
        assert np.array_equal(a["forces"], b["forces"][700:])
        assert np.array_equal(a["stress"][0], b["stress"][1])
        assert np.array_equal(a["local_var"], b["local_var"][700:])
        # forces of a periodic structure add up to zero
        assert np.abs(a["forces"].sum(0)).max() <= \
            (1e-12 if prec == "fp64" else 1e-5) * np.abs(a["forces"]).sum() + 1e-300
    B, norm = one.b2_values()
    B = B.cpu().numpy() / norm.cpu().numpy()[:, None]
    e, at = 0.0, 0
    for s, d in enumerate(dv.descriptors):
        c = B[sp == s] @ (d / dv.descriptor_norms[s][:, None]).T
        e += 1.5 ** 2 * (c ** 2 @ alpha[at:at + len(d)]).sum()
        at += len(d)
    a = gp.predict_batch([one], precision="fp64")
    assert abs(a["energy"][0] - e) <= 1e-12 * n * np.abs(alpha).sum() * 2.25
