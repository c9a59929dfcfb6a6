"""The structure sums where a large structure meets very many small ones."""
import numpy as np
import pytest

from test_gpu_small_kernels import lattice

pytestmark = pytest.mark.gpu


def potential(rc=3.5):
    import flare_gb300 as fg
    calc = fg.B2("chebyshev", "quadratic", [0.0, rc], [], [2, 3, 2])
    r = np.random.Generator(np.random.PCG64(1))
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = 2, calc.n_descriptors
    dv.descriptors = [r.normal(size=(m, calc.n_descriptors)) + 1.0
                      for m in (5, 3)]
    dv.descriptor_norms = [np.linalg.norm(d, axis=1) for d in dv.descriptors]
    dv.n_clusters_by_type = [5, 3]
    gp = fg.SparseGP([fg.NormalizedDotProduct(1.5, 2)], 0.1, 0.1, 0.1)
    gp.set_weights([fg.ClusterDescriptor.from_values(dv)], r.normal(size=8),
                   np.eye(8) * 0.1, [calc])
    return gp, calc


@pytest.mark.parametrize("sizes", [
    (2049, 0, 1, 4096, 2047),          # chunk edges, an empty one between
    (1, 2048, 6145, 0, 0, 3),          # empty ones at the end of a chunk
    (0, 4097, 0),
])
def test_sums_do_not_depend_on_the_batch(sizes):
    import flare_gb300 as fg
    gp, calc = potential()
    strucs = [fg.Structure(*lattice(n, 10 + n), 3.5, [calc]) if n else
              fg.Structure(np.eye(3) * 4.0, [], np.zeros((0, 3)), 3.5, [calc])
              for n in sizes]
    both = gp.predict_batch(strucs, precision="fp64")
    for k, s in enumerate(strucs):
        one = gp.predict_batch([s], precision="fp64")
        assert one["energy"][0] == both["energy"][k]
        assert np.array_equal(one["stress"][0], both["stress"][k])


def test_memory_follows_atoms_plus_structures():
    """97,336 atoms (48 chunks) with one empty structure, then with 40,000:
    the second call adds a list entry for each of them (below 1 kB) and no
    row of 48 partial sums (107 MB)."""
    import torch
    import flare_gb300 as fg
    gp, calc = potential()
    big = fg.Structure(*lattice(97336, 1), 3.5, [calc])
    none = fg.Structure(np.eye(3) * 4.0, [], np.zeros((0, 3)), 3.5, [calc])
    a = gp.predict_batch([big, none])
    free = torch.cuda.mem_get_info()[0]
    b = gp.predict_batch([big] + [none] * 40000)
    assert free - torch.cuda.mem_get_info()[0] < 64 << 20
    assert a["energy"][0] == b["energy"][0]
    assert np.array_equal(a["stress"][0], b["stress"][0])
    assert not b["energy"][1:].any() and not b["stress"][1:].any()
