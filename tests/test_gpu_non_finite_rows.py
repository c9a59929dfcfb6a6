"""Descriptors that overflow to infinity: the energies, forces and variances
of their atoms are NaN, as the general FP64 path gives them, and the other
atoms keep their values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RC = 4.0   # cutoff function (RC - r)^600: 1 at r = 3, 4e180 at r = 2
GOOD = [[0.0, 0, 0], [3.0, 0, 0]]
BAD = [[0.0, 20, 0], [2.0, 20, 0]]


def model(M, power):
    import flare_gb300 as fg
    calc = fg.B2("chebyshev", "power", [0.0, RC], [600.0], [1, 3, 2])
    r = np.random.Generator(np.random.PCG64(M))
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = 1, calc.n_descriptors
    dv.descriptors = [r.normal(size=(M, calc.n_descriptors)) + 0.5]
    dv.descriptor_norms = [np.linalg.norm(dv.descriptors[0], axis=1)]
    dv.n_clusters_by_type = [M]
    cd = fg.ClusterDescriptor.from_values(dv)
    gp = fg.SparseGP([fg.NormalizedDotProduct(1.5, power)], 0.1, 0.1, 0.1)
    gp.set_weights([cd], r.normal(size=M),
                   np.tril(r.normal(size=(M, M))) * 0.1, [calc])
    return gp, calc, cd


def structure(calc, pos):
    import flare_gb300 as fg
    return fg.Structure(np.eye(3) * 40.0, [0] * len(pos), np.array(pos), RC,
                        [calc])


# power 3 takes the general path; 20 and 400 rows the two forms of variances
@pytest.mark.parametrize("power", [1, 2, 3])
@pytest.mark.parametrize("M", [20, 400])
def test_predictions(M, power):
    gp, calc, _ = model(M, power)
    good, both = structure(calc, GOOD), structure(calc, GOOD + BAD)
    B, norm = both.b2_values()
    assert bool((norm[2:] == float("inf")).all())   # not NaN: not "empty"
    a = gp.predict_batch([good], precision="fp64")
    b = gp.predict_batch([both, good], precision="fp64")
    assert np.isfinite(a["energy"]).all() and np.isfinite(a["local_var"]).all()
    assert np.isnan(b["energy"][0]) and b["energy"][1] == a["energy"][0]
    assert np.isnan(b["local_var"][2:4]).all()
    assert np.isnan(b["forces"][2:4, 0]).all()
    for at in (0, 4):
        assert np.array_equal(b["local_var"][at:at + 2], a["local_var"])
        assert np.array_equal(b["forces"][at:at + 2], a["forces"])


@pytest.mark.parametrize("power", [1, 2, 3])
def test_stored_gradients(power):
    import flare_gb300 as fg
    _, calc, cd = model(40, power)
    k = fg.NormalizedDotProduct(1.5, power)
    K = k.envs_struc(cd, structure(calc, GOOD + BAD))
    G = k.envs_struc(cd, structure(calc, GOOD))
    assert np.isfinite(G).all()
    assert np.isnan(K[:, 0]).all()
    assert np.array_equal(K[:, 1:7], G[:, 1:7])
    assert np.isnan(K[:, [7, 10]]).all()   # x forces of the overflowed pair


def test_sparse_rows():
    """An infinite entry makes its row of the kernel matrix NaN, a norm that
    overflows makes it zero (finite over infinite); the others stay."""
    import flare_gb300 as fg
    _, calc, cd = model(40, 2)
    k, st = fg.NormalizedDotProduct(1.5, 2), structure(calc, GOOD)
    K = k.envs_struc(cd, st)
    cd.descriptors[0][7, 3] = np.inf
    cd.descriptors[0][9, 3] = 1e200
    G = k.envs_struc(cd, st)
    assert np.isnan(G[7, 0]) and np.isnan(G[7, 1]) and np.isnan(G[7, 4])
    assert (G[9] == 0.0).all()
    keep = np.delete(np.arange(40), [7, 9])
    assert np.array_equal(G[keep], K[keep])
