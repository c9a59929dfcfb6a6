"""Products of several species in one launch (all atoms within one chunk of
32,768 rows) against the oracle, and against a species at a time."""
import numpy as np
import pytest

from test_gpu_fp64_stage import weighted
from test_gpu_small_kernels import lattice

import oracle
from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,counts", [
    (64, (5, 130, 49)),        # three species, uneven tiles
    (200, (16, 0, 33)),        # one without sparse rows between two with
    (150, (1, 2, 3, 4, 5, 6, 7, 8)),   # the most species
    (40, (1400, 7)),           # K above one segment beside K of one chunk
])
def test_groups_match_oracle(atoms, counts):
    import flare_gb300 as fg
    ogp, gp, calc, args = weighted(counts, 3, 2, 2, seed=atoms + 1)
    S = len(counts)
    cell, sp, pos = syn.random_alloy(atoms, fractions=[1.0 / S] * S,
                                     density=0.05, dmin=1.6, seed=70 + atoms)
    sp[:S] = np.arange(S)
    st = oracle.Structure(cell, sp, pos, 4.0, [oracle.B2Settings(*args)])
    ogp.predict_local_uncertainties(st)
    var = oracle.sort_variances(st, st.local_uncertainties[0])
    r = gp.predict_batch([fg.Structure(cell, sp, pos, 4.0, [calc])],
                         precision="fp64")
    m = st.mean_efs
    # sums of up to 1,400 terms of FP64 level
    assert abs(r["energy"][0] - m[0]) <= 1e-10 * max(1.0, abs(m[0]))
    f = m[1:-6].reshape(-1, 3)
    np.testing.assert_allclose(r["forces"], f, rtol=0,
                               atol=1e-10 * max(1.0, np.abs(f).max()))
    np.testing.assert_allclose(r["local_var"], var, rtol=0,
                               atol=1e-10 * max(1.0, np.abs(var).max()))


def test_a_group_and_a_species_at_a_time_agree():
    """32,768 atoms in one call (grouped) and the same beside 700 more (a
    species at a time): the same bits."""
    import flare_gb300 as fg
    _, gp, calc, _ = weighted((20, 33), 3, 2, 2, seed=5)
    big = fg.Structure(*lattice(32768, 1), 4.0, [calc])
    more = fg.Structure(*lattice(700, 2), 4.0, [calc])
    a = gp.predict_batch([big], precision="fp64")
    b = gp.predict_batch([big, more], precision="fp64")
    assert a["energy"][0] == b["energy"][0]
    assert np.array_equal(a["forces"], b["forces"][:32768])
    assert np.array_equal(a["stress"][0], b["stress"][0])
    assert np.array_equal(a["local_var"], b["local_var"][:32768])


@pytest.mark.parametrize("atoms,M", [
    (8, 400), (1500, 400), (6000, 400),    # slices
    (1, 1), (9, 63), (8, 130), (33, 65), (1500, 130),   # the SIMT order
])
def test_triangular_operand_in_blocks(atoms, M):
    """What L_inv holds above its diagonal counts inside the 64-row diagonal
    blocks and nowhere else, whatever the tile height (16, 32 or 48 rows) and
    on both sides of the size (about 340 sparse rows here) where the variance
    product moves to the slices."""
    import flare_gb300 as fg
    _, gp, calc, _ = weighted((M,), 3, 2, 2, seed=9)
    r = np.random.Generator(np.random.PCG64(atoms))
    L = r.normal(size=(M, M)) * 0.1
    gp.set_weights(gp.sparse_descriptors, gp.alpha, L, [calc])
    cell, _, pos = lattice(atoms, 3)
    st = fg.Structure(cell, np.zeros(atoms, int), pos, 4.0, [calc])
    B, n = (x.cpu().numpy() for x in st.b2_values())
    d = gp.sparse_descriptors[0].descriptors[0]
    c = (B / n[:, None]) @ (d / np.linalg.norm(d, axis=1)[:, None]).T
    block = np.arange(M) // 64
    z = 1.5 ** 2 * c ** 2 @ (L * (block[None, :] <= block[:, None])).T
    want = 1.5 ** 2 - (z * z).sum(1)
    var = gp.predict_batch([st], precision="fp64")["local_var"]
    # sums of 130 products of FP64 level, squared and summed
    np.testing.assert_allclose(var, want, rtol=0,
                               atol=1e-12 * np.abs(want).max())
