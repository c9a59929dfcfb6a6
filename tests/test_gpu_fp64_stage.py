"""The FP64 path's kernel stage (exact 10-slice products) at the edges of its
tiles: 128-row blocks of atoms, B tiles of 32 and 48 rows, 16-deep k chunks
and a second K segment, against the FP64 oracle on the same weights."""
import numpy as np
import pytest

import oracle
from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

RC = 4.0


def weighted(counts, nmax, lmax, power, seed):
    """(oracle GP, GPU GP, calculator, B2 arguments) with random sparse rows,
    alpha and lower-triangular L_inv blocks per species."""
    import flare_gb300 as fg
    S = len(counts)
    args = ("chebyshev", "quadratic", [0.0, RC], [], [S, nmax, lmax])
    calc = fg.B2(*args)
    r = np.random.Generator(np.random.PCG64(seed))
    dv = fg.DescriptorValues()
    dv.n_types, dv.n_descriptors = S, calc.n_descriptors
    dv.descriptors = [r.normal(size=(n, calc.n_descriptors)) + 0.5
                      for n in counts]
    dv.descriptor_norms = [np.linalg.norm(d, axis=1) for d in dv.descriptors]
    dv.n_clusters_by_type = list(counts)
    cd = fg.ClusterDescriptor.from_values(dv)
    M = sum(counts)
    alpha, L = r.normal(size=M), np.zeros((M, M))
    at = 0
    for n in counts:
        L[at:at + n, at:at + n] = np.tril(r.normal(size=(n, n))) * 0.1
        at += n
    gp = fg.SparseGP([fg.NormalizedDotProduct(1.5, power)], 0.1, 0.1, 0.1)
    gp.set_weights([cd], alpha, L, [calc])
    ogp = oracle.SparseGP.from_weights(
        [oracle.NormalizedDotProduct(1.5, power)], [cd], alpha, L)
    return ogp, gp, calc, args


@pytest.mark.parametrize("atoms,counts,nmax,lmax,power", [
    (2, (1, 1), 3, 2, 2),          # one row, one column
    (64, (31, 16), 3, 2, 2),       # below a tile, a whole chunk
    (127, (33, 0), 4, 1, 2),       # a species without sparse rows
    (257, (48, 49), 3, 2, 1),      # power 1, tile edge and one above
    (300, (97, 128), 4, 2, 2),     # two row blocks
    (40, (1400, 7), 2, 1, 2),      # K above one segment (1,360)
])
def test_fp64_stage_matches_oracle(atoms, counts, nmax, lmax, power):
    import flare_gb300 as fg
    ogp, gp, calc, args = weighted(counts, nmax, lmax, power, seed=atoms)
    cell, sp, pos = syn.random_alloy(atoms, density=0.05, dmin=1.6,
                                     seed=900 + atoms)
    sp[:2] = (0, 1)
    st = oracle.Structure(cell, sp, pos, RC, [oracle.B2Settings(*args)])
    ogp.predict_local_uncertainties(st)
    var = oracle.sort_variances(st, st.local_uncertainties[0])
    r = gp.predict_batch([fg.Structure(cell, sp, pos, RC, [calc])],
                         precision="fp64")
    m = st.mean_efs
    # each energy and variance sums up to max(counts) products of size
    # |alpha| sigma^2 (|z|^2), with rounding errors of a few ulp in each
    # kernel value (n_d-term dot products on the oracle's side)
    eps = np.finfo(float).eps
    scale = np.abs(gp.alpha).sum() * 1.5 ** 2 * atoms
    assert abs(r["energy"][0] - m[0]) <= 64 * eps * scale
    f = m[1:-6].reshape(-1, 3)
    assert np.abs(r["forces"] - f).max() <= 1e-11 * max(1.0, np.abs(f).max())
    assert np.abs(r["stress"][0] - m[-6:]).max() <= \
        1e-11 * max(1.0, np.abs(m[-6:]).max())
    assert np.abs(r["local_var"] - var).max() <= \
        1e-12 * max(1.0, np.abs(var).max())


def test_fp64_stage_keeps_nan_weights():
    """A NaN among alpha comes through as NaN energies (the general path)."""
    import flare_gb300 as fg
    _, gp, calc, _ = weighted((8, 8), 3, 2, 2, seed=5)
    gp.alpha = gp.alpha.copy()
    gp.alpha[3] = np.nan
    gp._model = None
    cell, sp, pos = syn.random_alloy(20, density=0.05, dmin=1.6, seed=7)
    r = gp.predict_batch([fg.Structure(cell, sp, pos, RC, [calc])],
                         precision="fp64")
    assert np.isnan(r["energy"][0])
