"""Non-finite entries of a model's weights, wherever they stand: the variances
that they belong to are not finite."""
import numpy as np
import pytest

from test_gpu_fp64_stage import RC, weighted
from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [(0, 0), (39, 0), (39, 39), (40, 40), (56, 49)])
@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf])
def test_L_inv(at, value):
    import flare_gb300 as fg
    _, gp, calc, _ = weighted((40, 17), 3, 2, 2, seed=5)
    cell, sp, pos = syn.random_alloy(20, density=0.05, dmin=1.6, seed=7)
    st = fg.Structure(cell, sp, pos, RC, [calc])
    whole = gp.predict_batch([st], precision="fp64")
    L = gp.L_inv.copy()
    L[at] = value
    gp.set_weights(gp.sparse_descriptors, gp.alpha, L, [calc])
    r = gp.predict_batch([st], precision="fp64")
    hit = np.asarray(sp) == (0 if at[1] < 40 else 1)
    assert not np.isfinite(r["local_var"][hit]).any()
    np.testing.assert_allclose(r["local_var"][~hit], whole["local_var"][~hit],
                               rtol=0, atol=1e-12 * 2.25)
