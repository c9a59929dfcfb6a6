"""envs_envs put together from species blocks: one block that is the whole
matrix, blocks on the host and on the device, species without rows in one or
both sets, and two sets without a species in common."""
import numpy as np
import pytest

import oracle
from test_gpu_stored_gradients import cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c1,c2", [
    ((40, 0), (25, 0)),                # one block, all of it
    ((0, 300), (0, 280)),
    ((40, 0), (25, 3)),                # one block, zeros beside it
    ((5, 40, 3), (25, 0, 60)),         # on the host
    ((128, 128), (128, 128)),          # 2^16 entries: still on the host
    ((128, 129), (128, 128)),          # on the device
    ((150, 0, 200), (100, 90, 120)),
    ((12, 0), (0, 7)),                 # nothing in common
    ((300, 0), (0, 300)),
])
def test_blocks(c1, c2):
    import flare_gb300 as fg
    a, b = cluster(c1, 30, seed=1), cluster(c2, 30, seed=2)
    K0 = oracle.NormalizedDotProduct(2.0, 2).envs_envs(a, b)
    K1 = fg.NormalizedDotProduct(2.0, 2).envs_envs(a, b)
    assert K1.shape == K0.shape and K1.flags.writeable
    # |k| <= sigma^2 and each dot product rounds by at most n_d ulp
    assert np.abs(K1 - K0).max() <= 4 * 2 * 30 * 4.0 * 2.3e-16
    assert not K1[K0 == 0.0].any()
