"""FP64 variances of models with few sparse environments are those of the
SIMT products to the bit: a prediction (k_kernel_small, k_variance_small)
against the stored-gradient form's local variances (k_kernel_gemm,
k_variance_gemm) on the same descriptors."""
import numpy as np
import pytest

from test_gpu_fp64_stage import weighted
from test_gpu_small_kernels import lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [1, 2])
@pytest.mark.parametrize("atoms,counts", [
    (1, (1, 2)), (7, (8, 15)), (8, (9, 16)), (9, (17, 31)), (16, (32, 33)),
    (33, (47, 48)), (64, (49, 63)), (65, (64, 65)), (130, (129, 7)),
    (48, (200, 0)),                     # a species without sparse rows
])
def test_same_bits_as_the_general_products(atoms, counts, power):
    import torch
    import flare_gb300 as fg
    from flare_gb300 import _lib
    _, gp, calc, _ = weighted(counts, 3, 2, power, seed=atoms)
    # each species' M n_d + M^2 / 2 is below 65,536 (n_d 63)
    assert max(counts) * calc.n_descriptors + max(counts) ** 2 // 2 <= 65536
    st = fg.Structure(*lattice(atoms, atoms), 4.0, [calc])
    var = gp.predict_batch([st], precision="fp64")["local_var"]
    m = gp._device_model([calc])
    mean = torch.empty(1 + 3 * atoms + 6, dtype=torch.float64, device="cuda")
    want = torch.full((atoms,), np.nan, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().fgb_predict_plain(
        m.h, st.nlist().h, _lib.ptr(st._inputs()["species"]), _lib.ptr(mean),
        _lib.ptr(want), _lib.stream_ptr()), "plain")
    assert np.isfinite(var).all()
    assert np.array_equal(var, want.cpu().numpy())
