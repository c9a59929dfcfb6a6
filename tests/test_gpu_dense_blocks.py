"""The cluster-wide diagonal-block Cholesky and its inverse at the edges of
their 32- and 128-column blocks, against LAPACK in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 96, 97, 127, 128, 129, 160, 255, 289]


def spd(M, seed, scale=1.0):
    r = np.random.Generator(np.random.PCG64(seed))
    Q, _ = np.linalg.qr(r.normal(size=(M, M)))
    return (Q * np.geomspace(1.0, 1e-4, M)) @ Q.T * scale


def solve(K, jitter=0.0):
    """(L_inv, R_inv, alpha) of fgb_solve_qr without labels."""
    import torch
    from flare_gb300 import _lib
    M = K.shape[0]
    d = torch.from_numpy(np.ascontiguousarray(K)).cuda()
    out = [torch.full((M, M), np.nan, dtype=torch.float64, device="cuda")
           for _ in range(2)]
    a = torch.zeros(M, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().fgb_solve_qr(
        M, 0, _lib.ptr(d), None, None, None, jitter, _lib.ptr(a),
        _lib.ptr(out[0]), _lib.ptr(out[1]), _lib.stream_ptr()), "solve")
    return out[0].cpu().numpy(), out[1].cpu().numpy()


@pytest.mark.parametrize("M", SIZES)
@pytest.mark.parametrize("scale", [1.0, 1e40])
def test_block_cholesky_and_inverse(M, scale):
    import torch
    from flare_gb300 import _lib
    A = spd(M, M, scale)
    d = torch.from_numpy(A.copy()).cuda()
    _lib.check(_lib.lib().fgb_cholesky(M, _lib.ptr(d), _lib.stream_ptr()),
               "cholesky")
    L = d.cpu().numpy()
    assert np.all(np.triu(L, 1) == 0.0)
    # backward error of a blocked FP64 Cholesky: a few M ulp of the largest
    # entry
    assert np.abs(L @ L.T - A).max() <= 16 * M * 2.3e-16 * np.abs(A).max()
    X, R = solve(A)
    assert np.all(np.triu(X, 1) == 0.0)
    # |X| <= 1e2 / sqrt(scale), |L| <= sqrt(scale): residual of a blocked
    # inverse, a few M ulp of |X||L|
    assert np.abs(X @ L - np.eye(M)).max() <= 64 * M * 2.3e-16 * 1e2
    # no labels: R^T R = L L^T
    assert np.abs(R.T @ A @ R - np.eye(M)).max() <= 64 * M * 2.3e-16 * 1e4


@pytest.mark.parametrize("bad", [0, 31, 32, 100, 127, 128, 200])
def test_block_cholesky_names_the_first_bad_pivot(bad):
    import torch
    from flare_gb300 import _lib
    A = spd(210, 3)
    A[bad, bad] = -1.0
    d = torch.from_numpy(A).cuda()
    with pytest.raises(ValueError, match=f"leading minor {bad + 1} not"):
        _lib.check(_lib.lib().fgb_cholesky(210, _lib.ptr(d),
                                           _lib.stream_ptr()), "cholesky")
