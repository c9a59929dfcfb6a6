"""Slicing at the edges of its launch forms: rows read whole for their scale
(one part, or few rows of up to 2,048 columns) or scaled by a pass of their
own, as the operands of products against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (2432, 40, 512), (2432, 40, 513),      # many rows: one part, two parts
    (2424, 40, 17), (40, 33, 127), (40, 33, 129), (9, 33, 2048),
    (9, 33, 2049),                         # few rows: scales in the block, or not
])
def test_launch_forms(M, N, K):
    import torch
    from flare_gb300 import _lib
    r = np.random.Generator(np.random.PCG64(M + N + K))
    A = r.normal(size=(M, K)) * np.exp(r.uniform(-6, 2, size=(M, K)))
    B = r.normal(size=(N, K)) * np.exp(r.uniform(-6, 2, size=(N, K)))
    A[M // 2] = 0.0
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    dC = torch.full((M, N), np.nan, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().fgb_oz_dgemm_nt(M, N, K, _lib.ptr(dA), K,
                                          _lib.ptr(dB), K, _lib.ptr(dC), N,
                                          _lib.stream_ptr()))
    C = dC.cpu().numpy()
    # nine slices: 2^-54 of each row's largest entry, and one rounding
    bound = np.abs(A).max(1)[:, None] * np.abs(B).sum(1)[None, :] + \
        np.abs(A).sum(1)[:, None] * np.abs(B).max(1)[None, :]
    assert np.all(np.abs(C - A @ B.T) <= 2e-15 * bound + 1e-300)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 300, 513])
def test_same_rows_in_both_layouts(n):
    """The factor of a matrix whose trailing products L21 L21^T take one row
    set in two tile heights, and its inverse."""
    import torch
    from flare_gb300 import _lib
    r = np.random.Generator(np.random.PCG64(n))
    G = r.normal(size=(n, n))
    S = G @ G.T + n * np.eye(n)
    A = torch.from_numpy(S).cuda()
    _lib.check(_lib.lib().fgb_cholesky(n, _lib.ptr(A), _lib.stream_ptr()))
    L = np.tril(A.cpu().numpy())
    # backward error of a Cholesky factor: (n + 1) u |L| |L|^T
    u = 2.0 ** -53
    assert np.all(np.abs(L @ L.T - S) <=
                  4 * (n + 1) * u * (np.abs(L) @ np.abs(L).T))


@pytest.mark.parametrize("scale", [2.0 ** -990, 2.0 ** 970])
@pytest.mark.parametrize("n", [5, 33, 128])
def test_factor_of_extreme_scales(n, scale):
    """Pivots outside the range of the reciprocal's estimate, in a single
    diagonal block: the factor of the scaled matrix is the scaled factor."""
    import torch
    from flare_gb300 import _lib
    r = np.random.Generator(np.random.PCG64(n))
    G = r.normal(size=(n, n))
    S = G @ G.T + n * np.eye(n)
    out = []
    for f in (1.0, scale):
        A = torch.from_numpy(S * f).cuda()
        _lib.check(_lib.lib().fgb_cholesky(n, _lib.ptr(A), _lib.stream_ptr()))
        out.append(A.cpu().numpy() / np.sqrt(f))
    # each within the backward error of the exact factor, whose condition
    # here is below 10
    np.testing.assert_allclose(out[1], out[0], rtol=0,
                               atol=100 * n * 2.0 ** -53 * np.abs(out[0]).max())
