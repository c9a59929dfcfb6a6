"""Ten-slice products where a result is made of its rows' small entries alone
(near-orthogonal environments): their error is bounded by the rows' largest
entries, an absolute bound, not by the result."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def product(A, B):
    """A B^T by fgb_envs_envs: power 1, sigma 1, norms 1."""
    import torch
    from flare_gb300 import _lib
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
         for x in (A, np.ones(len(A)), B, np.ones(len(B)))]
    out = torch.full((len(A), len(B)), np.nan, dtype=torch.float64,
                     device="cuda")
    p = _lib.ptr
    _lib.check(_lib.lib().fgb_envs_envs(
        p(t[0]), p(t[1]), len(A), p(t[2]), p(t[3]), len(B), A.shape[1], 1.0,
        1.0, p(out), _lib.stream_ptr()))
    return out.cpu().numpy()


@pytest.mark.parametrize("small", [-8, -20, -40, -58])
@pytest.mark.parametrize("K", [17, 144, 1500])
def test_small_entries_beside_large_ones(K, small):
    r = np.random.Generator(np.random.PCG64(K - small))
    n = 6
    A, B = (r.normal(size=(n, K)) * 2.0 ** small for _ in range(2))
    A[:, 0] = r.normal(size=n) + 3.0     # meets zeros of B, and the other
    B[:, 0] = 0.0                        # way round
    B[:, 1] = r.normal(size=n) + 3.0
    A[:, 1] = 0.0
    C = product(A, B)
    exact = np.array([[float(sum(Fraction(a) * Fraction(b)
                                 for a, b in zip(x, y))) for y in B]
                      for x in A])
    # for each of the K entry pairs, with row scales of at most twice the
    # largest entries: 9 (then 8, 7, ...) dropped digit products of at most
    # 32 x 32 at 2^-72 (2^-78, ...), together 9.2 2^-60 of the product of the
    # largest entries, and 2^-60 of each row's for what is below its digits;
    # then one rounding
    top = np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    assert np.all(np.abs(C - exact) <= 2.0 ** -56 * K * top +
                  2.0 ** -52 * np.abs(exact))


def test_entries_with_all_their_bits():
    """Entries of four digits in which all but two are zero, 2^-24 of the
    row's largest: their products are among those kept, so the result is exact."""
    r = np.random.Generator(np.random.PCG64(3))
    A = r.integers(-15, 16, size=(5, 40)) * 2.0 ** -24
    B = r.integers(-15, 16, size=(7, 40)) * 2.0 ** -24
    A[:, 0], B[:, 0], B[:, 1], A[:, 1] = 1.0, 0.0, 1.0, 0.0
    assert np.array_equal(product(A, B), A @ B.T)


@pytest.mark.parametrize("up,down", [(1023, -1018), (1022, -1040), (-1040, 1000)])
def test_rows_at_the_ends_of_the_range(up, down):
    """Finite rows up to the largest double, and subnormal ones."""
    K = 40
    r = np.random.Generator(np.random.PCG64(up + 2000))
    A = np.ldexp(r.uniform(-2.0, 2.0, size=(5, K)), up)
    A[:, 3] = np.ldexp(1.875, up)
    B = np.ldexp(r.uniform(-2.0, 2.0, size=(7, K)), down)
    assert np.isfinite(A).all()
    # scaled exactly to where the sums can neither overflow nor underflow
    exact = np.array([[float(sum(Fraction(a) * Fraction(b)
                                 for a, b in zip(x, y))) for y in B]
                      for x in A])
    top = np.ldexp(np.abs(np.ldexp(A, -up)).max(1)[:, None] *
                   np.abs(np.ldexp(B, -down)).max(1)[None, :], up + down)
    assert np.all(np.abs(product(A, B) - exact) <= 2.0 ** -56 * K * top +
                  2.0 ** -52 * np.abs(exact))
