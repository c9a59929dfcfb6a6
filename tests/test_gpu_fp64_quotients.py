"""The FP64 quotients that the kernels form themselves against IEEE division:
the reciprocal of a Cholesky pivot and the division by a small integer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 20
EDGES = [0, 1, 2, (1 << 51) - 1, 1 << 51, (1 << 51) + 1, (1 << 52) - 2,
         (1 << 52) - 1]


def doubles(lo, hi, seed):
    """Random mantissas over the biased exponents [lo, hi], and EDGES'
    mantissas at all of them."""
    r = np.random.Generator(np.random.PCG64(seed))
    e = r.integers(lo, hi + 1, size=N).astype(np.uint64)
    m = r.integers(0, 1 << 52, size=N).astype(np.uint64)
    ee, em = np.meshgrid(np.arange(lo, hi + 1, dtype=np.uint64),
                         np.array(EDGES, np.uint64))
    bits = np.concatenate([(e << np.uint64(52)) | m,
                           ((ee << np.uint64(52)) | em).reshape(-1)])
    return bits.view(np.float64)


def quotients(k, x):
    import torch
    from flare_gb300 import _lib
    d = torch.from_numpy(x).cuda()
    y = torch.full_like(d, np.nan)
    _lib.check(_lib.lib().fgb_fp64_check(k, len(x), _lib.ptr(d), _lib.ptr(y),
                                         _lib.stream_ptr()))
    return y.cpu().numpy()


def test_pivot_reciprocal():
    """Within one ulp (the step leaves 2^-60 and one rounding) over all
    exponents; outside [60, 1979], where the estimate does not serve, the
    rounded quotient.  1/x below the normal range is left out: ulps there
    are absolute."""
    x = doubles(1, 2044, 1)
    y, want = quotients(0, x), 1.0 / x
    ulps = np.abs(y.view(np.int64) - want.view(np.int64))
    assert ulps.max() <= 1
    e = x.view(np.int64) >> 52
    assert (ulps[(e < 60) | (e > 1979)] == 0).all()
    # nearly all are the rounded quotient: the tail beyond half an ulp is
    # 2^-7 of an ulp wide on either side
    assert (ulps > 0).mean() < 0.05


@pytest.mark.parametrize("k", range(1, 22))
def test_division_by_a_small_integer(k):
    x = doubles(1023 - 900, 1023 + 999, k)
    x[::2] *= -1.0
    assert np.array_equal(quotients(k, x), x / k)
    assert np.array_equal(quotients(k, np.zeros(3)), np.zeros(3))
