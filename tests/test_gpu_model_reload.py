"""New weights on a model handle that has predicted before: nothing of the
earlier weights is used, R_inv included."""
import ctypes

import numpy as np
import pytest

from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def weights(M, n_d, seed):
    r = np.random.Generator(np.random.PCG64(seed))
    tri = [np.tril(r.normal(size=(M, M))) * 0.1 + np.eye(M) for _ in range(2)]
    return (np.array([M - M // 3, M // 3], np.int32),
            r.normal(size=(M, n_d)) + 0.5, r.normal(size=M), tri[0],
            np.ascontiguousarray(tri[1].T))


@pytest.mark.parametrize("dtc", [False, True])
def test_solved_variances_need_the_new_R_inv(dtc):
    import torch
    import flare_gb300 as fg
    from flare_gb300 import _lib
    from flare_gb300.core import _Model
    lib, ptr = _lib.lib(), _lib.ptr
    calc = fg.B2("chebyshev", "quadratic", [0.0, 4.0], [], [2, 3, 2])
    cell, sp, pos = syn.random_alloy(24, density=0.05, dmin=1.6, seed=3)
    st = fg.Structure(cell, sp, pos, 4.0, [calc])
    call = lib.fgb_predict_dtc if dtc else lib.fgb_predict_sor

    def predict(m):
        out = torch.full((2, 1 + 3 * 24 + 6), np.nan, dtype=torch.float64,
                         device="cuda")
        _lib.check(call(m.h, st.nlist().h, ptr(st._inputs()["species"]),
                        ptr(out[0]), ptr(out[1]), _lib.stream_ptr()), "predict")
        return out.cpu().numpy()

    def load(m, w):
        m.set(*w[:4])
        _lib.check(lib.fgb_model_set_R_inv(m.h, ptr(w[4])), "R_inv")

    first, same, more = (weights(M, calc.n_descriptors, s)
                         for M, s in ((20, 1), (20, 2), (75, 3)))
    m = _Model(calc, 1.5, 2)
    load(m, first)
    assert np.isfinite(predict(m)).all()
    # the same number of rows, then more than R_inv has: refused
    for w in (same, more):
        m.set(*w[:4])
        with pytest.raises(RuntimeError, match="up to date"):
            predict(m)
        load(m, w)
        fresh = _Model(calc, 1.5, 2)
        load(fresh, w)
        assert np.array_equal(predict(m), predict(fresh))


def test_refused_weights_leave_the_model_as_it_was():
    import flare_gb300 as fg
    from flare_gb300 import _lib
    from flare_gb300.core import _Model
    calc = fg.B2("chebyshev", "quadratic", [0.0, 4.0], [], [2, 3, 2])
    w = weights(20, calc.n_descriptors, 1)
    m = _Model(calc, 1.5, 2)
    m.set(*w[:4])
    fold = [ctypes.c_double(-1.0) for _ in range(2)]
    for f, counts in zip(fold, (None, [4, -1])):
        if counts:
            with pytest.raises(ValueError, match="negative count"):
                m.set(np.array(counts, np.int32), *w[1:4])
        _lib.check(_lib.lib().fgb_model_fold_guard(
            m.h, ctypes.byref(f), None, _lib.stream_ptr()), "fold")
    assert fold[0].value == fold[1].value > 0.0
