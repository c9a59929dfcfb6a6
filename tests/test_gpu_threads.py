"""Stored-gradient calls, kernel matrices and solves from several threads on
streams of their own, which share the scratch pool: the same bits as one after
the other."""
import threading

import numpy as np
import pytest

from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def job(k):
    """The results of thread k's calls, all on the current stream."""
    import torch
    import flare_gb300 as fg
    from flare_gb300 import _lib
    from test_gpu_dense_blocks import spd
    from test_gpu_stored_gradients import cluster
    calc = fg.B2("chebyshev", "quadratic", [0.0, 4.0], [], [2, 3, 2])
    cd = cluster((9 + 20 * k, 17), calc.n_descriptors, seed=k)
    kernel = fg.NormalizedDotProduct(1.5, 2)
    cell, sp, pos = syn.random_alloy(20 + 9 * k, density=0.05, dmin=1.6, seed=k)
    sp[:2] = (0, 1)
    out = [kernel.envs_struc(cd, fg.Structure(cell, sp, pos, 4.0, [calc])),
           kernel.envs_envs(cd, cd)]
    M = 60 + 50 * k
    A = torch.from_numpy(spd(M, k)).cuda()
    X = torch.empty_like(A)
    for call in (lambda: _lib.lib().fgb_cholesky(M, _lib.ptr(A),
                                                 _lib.stream_ptr()),
                 lambda: _lib.lib().fgb_trtri_lower(M, _lib.ptr(A), _lib.ptr(X),
                                                    _lib.stream_ptr())):
        _lib.check(call())
    return out + [A.cpu().numpy(), X.cpu().numpy()]


def test_threads_with_streams():
    import torch
    T, rounds = 4, 6
    alone = [job(k) for k in range(T)]
    errors = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(rounds):
                    for a, b in zip(job(k), alone[k]):
                        assert np.array_equal(a, b)
        except BaseException as e:
            errors.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(T)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
