"""Calls of the stored-gradient form on a stream that is still busy with
earlier work: the species and pair counts that they read back belong to
their own structure."""
import numpy as np
import pytest

from flare_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def test_envs_struc_behind_queued_work():
    import torch
    import flare_gb300 as fg
    from test_gpu_stored_gradients import cluster
    calc = fg.B2("chebyshev", "quadratic", [0.0, 4.0], [], [2, 3, 2])
    cd = cluster((9, 17), calc.n_descriptors, seed=1)
    kernel = fg.NormalizedDotProduct(1.5, 2)
    strucs = []
    for n in (40, 7, 23):   # other counts of species and pairs each
        cell, sp, pos = syn.random_alloy(n, density=0.05, dmin=1.6, seed=n)
        sp[:2] = (0, 1)
        strucs.append((cell, sp, pos))

    def call(s):
        return kernel.envs_struc(cd, fg.Structure(*s, 4.0, [calc]))

    quiet = [call(s) for s in strucs]
    big = torch.randn(4096, 4096, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for k in (0, 1, 2, 1, 0):
            for _ in range(8):   # some ms in the queue ahead of the call
                big = torch.tanh(big @ big)
            assert np.array_equal(call(strucs[k]), quiet[k])
