"""fgb_envs_envs as a queued call: it returns while earlier work of its stream
still runs, and can be captured into a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N1, N2, ND = 150, 130, 144


@pytest.fixture(scope="module")
def inputs():
    import torch
    r = np.random.Generator(np.random.PCG64(1))
    d = [r.normal(size=(n, ND)) + 0.5 for n in (N1, N2)]
    n = [np.linalg.norm(x, axis=1) for x in d]
    want = 2.25 * ((d[0] / n[0][:, None]) @ (d[1] / n[1][:, None]).T) ** 2
    return [torch.from_numpy(x).cuda() for x in (d[0], n[0], d[1], n[1])], want


def queue(t, out):
    from flare_gb300 import _lib
    p = _lib.ptr
    _lib.check(_lib.lib().fgb_envs_envs(p(t[0]), p(t[1]), N1, p(t[2]), p(t[3]),
                                        N2, ND, 2.25, 2.0, p(out),
                                        _lib.stream_ptr()), "envs_envs")


def error(out, want):
    # |k| <= sigma^2, each dot product rounds by at most ND ulp
    return np.abs(out.cpu().numpy() - want).max() / (4 * 2 * ND * 2.25 * 2.3e-16)


def test_returns_before_earlier_work(inputs):
    import torch
    t, want = inputs
    out = torch.empty((N1, N2), dtype=torch.float64, device="cuda")
    queue(t, out)   # kernels loaded, scratch made
    torch.cuda.synchronize()
    out.fill_(np.nan)
    x = torch.randn(8192, 8192, device="cuda")
    for _ in range(40):   # some 100 ms of work ahead of the call
        x = torch.tanh(x @ x)
    ahead = torch.cuda.Event()
    ahead.record()
    queue(t, out)
    assert not ahead.query()
    assert error(out, want) <= 1.0


def test_captured(inputs):
    import torch
    t, want = inputs
    out = torch.empty((N1, N2), dtype=torch.float64, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        queue(t, out)
    for _ in range(2):
        out.fill_(np.nan)
        g.replay()
        assert error(out, want) <= 1.0
