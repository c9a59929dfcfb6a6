"""CPU: packing of structures, whatever their species lists hold."""
import types

import numpy as np
import pytest

from flare_gb300.core import pack_structures


@pytest.mark.parametrize("species", [
    [[0, 1, 0], [1]], [[], [2, 0]], [[], []], [[]],
    [(0, 1), [255, 0]], [[256, 0], [1]], [[-1, 0], [1]],
    [np.array([0, 3]), [1, 2]], [np.array([1, 0, 2])[::-1], [7]],
    [np.array([0, 1], np.int64), np.array([300, 2], np.int16)],
    [[np.int64(4), np.int32(5)], [True, False]], [[1.0, 2.0], [0]],
])
def test_species(species):
    s = [types.SimpleNamespace(noa=len(x), cell=np.eye(3), species=x,
                               positions=np.ones((len(x), 3)))
         for x in species]
    offsets, cells, pos, sp = pack_structures(s)
    want = np.concatenate([np.asarray(x, np.int32) for x in species])
    assert sp.dtype == np.int32 and sp.flags.c_contiguous
    assert np.array_equal(sp, want)
    assert offsets.tolist() == np.cumsum([0] + [len(x) for x in species]).tolist()
    assert cells.shape == (len(s), 9) and pos.shape == (len(want), 3)


def test_many_lists_are_joined_once(monkeypatch):
    """One conversion of all lists, not one array for each: a batch of 3,000
    structures of 4 atoms had come to spend 6 ms here instead of 2."""
    from flare_gb300 import core
    calls = []
    asarray = np.asarray
    monkeypatch.setattr(core.np, "asarray",
                        lambda *a, **k: calls.append(a) or asarray(*a, **k))
    frombuffer = np.frombuffer
    monkeypatch.setattr(core.np, "frombuffer",
                        lambda *a, **k: calls.append(a) or frombuffer(*a, **k))
    s = [types.SimpleNamespace(noa=4, cell=np.eye(3), species=[0, 1, 0, 1],
                               positions=np.ones((4, 3))) for _ in range(50)]
    assert np.array_equal(pack_structures(s)[3], [0, 1] * 100)
    assert len(calls) == 1
