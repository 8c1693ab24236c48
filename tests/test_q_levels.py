"""q_frame uses the levels of its own limit, also when another thread asks for another limit meanwhile."""
import ctypes
from types import SimpleNamespace

import numpy as np
import torch


def test_levels_are_those_of_the_call(monkeypatch):
    from stonewall import solver as S
    s = S.WallSolver.__new__(S.WallSolver)
    s.device, s.grid, s.flags = torch.device("cpu"), SimpleNamespace(nx=4, ny=4, nz=4), None
    s._u, s._q_levels = object(), (None, None)
    seen = []

    def sw_quantise_levels(q, n, scale, qmax, levels, out, stream):
        seen.append((qmax, np.ctypeslib.as_array((ctypes.c_float * 255).from_address(levels.value)).copy()))
        return 0

    def lib():
        s._q_levels = (9.0, torch.from_numpy(S.quantise_levels(9.0).copy()))      # what the other thread does
        return SimpleNamespace(sw_quantise_levels=sw_quantise_levels)
    monkeypatch.setattr(S.K, "k_qcoarse", lambda *a, **k: None)
    monkeypatch.setattr(S.N, "lib", lib)
    monkeypatch.setattr(S, "_stream", lambda stream=None: None)
    for qmax in (400.0, 17.0, 400.0):
        s.q_frame(1, 1, (2, 2, 2), 1e5, qmax, macro_ready=True)
    assert [v for v, _ in seen] == [400.0, 17.0, 400.0]
    for qmax, levels in seen:
        np.testing.assert_array_equal(levels, S.quantise_levels(qmax))
