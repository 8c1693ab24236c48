"""The rounding family of a 16-bit wall's accumulating steps follows its size, not a timing: one cell per thread where those
configurations are the faster ones, two elsewhere and in what walls of several sizes share."""
from types import SimpleNamespace

import numpy as np
import pytest


@pytest.mark.parametrize("shape,alone,one_cell", [((180, 36, 36), True, False), ((198, 31, 38), True, True),
                                                  ((240, 48, 48), True, True), ((266, 53, 56), True, True),
                                                  ((300, 60, 60), True, False), ((240, 48, 48), False, False)])
@pytest.mark.parametrize("fastest", [1, 11])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_family_of_the_accumulating_steps(dtype, fastest, shape, alone, one_cell, monkeypatch):
    import torch
    from stonewall import _native as N
    from stonewall import autotune
    from stonewall.fields import Grid
    L, code = N.lib(), N.dtype_code(dtype)
    old = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)

    def times(solver, cfgs=None, **_):
        return {c: 1.0 + (c != fastest) + 0.01 * c for c in (range(18) if cfgs is None else cfgs)}
    monkeypatch.setattr(autotune, "time_configs", times)
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.setattr("stonewall.fields.Accum", lambda grid, device: None)
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "none")
    try:
        autotune.tune(SimpleNamespace(dtype=code, grid=Grid(*shape), device="cpu"), alone=alone)
        got = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)
    finally:
        L.sw_set_step_config(code, old[0])
        L.sw_set_step_config_accum(code, old[1])
    assert got[0] >= 4
    assert (got[1] < 4) == one_cell


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_every_accumulating_configuration_solves_alike(dtype, cuda):
    """A wall whose accumulating steps run one cell per thread: state, forces and sums after 12 steps, bit for bit."""
    from gpu_helpers import inlet, make_mask
    from stonewall import _native as N
    from stonewall import autotune
    from stonewall.solver import WallSolver
    L, code = N.lib(), N.dtype_code(dtype)
    old = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)
    flag = make_mask(198, 31, 38, 5, density=0.05)
    want = None
    try:
        for plain, accum in [(4, 0), (4, 1), (4, 2), (4, 3), (11, 2), (17, 0)]:
            s = WallSolver(flag, inlet(38, 9), 2e-3, 0.1, 160, 12, n_spin=2, dtype=dtype, acc_every=2, chunk=4)
            assert accum in autotune.candidates(code, s.grid, accumulating=True)
            N.check(L.sw_set_step_config(code, plain), "sw_set_step_config")
            N.check(L.sw_set_step_config_accum(code, accum), "sw_set_step_config_accum")
            s.init(noise=0.03, seed=7, noise_kind="gauss").advance(12)
            got = s.state.numpy(np.float64), s.force.data.cpu().numpy(), s.sums()
            want = want or got
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
    finally:
        L.sw_set_step_config(code, old[0])
        L.sw_set_step_config_accum(code, old[1])
    assert s.n_acc == 5
