"""What a solve computes does not depend on which configuration a timing came out fastest for."""
from types import SimpleNamespace

import numpy as np
import pytest


@pytest.mark.parametrize("dtype", ["f32", "f64", "f16", "bf16"])
def test_tuning_installs_one_rounding_family(dtype, monkeypatch):
    """With the one-cell configurations timed fastest, 16 bits still get one of the two-cell ones."""
    import torch
    from stonewall import _native as N
    from stonewall import autotune
    from stonewall.fields import Grid
    L, code = N.lib(), N.dtype_code(dtype)
    old = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)
    supported = range(18 if dtype in ("f16", "bf16") else 4)

    def times(solver, acc=None, cfgs=None, **_):
        fastest = 3 if acc is None else 2
        return {c: 1.0 + (c != fastest) + 0.01 * c for c in (supported if cfgs is None else cfgs) if c in supported}
    monkeypatch.setattr(autotune, "time_configs", times)
    monkeypatch.setattr(autotune, "_CACHE", {})
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "none")
    try:
        autotune.tune(SimpleNamespace(dtype=code, grid=Grid(8, 4, 4), device="cpu"))
        got = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)
    finally:
        L.sw_set_step_config(code, old[0])
        L.sw_set_step_config_accum(code, old[1])
    assert got == ((4, 4) if dtype in ("f16", "bf16") else (3, 2))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["f32", "f64", "f16", "bf16"])
def test_every_installable_configuration_solves_alike(dtype, cuda):
    """State, forces and sums after 50 steps of a small wall, bit for bit."""
    from gpu_helpers import inlet, make_mask
    from stonewall import _native as N
    from stonewall import autotune
    from stonewall.solver import WallSolver
    L, code = N.lib(), N.dtype_code(dtype)
    old = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)
    flag = make_mask(90, 21, 22, 5, density=0.05)
    want = None
    try:
        for cfg in autotune.candidates(code):
            if L.sw_set_step_config(code, cfg) == N.SW_ERR_UNSUPPORTED:
                continue
            N.check(L.sw_set_step_config_accum(code, cfg), "sw_set_step_config_accum")
            s = WallSolver(flag, inlet(22, 6), 2e-3, 0.1, 72, 50, n_spin=10, dtype=dtype, chunk=10)
            s.init(noise=0.03, seed=7, noise_kind="gauss").advance(50)
            got = s.state.numpy(np.float64), s.force.data.cpu().numpy(), s.sums()
            want = want or got
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
    finally:
        L.sw_set_step_config(code, old[0])
        L.sw_set_step_config_accum(code, old[1])
    assert want is not None
