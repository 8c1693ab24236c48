"""A solver reloaded with another mask gives what a new solver of that mask gives."""
import os

import numpy as np
import pytest

from gpu_helpers import inlet, make_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pattern", ["ab", "aa"])
@pytest.mark.parametrize("asked", [False, True])       # whether the first mask was asked for before
def test_reload_with_another_mask(cuda, tmp_path, pattern, asked):
    import torch
    from stonewall.solver import WallSolver
    nx, ny, nz = 70, 9, 11
    first, second = make_mask(nx, ny, nz, 1), make_mask(nx, ny, nz, 2)
    uin = inlet(nz, 3)

    def solver(mask):
        return WallSolver(mask, uin, 2e-3, 0.1, nx - 12, 8, n_spin=0, dtype="f32", acc_every=2, pattern=pattern)

    def solve(s):
        s.init(noise=0.02, seed=3, noise_kind="gauss")
        if pattern == "ab":
            s.f[1].zero_()
        return s.advance(8, use_graphs=False)
    want = solve(solver(second))
    got = solve(solver(first))
    bytes_of_a_new_one = solver(first).memory_bytes()
    if asked:
        np.testing.assert_array_equal(got.flags.host, first)
        got.sums()
    got.reload(torch.from_numpy(second), torch.from_numpy(uin))
    assert got.memory_bytes() - bytes_of_a_new_one == (0 if asked else first.size)
    solve(got)
    np.testing.assert_array_equal(got.flags.solid(), second != 0)
    np.testing.assert_array_equal(got.sums(), want.sums())
    np.testing.assert_array_equal(got.mean_field(), want.mean_field())
    got.save_checkpoint(str(tmp_path / "a"), "s")
    want.save_checkpoint(str(tmp_path / "b"), "s")
    np.testing.assert_array_equal(np.load(os.path.join(tmp_path, "a", "uacc.npy")),
                                  np.load(os.path.join(tmp_path, "b", "uacc.npy")))
    np.testing.assert_array_equal(got.flags.host, first)             # what the construction was given
