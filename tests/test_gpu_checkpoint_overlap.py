"""A background checkpoint returns while the steps queued before it still run, the first one of a solver too."""
import os

import numpy as np
import pytest

from gpu_helpers import inlet, make_mask

pytestmark = pytest.mark.gpu


def test_first_background_checkpoint_waits_for_no_step(cuda, tmp_path):
    import torch
    from stonewall.solver import WallSolver
    nx, ny, nz = 70, 9, 11
    masks = [make_mask(nx, ny, nz, k) for k in (1, 2)]

    def solver():
        s = WallSolver(masks[0], inlet(nz, 3), 2e-3, 0.1, nx - 12, 8, dtype="f32")
        return s.init(noise=0.02, seed=3, noise_kind="gauss").advance(6, use_graphs=False)

    def checkpoint(s, name):
        torch.cuda._sleep(1_000_000_000)                # about half a second on the stream, before what is taken
        queued = torch.cuda.Event()
        queued.record()
        s.save_checkpoint(str(tmp_path / name), "s", background=True)
        waited = queued.query()
        s.wait_checkpoint()
        return waited, np.load(os.path.join(tmp_path, name, "uacc.npy"))
    checkpoint(solver(), "warm")                        # modules loaded, pinned blocks kept by the allocator
    s = solver()
    for name, mask in (("a", masks[0]), ("b", masks[0]), ("c", masks[1])):
        if name == "c":
            s.reload(torch.from_numpy(mask), torch.from_numpy(inlet(nz, 3)))
            s.init(noise=0.02, seed=3, noise_kind="gauss").advance(6, use_graphs=False)
        waited, uacc = checkpoint(s, name)
        assert not waited
        if name != "a":                                 # ("b" takes the mask that "a" downloaded)
            np.testing.assert_array_equal(uacc, s.sums())
        solid = mask != 0
        assert (uacc[0][solid] == s.n_acc).all() and (uacc[1:, solid] == 0).all() and (uacc[1, ~solid] != 0).any()
