"""Flags made and loaded on a stream of their own, with the current stream busy."""
import numpy as np
import pytest

from gpu_helpers import make_mask

pytestmark = pytest.mark.gpu
SHAPE = (37, 5, 7)


def on_device(f):
    g = f.grid
    return f.flag.cpu().numpy().reshape(g.nz, g.ny, -1)[:, :, :g.nx].transpose(2, 1, 0)


@pytest.mark.parametrize("pinned", [False, True])
def test_construction_on_another_stream(cuda, pinned):
    """The caller's array is the caller's again when the constructor returns, pinned memory as well."""
    import torch
    from stonewall.fields import Flags, Grid
    want = make_mask(*SHAPE, 1)
    given = torch.from_numpy(want.copy())
    given = (given.pin_memory() if pinned else given).numpy()
    torch.cuda._sleep(400_000_000)
    f = Flags(Grid(*SHAPE), given, stream=torch.cuda.Stream())
    given[...] = 0
    np.testing.assert_array_equal(on_device(f), want)
    np.testing.assert_array_equal(f.host, want)


def test_load_on_another_stream(cuda):
    """A mask that the current stream is still making, dropped by the caller right after load()."""
    import torch
    from stonewall.fields import Flags, Grid
    want = make_mask(*SHAPE, 2)
    f, ready, s = Flags(Grid(*SHAPE), make_mask(*SHAPE, 1)), torch.from_numpy(want).cuda(), torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)
    made = torch.zeros_like(ready)
    made.copy_(ready)
    f.load(made, stream=s)
    del made
    torch.full(SHAPE, 7, dtype=torch.uint8, device="cuda")
    s.synchronize()
    np.testing.assert_array_equal(on_device(f), want)
    np.testing.assert_array_equal(f.solid(), want != 0)
