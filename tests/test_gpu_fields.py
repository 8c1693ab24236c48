"""Host transfers of the fields: flags from any array, independent of the caller's afterwards, and large downloads."""
import numpy as np
import pytest

from gpu_helpers import make_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["uint8", "read-only", "bool", "int64", "strided"])
def test_flags_keep_what_they_were_given(cuda, form):
    import torch
    from stonewall.fields import Flags, Grid
    nx, ny, nz = 37, 5, 7
    flag = make_mask(nx, ny, nz, 1)
    if form == "bool":
        flag = flag > 0
    elif form == "int64":
        flag = flag.astype(np.int64)
    elif form == "strided":
        flag = np.asfortranarray(flag)
    elif form == "read-only":
        flag.flags.writeable = False
    want = flag.astype(np.uint8)
    f = Flags(Grid(nx, ny, nz), flag)
    if form != "read-only":
        flag[...] = 0                                     # the caller's array is the caller's again
    np.testing.assert_array_equal(f.flag.cpu().numpy().reshape(nz, ny, -1)[:, :, :nx], want.transpose(2, 1, 0))
    f.load(torch.zeros((nx, ny, nz), dtype=torch.uint8))
    assert int(f.flag.sum()) == 0
    np.testing.assert_array_equal(f.host, want)           # the construction's flags, as numpy() gives them
    np.testing.assert_array_equal(f.numpy(), want)
    assert f.numpy() is not f.host


@pytest.mark.parametrize("shape", [(40, 6, 7), (160, 64, 31)])     # below and above the size whose pages are touched
def test_state_round_trip(cuda, shape):
    from stonewall.fields import Grid, Lattice
    rng = np.random.default_rng(0)
    f = rng.uniform(0.01, 0.4, (19,) + shape).astype(np.float32)
    np.testing.assert_array_equal(Lattice(Grid(*shape), "f32").assign(f).numpy(), f)
