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


@pytest.mark.parametrize("shape", [(1, 1, 1), (63, 2, 31), (64, 1, 32), (65, 3, 33), (130, 2, 65)])
@pytest.mark.parametrize("dtype", ["f32", "f64", "f16", "bf16"])
@pytest.mark.parametrize("ref", [np.float32, np.float64])
def test_layout_round_trip_at_tile_edges(cuda, shape, dtype, ref):
    """Pack and unpack against the storage type's own rounding (torch on the host), padding included."""
    import torch
    from stonewall.fields import Grid, Lattice
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12).astype(np.float32).reshape(19, 1, 1, 1)
    f = (w * np.random.default_rng(1).uniform(0.8, 1.2, (19,) + shape)).astype(ref)
    g = Grid(*shape)
    lat = Lattice(g, dtype).assign(f)
    if dtype in ("f16", "bf16"):
        t = {"f16": torch.float16, "bf16": torch.bfloat16}[dtype]
        stored = torch.from_numpy(f.astype(np.float32) - w).to(t)
        want, pad = (w + stored.float().numpy()).astype(ref), np.zeros_like(w)
    else:
        t = {"f32": torch.float32, "f64": torch.float64}[dtype]
        stored = torch.from_numpy(f.astype({"f32": np.float32, "f64": np.float64}[dtype]))
        want, pad = stored.numpy().astype(ref), w if dtype == "f32" else np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    dev = lat.data.view(t).view(19, g.nz, g.ny, g.pitch).cpu()
    assert torch.equal(dev[..., :g.nx], stored.permute(0, 3, 2, 1))
    if g.pitch > g.nx:
        np.testing.assert_array_equal(dev[..., g.nx:].double().numpy(),
                                      np.broadcast_to(np.asarray(pad, np.float64).reshape(19, 1, 1, 1),
                                                      (19, g.nz, g.ny, g.pitch - g.nx)))
    np.testing.assert_array_equal(lat.numpy(ref), want)
