"""Segment classes (sw_build_tiles) against a per-cell NumPy restatement of the pull sources of
lbm3d.py:77-88, and k_init's two cells per thread at row ends, where a row is no multiple of a segment."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import inlet, make_mask

pytestmark = pytest.mark.gpu

ALL_SOLID, CHECK, FORCE = 1, 2, 4


def classes(flag, pitch):
    from stonewall.lattice import C
    nx, ny, nz = flag.shape
    x, y, z = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
    fluid = flag == 0
    src_solid, src_wall = np.zeros_like(fluid), np.zeros_like(fluid)
    for c in C[1:]:
        xs = np.clip(x - c[0], 0, nx - 1)
        zs = np.minimum(z - c[2], nz - 1)
        f = np.where(zs < 0, 2, flag[xs, (y - c[1]) % ny, np.maximum(zs, 0)])
        src_solid |= f != 0
        src_wall |= f == 1
    pulls = fluid & (x > 0)
    pad = lambda a: np.pad(a, ((0, pitch - nx), (0, 0), (0, 0))).transpose(2, 1, 0).reshape(nz, ny, -1, 32).any(3)  # noqa: E731
    t = np.where(pad(fluid), 0, ALL_SOLID) | np.where(pad(~fluid | (pulls & src_solid)), CHECK, 0)
    return (t | np.where(pad(pulls & src_wall), FORCE, 0)).astype(np.uint8)


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (31, 3, 4), (32, 2, 5), (33, 1, 6), (64, 5, 3), (65, 4, 2),
                                   (97, 7, 9)])
@pytest.mark.parametrize("density,ground", [(0.0, True), (0.02, True), (0.02, False), (0.6, True)])
@pytest.mark.parametrize("shift", [0, 1])
def test_segment_classes(cuda, shape, density, ground, shift):
    """shift 1: a flag array off the 16-byte grid, which the C interface takes."""
    import torch
    from stonewall import _native as N
    from stonewall.fields import Grid
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 10 * ny)
    flag = rng.choice([0, 1, 2], p=[1 - density, 0.8 * density, 0.2 * density], size=shape).astype(np.uint8)
    if ground:
        flag[:, :, 0] = 2
    g = Grid(*shape)
    dev = np.zeros((nz, ny, g.pitch), np.uint8)
    dev[:, :, :nx] = flag.transpose(2, 1, 0)
    buf = torch.zeros(g.cells_padded + 64, dtype=torch.uint8, device="cuda")
    buf[shift:shift + g.cells_padded] = torch.from_numpy(dev.ravel()).cuda()
    tiles = torch.full((g.tiles,), 255, dtype=torch.uint8, device="cuda")
    N.check(N.lib().sw_build_tiles(g.gp, ctypes.c_void_p(buf.data_ptr() + shift), ctypes.c_void_p(tiles.data_ptr()),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "sw_build_tiles")
    np.testing.assert_array_equal(tiles.cpu().numpy().reshape(nz, ny, -1), classes(flag, g.pitch))


@pytest.mark.parametrize("nx", [5, 31, 32, 33, 66])
@pytest.mark.parametrize("dtype", ["f32", "f64", "f16", "bf16"])
@pytest.mark.parametrize("kind", ["uniform", "gauss"])
def test_init_at_row_ends(cuda, oracle_mod, nx, dtype, kind):
    from stonewall.fields import Flags, Grid, Lattice
    from stonewall.kernels import DeviceVector, k_init
    ny, nz = 3, 7
    flag, uin = make_mask(max(nx, 8), ny, nz, 2)[:nx], inlet(nz, 3)
    g = Grid(nx, ny, nz)
    f = Lattice(g, dtype).zero_()
    k_init(f, Flags(g, flag), DeviceVector(uin), 0.02, 9, kind)
    want = oracle_mod.init(flag, uin, noise=np.float32(0.02), seed=9, noise_kind=int(kind == "gauss"))
    same = Lattice(g, dtype).assign(want)            # the oracle's state in the storage type
    tol = {"f32": 1e-6, "f64": 1e-6, "f16": 2e-5, "bf16": 2e-4}[dtype]   # Gaussian noise in float; one storage unit
    np.testing.assert_allclose(f.numpy(np.float64), same.numpy(np.float64), rtol=0, atol=tol)
