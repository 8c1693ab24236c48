"""Snapshot planes of every grid the library takes."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import inlet, make_mask


def test_planes_of_a_long_thin_grid_are_not_refused(native_lib):
    """1.6e9 cells in one plane, three components: 4.8e9 values.  Without a device the call gets as far as
    the launch; with one it is not made (the pointers are the host's)."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("launches on a host pointer")
    from stonewall import _native as N
    buf = np.zeros(64, np.uint8)
    p = ctypes.c_void_p(buf.ctypes.data)
    for extents in ((40000, 1, 40000), (40000, 40000, 1), (64, 8, 9)):
        g = N.geom(*extents)
        assert native_lib.sw_snapshot_planes(ctypes.byref(g), p, 0, 0, p, None) == N.SW_ERR_CUDA
        assert native_lib.sw_snapshot_planes(ctypes.byref(g), p, 0, extents[2], p, None) == N.SW_ERR_BAD_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 2), (65, 1, 14), (31, 17, 2), (256, 3, 5), (129, 9, 14)])
def test_planes_and_their_bits(cuda, shape):
    """Odd extents, a cell that is no number, and values beyond half precision."""
    from stonewall.solver import WallSolver
    nx, ny, nz = shape
    flag = make_mask(nx, ny, nz, 6, density=0.05, extras=False) if nx > 4 and nz > 2 else np.zeros(shape, np.uint8)
    s = WallSolver(flag, inlet(nz, 3), 2e-3, 0.1, nx, 8).init(noise=0.3, seed=2)
    f = s.state.numpy()
    f[:, 0, 0, nz - 1] = np.nan
    f[1, nx - 1, ny - 1, nz - 1] = 1e9
    s.state.assign(f)
    u = s.macro()
    xz, xy = s.snapshot(ny - 1, nz - 1)
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(xz.view(np.uint16), u[1:, :, ny - 1].astype(np.float16).view(np.uint16))
        np.testing.assert_array_equal(xy.view(np.uint16), u[1:, :, :, nz - 1].astype(np.float16).view(np.uint16))
