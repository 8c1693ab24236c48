"""Viewer payload kernels at block edges: Q frames whose voxels do not fill a block (or exceed one), the planes
of a snapshot, and the quantisation of a frame against the host expression of lbm3d.py:317-318."""
import numpy as np
import pytest

from gpu_helpers import inlet, make_mask

pytestmark = pytest.mark.gpu


def _macro(grid, seed):
    from stonewall.fields import Macro
    import torch
    u = Macro(grid)
    rng = np.random.default_rng(seed)
    a = rng.normal(0, 0.05, (4, grid.nx, grid.ny, grid.nz)).astype(np.float32)
    v = u.data.view(4, grid.nz, grid.ny, grid.pitch)
    v[..., :grid.nx] = torch.from_numpy(a).permute(0, 3, 2, 1).cuda()
    return u, a


@pytest.mark.parametrize("shape,x0,ds,dims", [
    ((260, 4, 5), 0, 1, (260, 4, 5)), ((259, 6, 7), 3, 2, (128, 3, 3)), ((200, 9, 10), 1, 3, (66, 3, 3)),
    ((70, 70, 66), 2, 65, (1, 1, 1)), ((134, 130, 131), 3, 129, (1, 1, 1)), ((40, 8, 9), 5, 7, (5, 1, 1))])
def test_q_frame_blocks(cuda, oracle_mod, shape, x0, ds, dims):
    import torch
    from stonewall.fields import Flags, Grid
    from stonewall.kernels import k_qcoarse
    g = Grid(*shape)
    flag = make_mask(*shape, 4, density=0.002)
    u, a = _macro(g, 1)
    q = torch.full(dims, -1.0, dtype=torch.float32, device="cuda")
    k_qcoarse(u, Flags(g, flag), x0, ds, *shape, q)
    np.testing.assert_array_equal(q.cpu().numpy(), oracle_mod.qcoarse(a, flag, x0, ds, dims))


@pytest.mark.parametrize("scale,qmax", [(1e5, 400.0), (3, 400), (2.5e4, 17.3), (np.float64(1e5), 400.0), (1e9, 0.02)])
def test_snapshot_and_q_bytes(cuda, scale, qmax):
    from stonewall.solver import WallSolver
    nx, ny, nz = 65, 9, 14
    flag, uin = make_mask(nx, ny, nz, 6, density=0.05), inlet(nz, 3)
    s = WallSolver(flag, uin, 2e-3, 0.1, nx - 8, 8).init(noise=0.3, seed=2)
    s.advance(3)
    u = s.macro()
    xz, xy = s.snapshot(ny // 2, 5)
    np.testing.assert_array_equal(xz, u[1:, :, ny // 2].astype(np.float16))
    np.testing.assert_array_equal(xy, u[1:, :, :, 5].astype(np.float16))
    dims = ((nx - 3) // 2, ny // 2, nz // 2)
    got = s.q_frame(2, 2, dims, scale, qmax, macro_ready=True)
    import torch
    from stonewall.kernels import k_qcoarse
    q = torch.empty(dims, dtype=torch.float32, device="cuda")
    k_qcoarse(s._u, s.flags, 2, 2, nx, ny, nz, q)
    v = np.clip(q.cpu().numpy() * scale, 0, qmax)
    want = np.round(255 * np.log1p(v) / np.log1p(qmax)).astype(np.uint8)
    assert got.dtype == np.uint8
    np.testing.assert_array_equal(got, want)
