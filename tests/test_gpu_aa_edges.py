"""The 16-bit in-place odd step at the ends of rows, at the top and next to stones there: its edge and checked
two-cell paths against the two-lattice step (the bar of test_gpu_aa.py), on grids of one or a few segment pairs."""
import numpy as np
import pytest

from test_gpu_aa import _close, _pair

pytestmark = pytest.mark.gpu


def _mask(nx, ny, nz, kind):
    flag = np.zeros((nx, ny, nz), np.uint8)
    if kind != "open":
        flag[:, :, 0] = 2
    if kind == "stones":
        flag[nx // 2, 0, 1] = flag[nx - 1, ny - 1, nz - 1] = flag[0, 0, 2] = flag[nx - 1, 0, 1] = 1
        flag[min(1, nx - 1), ny // 2, nz - 1] = 1
    return flag


@pytest.mark.parametrize("nx", [2, 3, 33, 63, 64, 65, 66, 128, 129, 191])
@pytest.mark.parametrize("ny,nz", [(1, 4), (5, 6)])
@pytest.mark.parametrize("kind", ["open", "ground", "stones"])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_odd_step_edges(cuda, nx, ny, nz, kind, dtype):
    from gpu_helpers import inlet
    flag, uin = _mask(nx, ny, nz, kind), inlet(nz, 2)
    ab, aa = _pair(flag, uin, 8, 2, dtype, chunk=4)
    ab.advance(8)
    aa.advance(8)
    a, b = aa.state_numpy(np.float32), ab.state_numpy(np.float32)
    fluid = np.broadcast_to(flag == 0, a.shape)
    np.testing.assert_array_equal(a[~fluid], b[~fluid])
    _close(a[:, flag == 0], b[:, flag == 0], dtype, "state")
    tol = {"f16": 2e-4, "bf16": 1.6e-3}[dtype]
    sa, sb = aa.sums(), ab.sums()
    np.testing.assert_allclose(sa, sb, rtol=0, atol=aa.n_acc * tol)
    fa, fb = aa.force_series(), ab.force_series()
    np.testing.assert_allclose(fa, fb, rtol=0, atol={"f16": 1e-3, "bf16": 8e-3}[dtype] * max(np.abs(fb).max(), 1e-30))
