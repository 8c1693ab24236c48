"""In-place steps on a grid one cell long, whose inlet cells are its outlet cells: stones keep their bits."""
import numpy as np
import pytest

from test_gpu_aa import _close, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f64", "f16", "bf16"])
@pytest.mark.parametrize("nx", [1, 2])
def test_stones_in_a_column(cuda, dtype, nx):
    from gpu_helpers import inlet
    flag = np.zeros((nx, 6, 9), np.uint8)
    flag[:, :, 0] = 2
    flag[0, 2, 4] = flag[0, 0, 8] = flag[nx - 1, 5, 6] = 1
    ab, aa = _pair(flag, inlet(9, 3), 8, 2, dtype, chunk=4)
    ab.advance(8)
    aa.advance(8)
    rd = np.float64 if dtype == "f64" else np.float32
    a, b = aa.state_numpy(rd), ab.state_numpy(rd)
    fluid = np.broadcast_to(flag == 0, a.shape)
    np.testing.assert_array_equal(a[~fluid], b[~fluid])
    _close(a[:, flag == 0], b[:, flag == 0], dtype, "state")
    tol = {"f64": 1e-12, "f32": 1e-5, "f16": 2e-4, "bf16": 1.6e-3}[dtype]
    np.testing.assert_allclose(aa.sums(), ab.sums(), rtol=0, atol=aa.n_acc * tol)
