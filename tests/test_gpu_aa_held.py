"""In-place steps on both sides of the lattice sizes at which they start or stop holding lines in L2 (16-bit even steps 180 MB,
plain float32 steps 112 MB), against the two-lattice step at the bar of test_gpu_aa.py; rows, span and height fill no
tile."""
import numpy as np
import pytest

from test_gpu_aa import _close, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape,line", [("f16", (449, 99, 99), 180e6), ("f16", (489, 97, 97), 180e6),
                                              ("bf16", (489, 97, 97), 180e6), ("f32", (319, 67, 67), 112e6),
                                              ("f32", (311, 69, 69), 112e6), ("f32", (489, 97, 97), 112e6)])
def test_large_lattices(cuda, dtype, shape, line):
    from gpu_helpers import inlet, make_mask
    nx, ny, nz = shape
    flag = make_mask(nx, ny, nz, 5, density=0.01)
    ab, aa = _pair(flag, inlet(nz, nz // 4), 8, 2, dtype, chunk=4)
    assert (aa.f[0].nbytes > line) == (ny in (97, 69))
    ab.advance(8, use_graphs=False)
    aa.advance(8, use_graphs=False)                    # accumulates in an odd and in an even step (t = 2 and 7)
    assert aa.n_acc == ab.n_acc == 2
    a, b = aa.state_numpy(np.float32), ab.state_numpy(np.float32)
    fluid = np.broadcast_to(flag == 0, a.shape)
    np.testing.assert_array_equal(a[~fluid], b[~fluid])
    _close(a[:, flag == 0], b[:, flag == 0], dtype, "state")
    force_rel, rho_tol, u_tol = {"f32": (1e-5, 1e-5, 1e-6), "f16": (1e-3, 2e-4, 1e-4), "bf16": (8e-3, 1.6e-3, 8e-4)}[dtype]
    sa, sb = aa.sums(), ab.sums()
    np.testing.assert_allclose(sa[0], sb[0], rtol=0, atol=aa.n_acc * rho_tol)
    np.testing.assert_allclose(sa[1:], sb[1:], rtol=0, atol=aa.n_acc * u_tol)
    fa, fb = aa.force_series(), ab.force_series()
    np.testing.assert_allclose(fa, fb, rtol=0, atol=force_rel * np.abs(fb).max())
