"""The TMA-staged step on both sides of the size from which it holds lines in L2 and groups its copies.

A pair of lattices of 118 MB is the line: the smaller grid (109 MB) takes one copy per
population, the larger ones (125 and 124 MB, the last with rows that fill no segment and a
span that fills no row group) the grouped copies.  Same cells and same arithmetic as the
two-cells-per-thread step, so the same bits, plain and accumulating, ring and one-item forms.
"""
import numpy as np
import pytest

from gpu_helpers import inlet, make_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("shape", [(352, 64, 64), (352, 68, 69), (333, 67, 70)])
def test_staged_step_has_the_bits_of_the_two_cell_step(shape, dtype, cuda):
    from stonewall import _native as N
    from stonewall.solver import WallSolver
    nx, ny, nz = shape
    L, code = N.lib(), N.dtype_code(dtype)
    old = L.sw_get_step_config(code), L.sw_get_step_config_accum(code)
    flag = make_mask(nx, ny, nz, 5, density=0.01)
    got = {}
    try:
        for plain, acc in ((4, 4), (10, 15), (8, 9)):
            N.check(L.sw_set_step_config(code, plain), "sw_set_step_config")
            N.check(L.sw_set_step_config_accum(code, acc), "sw_set_step_config_accum")
            s = WallSolver(flag, inlet(nz, nz // 4), 2e-3, 0.1, nx - nx // 5, 7, n_spin=2, dtype=dtype)
            s.init(noise=0.03, seed=7, noise_kind="gauss")
            s.advance(7, use_graphs=False)
            got[plain] = s.state.numpy(np.float64), s.force.data.cpu().numpy().copy(), s.sums()
    finally:
        L.sw_set_step_config(code, old[0])
        L.sw_set_step_config_accum(code, old[1])
    for plain in (10, 8):
        for want, have in zip(got[4], got[plain]):
            np.testing.assert_array_equal(have, want)
