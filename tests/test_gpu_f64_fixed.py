"""Float64 storage collides in fixed point where a cell is in range and in double elsewhere: both, mixed within a
warp, against the float64 oracle (two-lattice step in each configuration, accumulating step, in-place steps)."""
import numpy as np
import pytest

from gpu_helpers import assert_force_close, inlet, make_mask

pytestmark = pytest.mark.gpu

TOL = 1e-12                       # the float64 bar of the step tests
NU, CS, NUS = 2e-3, 0.1, 0.05


def _state(oracle, flag, uin, kind, seed):
    """k_init's state; "edge": some cells have one population outside the fixed-point range."""
    f = oracle.init(flag, uin, noise=0.02, seed=seed).astype(np.float64)
    if kind == "edge":
        rng = np.random.default_rng(seed)
        x, y, z = np.nonzero(flag == 0)
        pick = rng.choice(len(x), len(x) // 5, replace=False)
        pops = rng.integers(0, 19, len(pick))
        vals = rng.choice([0.6, 1e-5, -1e-3, 0.26, 0.13], len(pick))
        f[pops, x[pick], y[pick], z[pick]] = vals
    return f


@pytest.mark.parametrize("shape", [(33, 7, 9), (64, 5, 6), (31, 4, 5)])
@pytest.mark.parametrize("kind", ["flow", "edge"])
def test_step_against_oracle(cuda, oracle_mod, shape, kind):
    import torch
    from stonewall.fields import Accum, Flags, ForceSeries, Grid, Lattice
    from stonewall.kernels import DeviceVector, k_step
    nx, ny, nz = shape
    flag, uin = make_mask(nx, ny, nz, 3), inlet(nz, 3)
    f0 = _state(oracle_mod, flag, uin, kind, 11)
    want, want_force = oracle_mod.run(f0, flag, uin, NU, CS, nx - 8, 1, NUS)
    g = Grid(nx, ny, nz)
    fl, uv = Flags(g, flag), DeviceVector(uin)
    bits = None
    for cfg in range(4):
        for accum in (False, True):
            a, b = Lattice(g, "f64").assign(f0), Lattice(g, "f64").zero_()
            force, acc = ForceSeries(1, nz), Accum(g)
            k_step(a, b, fl, uv, nx, ny, nz, NU, CS, nx - 8, NUS, force, 0, acc=acc if accum else None, cfg=cfg)
            got = b.numpy(np.float64)
            scale = np.abs(want).max()
            fluid = np.broadcast_to(flag == 0, want.shape)
            np.testing.assert_allclose(got[fluid], want[fluid], rtol=TOL, atol=TOL * scale)
            assert_force_close(force.numpy(), want_force, TOL)
            if accum:
                rho = want.sum(0)
                np.testing.assert_allclose(acc.numpy()[0][flag == 0], rho[flag == 0], rtol=TOL, atol=TOL)
            bits = got if bits is None else bits
            np.testing.assert_array_equal(got, bits)           # every configuration gives the same bits
    torch.cuda.synchronize()


@pytest.mark.parametrize("kind", ["flow", "edge"])
def test_in_place_steps_against_oracle(cuda, oracle_mod, kind):
    from stonewall.solver import WallSolver
    nx, ny, nz = 37, 6, 9
    flag, uin = make_mask(nx, ny, nz, 5), inlet(nz, 3)
    f0 = _state(oracle_mod, flag, uin, kind, 12)
    want, want_force = oracle_mod.run(f0, flag, uin, NU, CS, nx - 8, 2, NUS)
    s = WallSolver(flag, uin, NU, CS, nx - 8, 2, nu_sponge=NUS, dtype="f64", pattern="aa", chunk=2)
    s.f[0].assign(f0)
    s.advance(2, use_graphs=False)
    got = s.state_numpy(np.float64)
    fluid = np.broadcast_to(flag == 0, want.shape)
    np.testing.assert_allclose(got[fluid], want[fluid], rtol=TOL, atol=TOL * np.abs(want).max())
    assert_force_close(s.force_series(), want_force, TOL)


def test_uniform_rest_and_nan(cuda, oracle_mod):
    """A uniform rest state stays (its stress is exactly zero); a NaN reaches the status word."""
    from stonewall.lattice import W
    from stonewall.solver import Diverged, WallSolver
    nx, ny, nz = 40, 4, 6
    flag = np.zeros((nx, ny, nz), np.uint8)
    flag[:, :, 0] = 2
    rest = np.broadcast_to(W.astype(np.float64)[:, None, None, None], (19, nx, ny, nz)).copy()
    s = WallSolver(flag, np.zeros(nz, np.float32), NU, CS, nx - 8, 8, dtype="f64")
    s.state.assign(rest)
    s.advance(2)
    fluid = np.broadcast_to(flag == 0, rest.shape)
    np.testing.assert_allclose(s.state_numpy(np.float64)[fluid], rest[fluid], rtol=1e-7)
    rest[4, 20, 2, 3] = np.nan
    s.state.assign(rest)
    with pytest.raises(Diverged):
        s.advance(2)
