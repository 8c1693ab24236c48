"""Relaxation times that the float64 fixed-point collision takes, and those that it leaves to double."""
import numpy as np
import pytest

from test_f64_fixed import W, cells, fx  # noqa: F401  (fx is a fixture)

NAN, INF = np.nan, np.inf


@pytest.mark.parametrize("tau0,c18", [(NAN, 0.25), (0.6, NAN), (INF, 0.25), (0.6, INF), (-INF, 0.25), (0.6, -INF), (0.0, 0.0),
                                      (-0.4, 0.0), (-2.5, 0.25), (0.6, -1e6), (0.3, 0.0), (0.2, 1e-9), (4.1, 0.0),
                                      (1e300, 0.25), (0.6, 1e300), (-1e300, 0.25)])
def test_out_of_range_is_left_to_double(fx, tau0, c18):  # noqa: F811
    """NaN, infinities, negative and zero relaxation times, tau below 1/2 and of 4 and above."""
    f = cells(np.random.default_rng(3), 200, 0.05, 1e-3)
    assert not fx(f, tau0, c18)[2].any()


@pytest.mark.parametrize("tau0,c18", [(0.5, 0.0), (np.nextafter(0.5, 1), 0.0), (0.5, 0.25), (0.5, 1e-300), (1.0, 0.0), (2.0, 0.0),
                                      (3.99, 0.0)])
def test_in_range_is_taken(fx, tau0, c18):  # noqa: F811
    """tau = 1/2 (keep = -1) to just below 4, at the bound of the range's own test."""
    f = cells(np.random.default_rng(4), 2000, 0.05, 1e-3)
    out, mom, ok, err, merr = fx(f, tau0, c18)
    assert ok.all()
    assert (np.abs(err) <= 2.0 ** -53 * np.abs(out) + 2.0 ** -50 * W).all() and np.abs(merr).max() <= 2.0 ** -51


@pytest.mark.gpu
def test_a_model_constant_that_is_no_number_diverges(cuda):
    from gpu_helpers import inlet, make_mask
    from stonewall.solver import Diverged, WallSolver
    s = WallSolver(make_mask(40, 6, 7, 1), inlet(7, 2), 2e-3, NAN, 30, 5, dtype="f64").init(noise=0.02, seed=1)
    with pytest.raises(Diverged):
        s.advance(5, use_graphs=False)
