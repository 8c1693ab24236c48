"""The velocity that the float64 fixed-point collision gives to the running sums keeps its relative precision near rest."""
import numpy as np
import pytest

from test_f64_fixed import W, cells, fx  # noqa: F401  (fx is a fixture)


@pytest.mark.parametrize("u", [0.1, 1e-3, 1e-6, 1e-9, 1e-12])
def test_relative_error_of_the_velocity(fx, u):  # noqa: F811
    """m is exact and u = m / rho: three roundings (of m, of 1 / rho with its last correction, of the product) of 2^-53 each,
    two units more for the reciprocal's own error."""
    f = cells(np.random.default_rng(6), 4000, u, 1e-4)
    out, mom, ok, err, merr = fx(f, 0.6, 0.25)
    assert ok.all()
    assert (np.abs(merr[:, 1:]) <= 5 * 2.0 ** -53 * np.abs(mom[:, 1:])).all()


def test_rest_has_no_velocity(fx):  # noqa: F811
    out, mom, ok, err, merr = fx(np.tile(W, (3, 1)) * [[1.0], [0.7], [1.3]], 0.6, 0.25)
    assert ok.all() and (mom[:, 1:] == 0).all()
