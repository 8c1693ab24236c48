"""Moving cells over the whole density range that the float64 fixed-point collision takes, its ends above all."""
import fractions

import numpy as np
import pytest

from test_f64_fixed import W, cells, fx  # noqa: F401  (fx is a fixture)


def held(fx, f, tau0=0.6, c18=0.25):
    """Every cell that is taken meets the bound of test_error_against_long_double, rho and u included."""
    out, mom, ok, err, merr = fx(f, tau0, c18)
    assert (np.abs(err[ok]) <= 2.0 ** -53 * np.abs(out[ok]) + 2.0 ** -50 * W).all()
    assert np.abs(merr[ok]).max(initial=0.0) <= 2.0 ** -51
    return ok


def test_density_of_one_half_and_its_neighbours(fx):  # noqa: F811
    """rho = 1/2 + k 2^-59 with m != 0: 1 / rho rounds to 2 at and next to 1/2."""
    rng = np.random.default_rng(11)
    rows, steps = [], [0, 1, 7, 16, 31, 32, 33, 63, 64, 65, 128, 129, 512, 4096]
    for f in np.round(cells(rng, 300, 0.05, 1e-3) * 0.5 * 2.0 ** 59) * 2.0 ** -59:
        for k in steps + [-s for s in steps[1:]]:
            g = f.copy()                               # multiples of 2^-59
            g[0] = float(fractions.Fraction(1, 2) - sum(map(fractions.Fraction, g[1:])))
            rest = fractions.Fraction(1, 2) + fractions.Fraction(k, 2 ** 59) - sum(map(fractions.Fraction, g))
            g[7 + g[7:].argmin()] += float(rest)       # one below 2^-6 takes what the rest population rounds off
            assert sum(map(fractions.Fraction, g)) == fractions.Fraction(1, 2) + fractions.Fraction(k, 2 ** 59)
            rows.append(g)
    held(fx, np.array(rows))


def moving(rng, lo, hi):
    """Cells of densities in [lo, hi), the rest population's excess over its limit moved to the axes."""
    f = cells(rng, 4000, 0.08, 1e-3)
    f *= (rng.uniform(lo, hi, len(f)) / f.sum(1))[:, None]
    over = np.maximum(f[:, 0] - 0.4999, 0.0)
    f[:, 0] -= over
    f[:, 1:7] += over[:, None] / 6
    return f


@pytest.mark.parametrize("lo,hi", [(0.5, 0.5 + 1e-12), (0.5, 0.52), (0.5, 2.0), (1.98, 2.0), (2.0 - 1e-12, 2.0)])
def test_density_range(fx, lo, hi):  # noqa: F811
    ok = held(fx, moving(np.random.default_rng(12), lo, hi))
    assert ok.mean() > 0.9 or lo > 1.9                 # (next to 2 the moved excess leaves rho - 3 tr B above 2: refused)


@pytest.mark.parametrize("lo,hi", [(0.5, 0.52), (1.98, 2.0), (2.0 - 1e-12, 2.0)])
def test_density_range_relaxed_to_equilibrium(fx, lo, hi):  # noqa: F811
    """tau = 1.1: next to 2 these cells are taken as well."""
    assert held(fx, moving(np.random.default_rng(13), lo, hi), 1.1, 0.0).mean() > 0.9
