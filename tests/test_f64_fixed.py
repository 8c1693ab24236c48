"""The float64 collision in fixed point (csrc/sw_f64.cuh) against long double on the CPU, over the whole range it
takes, and which cells it leaves to the double form."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fx") / "fx.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I",
                    os.path.join(PKG, "csrc"), os.path.join(ROOT, "tests", "fx_collide.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731

    def run(f, tau0, c18):
        f = np.ascontiguousarray(f, np.float64)
        n = len(f)
        tau0, c18 = (np.ascontiguousarray(np.broadcast_to(v, n), np.float64) for v in (tau0, c18))
        out, mom, ok = np.zeros((n, 19)), np.zeros((n, 4)), np.zeros(n, np.uint8)
        err, merr = np.zeros((n, 19)), np.zeros((n, 4))
        lib.fx_cells(ptr(f), n, ptr(tau0), ptr(c18), ptr(out), ptr(mom), ptr(ok))
        lib.long_cells(ptr(f), n, ptr(tau0), ptr(c18), ptr(out), ptr(mom), ptr(err), ptr(merr))
        return out, mom, ok.astype(bool), err, merr
    return run


def cells(rng, n, u, neq):
    from stonewall.lattice import C
    rho = 1 + rng.uniform(-0.05, 0.05, (n, 1))
    vel = rng.uniform(-u, u, (n, 3))
    cu = 3 * vel @ C.T
    a = rng.uniform(-neq, neq, (n, 3, 3))
    q = np.einsum("ia,ib->iab", C, C) - np.eye(3) / 3
    return W * (rho * (1 + cu + 0.5 * cu * cu - 1.5 * (vel ** 2).sum(1, keepdims=True))
                + 4.5 * np.einsum("iab,nab->ni", q, a + a.transpose(0, 2, 1)) / 2)


@pytest.mark.parametrize("u", [0.0, 1e-9, 0.03, 0.1, 0.2])
@pytest.mark.parametrize("neq", [0.0, 1e-14, 1e-8, 1e-4, 2e-2])
def test_error_against_long_double(fx, u, neq):
    """One rounding of the result (2^-53 of it) plus the products' units and the double scalars: below 2^-50 w."""
    rng = np.random.default_rng(5)
    f = cells(rng, 4000, u, neq)
    tau0 = 0.5 + 10.0 ** rng.uniform(-9, 0, 4000)
    out, mom, ok, err, merr = fx(f, tau0, rng.choice([0.0, 0.25, 0.65], 4000))
    assert ok.mean() > (0.99 if u <= 0.1 else 0.5)
    assert (np.abs(err[ok]) <= 2.0 ** -53 * np.abs(out[ok]) + 2.0 ** -50 * W).all()
    assert np.abs(merr[ok]).max() <= 2.0 ** -51


@pytest.mark.parametrize("i,limit", [(0, 0.5), (3, 0.25), (12, 0.125)])
def test_range_of_a_population(fx, i, limit):
    """A population is taken from 2^-10 to just below its limit, and nothing outside of that is."""
    f = np.tile(W, (10, 1))
    f[:, i] = [limit, np.nextafter(limit, 0), 2.0 ** -10, np.nextafter(2.0 ** -10, 0), 0.0, -W[i], np.inf, -np.inf, np.nan,
               1e-310]
    f[1, 0] -= 0.1 if i else 0.0                       # (keeps the results in range)
    ok = fx(f, 0.6, 0.25)[2]
    assert ok[0] == 0 and not ok[3:].any()
    rest = np.tile(W, (1, 1))
    assert fx(rest, 0.6, 0.25)[2].all()


def test_cells_left_to_double(fx):
    """Density outside [1/2, 2), a stress entry of 1/2 and results below 2^-10 are reported, not computed."""
    base = np.tile(W, (4, 1))
    base[0] *= 0.49
    base[1] = np.minimum(W * 1.4, [0.49] + [0.249] * 6 + [0.1249] * 12)
    base[1, 1:] = [0.249] * 6 + [0.1249] * 12             # density above 2
    base[2, 1], base[2, 2], base[2, 3:7] = 0.249, 0.249, 0.002   # a large stress: negative results at tau = 1/2
    assert not fx(base[:3], 0.5 + 1e-12, 0.0)[2].any()
    assert fx(base[3:], 0.5 + 1e-12, 0.0)[2].all()


def test_rounding_carries_into_the_exponent(fx):
    """Rest states scaled around powers of two: results next to 2^-k round up to it."""
    s = np.concatenate([np.nextafter(v, [0, 1]) for v in (0.5625, 1.125, 0.75, 1.5, 0.9, 1.0)])
    out, _, ok, err, _ = fx(W * s[:, None], 0.6, 0.25)
    assert ok.all() and (np.abs(err) <= 2.0 ** -53 * out + 2.0 ** -50 * W).all()
