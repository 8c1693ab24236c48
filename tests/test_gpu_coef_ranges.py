"""sw_coefficients and sw_coef_stats at the ends of their ranges: rows longer than one integer block, values near
the fixed-point limit, series shorter than a cluster, and infinities among the coefficients."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,size", [(3, 70000, 2 ** 36), (9, 8, 2 ** 62), (1, 1, 2 ** 40), (33, 65536, 2 ** 62),
                                       (5, 65537, 2 ** 61)])
def test_coefficients_against_exact_sums(cuda, n, nz, size):
    import torch
    from stonewall.fields import ForceSeries
    from stonewall.metrics import device_coefficients
    rng = np.random.default_rng(nz)
    v = rng.integers(-size, size, (n, nz, 2), dtype=np.int64)
    fs = ForceSeries(n, nz)
    fs.data.copy_(torch.from_numpy(v))
    UH, H, ny = 0.05, 40.0, 160
    got = device_coefficients(fs, UH, H, ny).cpu().numpy()
    qa = 0.5 * UH * UH * H * ny
    w = 2 * np.arange(nz) - 1
    for t in range(n):
        fx, fz = (sum(int(a) for a in v[t, :, k]) / 2 ** 40 for k in (0, 1))
        m = sum(int(a) * int(b) for a, b in zip(v[t, :, 0], w)) / 2 ** 41
        # each lane rounds its sum once, the butterfly three times: 2^-50 of the magnitudes summed
        mag = np.abs(v[t].astype(np.float64)).sum(0) / 2 ** 40
        mag_m = (np.abs(v[t, :, 0].astype(np.float64)) * np.abs(w)).sum() / 2 ** 41
        for g, e, s in ((got[0, t], fx / qa, mag[0] / qa), (got[1, t], fz / qa, mag[1] / qa),
                        (got[2, t], m / (qa * H), mag_m / (qa * H))):
            assert abs(g - e) <= 2.0 ** -50 * s


@pytest.mark.parametrize("n,n_spin", [(1, 0), (2, 1), (255, 0), (2047, 3), (2048, 0), (2049, 1), (6200, 55)])
def test_stats_against_numpy(cuda, n, n_spin):
    import ctypes

    import torch
    from stonewall import _native as N
    from stonewall.metrics import STAT_KEYS, stats
    rng = np.random.default_rng(n)
    coef = -1.0 + 0.3 * rng.standard_normal((3, n))          # negative: the maxima are not the initial value
    dev, out = torch.from_numpy(coef).cuda(), torch.empty(6, dtype=torch.float64, device="cuda")

    def run():
        N.check(N.lib().sw_coef_stats(ctypes.c_void_p(dev.data_ptr()), n, n_spin, ctypes.c_void_p(out.data_ptr()),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "sw_coef_stats")
        return dict(zip(STAT_KEYS, out.cpu().tolist()))
    got, want = run(), stats(coef[0], coef[2], coef[1], n_spin)
    for k in STAT_KEYS:
        assert abs(got[k] - want[k]) <= 1e-12 * max(abs(want[k]), 1.0), k
    assert got["CdMax"] == want["CdMax"] and got["CmMax"] == want["CmMax"]
    dev[0, n - 1], dev[2, n - 1] = np.inf, np.nan
    got = run()
    assert got["CdMax"] == np.inf and np.isnan(got["Cm"])
    rest = coef[2, n_spin:n - 1]
    assert got["CmMax"] == (rest.max() if len(rest) else -np.inf)      # fmax ignores a NaN
