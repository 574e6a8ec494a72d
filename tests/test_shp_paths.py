"""The SHP tests' direct forms against the general ones: the KS envelope against the merge
walk (CPU), and both mask kernels at the edges of their tiles, words and value ranges."""

import numpy as np
import pytest

from oracle import phase_link as O


def ks_envelope(n, cutoff):
    """(lo, hi) indices into x1 that bound sample t of x2 (-1: unbounded), as the kernel's
    host side derives them from the admissible intervals."""
    T = np.zeros(n + 1)
    for k in range(1, n + 1):
        T[k] = T[k - 1] + 1 / n
    hi = [max(np.nonzero(np.abs(T[i] - T) < cutoff)[0], default=-1) for i in range(n + 1)]
    env_lo, env_hi = [-1] * n, [-1] * n
    for t in range(n - 1, -1, -1):
        m = next((i for i in range(n + 1) if hi[i] >= t + 1), n + 1)
        env_lo[t] = m - 1
        if 1 <= m <= n:
            env_hi[m - 1] = t
    return env_lo, env_hi


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 20, 33])
def test_ks_envelope_is_the_walk(n):
    rng = np.random.default_rng(n)
    decided = 0
    for cutoff in [1e-3, 0.1, 1 / n, 2 / n, 0.5, 0.43, 0.97, 1.0]:
        lo, hi = ks_envelope(n, cutoff)
        # continuous samples, and samples with many ties
        for x in (rng.normal(size=(400, 2, n)) + rng.normal(size=(400, 2, 1)),
                  rng.integers(0, max(2, n), size=(400, 2, n)).astype(float)):
            x = np.sort(x, axis=-1)
            x1, x2 = x[:, 0], x[:, 1]
            low = np.stack([x1[:, i] if i >= 0 else np.full(400, -np.inf) for i in lo], -1)
            high = np.stack([x1[:, i] if i >= 0 else np.full(400, np.inf) for i in hi], -1)
            f = np.minimum(x2 - low, high - x2).min(-1)
            want = O.ks_max_cdf_dist(x1, x2) < cutoff
            np.testing.assert_array_equal((f > 0)[f != 0], want[f != 0])
            decided += int((f != 0).sum())
    assert decided > 1000


gpu = pytest.mark.gpu


def _dp():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU")
    import dolphin_gb300 as dp

    return dp


@gpu
@pytest.mark.parametrize("n", [1, 2, 4, 5, 21, 64])
@pytest.mark.parametrize("hw,strides", [((1, 2), (1, 1)), ((2, 17), (1, 1)), ((3, 2), (3, 6)), ((0, 0), (2, 1))])
def test_ks_masks(n, hw, strides):
    dp = _dp()
    rng = np.random.default_rng(100 * n + hw[1])
    rows, cols = 26, 75
    amp = rng.rayleigh(3.0, size=(n, rows, cols)).astype(np.float32)
    amp[:, :, 40:] *= 1.7
    amp[:, 5:12] = np.round(amp[:, 5:12])  # ties
    amp[0, 8, 10:20] = np.nan
    amp[-1, 14, 30:34] = np.inf
    amp[:, 15, 30:34] = np.inf
    amp[:, 16:18, 50:60] = 0.0
    got = dp.estimate_neighbors(halfwin_rowcol=hw, strides=dp.Strides(*strides), amp_stack=amp, alpha=0.05, method="ks")
    np.testing.assert_array_equal(got, O.estimate_neighbors_ks(amp, hw, strides, 0.05))


@gpu
@pytest.mark.parametrize("nslc,alpha", [(1, 0.001), (20, 0.05), (20, 0.001), (300, 0.5), (2, 1e-9)])
@pytest.mark.parametrize("hw,strides", [((2, 3), (1, 1)), ((1, 20), (1, 1)), ((60, 1), (1, 1)), ((2, 2), (3, 6))])
def test_glrt_masks(nslc, alpha, hw, strides):
    """Every decision is the float64 one, over ordinary, zero, negative, tiny, huge,
    infinite and NaN scales."""
    dp = _dp()
    rng = np.random.default_rng(nslc + hw[0])
    rows, cols = 125, 77
    mean = rng.gamma(9.0, 0.3, size=(rows, cols)).astype(np.float32)
    var = (0.3 * mean**2 * rng.gamma(9.0, 0.11, size=mean.shape)).astype(np.float32)
    mean[40:44, 10:30] *= 1e-12
    var[40:44, 10:30] *= 1e-24
    mean[50, 10:14], var[50, 10:14] = 0.0, 0.0
    mean[51, 10:14], var[51, 10:14] = 0.0, -1.0
    var[52, 10], var[53, 10] = np.nan, np.inf
    mean[100:104, 40:60] *= 1e11
    var[100:104, 40:60] *= 1e22
    got = dp.estimate_neighbors(halfwin_rowcol=hw, strides=dp.Strides(*strides), mean=mean, var=var, nslc=nslc,
                                alpha=alpha)
    with np.errstate(all="ignore"):
        want = O.estimate_neighbors_glrt(mean, var, hw, strides, nslc, alpha, exact=True)
        # a negative scale has no logarithm
        neg = ((var + mean**2) / 2 < 0).astype(np.float32)
    if neg.any():
        bad = O.estimate_neighbors_glrt(mean, np.where(neg > 0, np.nan, var), hw, strides, nslc, alpha, exact=True)
        want = want & bad
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("alpha", [0.5, 0.05, 0.01, 0.001, 1e-9])
def test_ks_critical_distance_is_the_scan(alpha):
    from dolphin_gb300 import _build
    from dolphin_gb300.shp import ks_critical_distance

    _build.build_library()
    for n in [1, 2, 3, 5, 10, 17, 30, 45, 64, 300]:
        assert ks_critical_distance(n, alpha) == O.ks_critical_distance(n, alpha)


def test_glrt_threshold_is_the_quantile():
    stats = pytest.importorskip("scipy.stats")
    from dolphin_gb300.shp import glrt_threshold

    for alpha in [0.0, 1e-12, 1e-5, 0.001, 0.01, 0.05, 0.3, 0.9, 1.0]:
        assert glrt_threshold(alpha) == float(stats.chi2.ppf(1 - alpha, df=1))


@gpu
@pytest.mark.parametrize("nslc", [3, 4, 30, 1000])
@pytest.mark.parametrize("hx", [0, 1, 3, 7, 11, 14, 15, 16, 31])
def test_glrt_interval_ends(nslc, hx):
    """Scales within a few float32 steps of the interval's two ends, at every remainder of a
    window row's offsets: each decision is the float64 one."""
    dp = _dp()
    rng = np.random.default_rng(nslc + hx)
    rows, cols = 19, 70
    c = np.exp(10.827566170662733 / nslc)  # the 0.999 quantile of chi2(1)
    end = 2 * c - 1 + 2 * np.sqrt(c * (c - 1))
    level = end ** rng.integers(0, 3, size=(rows, cols))
    var = (2 * level * (1 + rng.integers(-6, 7, size=level.shape) * 2.0**-24)).astype(np.float32)
    mean = np.zeros_like(var)
    got = dp.estimate_neighbors(halfwin_rowcol=(2, hx), mean=mean, var=var, nslc=nslc, alpha=0.001)
    want = O.estimate_neighbors_glrt(mean, var, (2, hx), (1, 1), nslc, 0.001, exact=True)
    np.testing.assert_array_equal(got, want)
    assert want.any()


@gpu
@pytest.mark.parametrize("n,hw", [(2, (78, 79)), (4, (55, 56)), (1, (400, 1))])
def test_ks_windows_at_the_limit(n, hw):
    """Windows whose samples fill shared memory: the unpadded pitch, one pixel per CTA."""
    dp = _dp()
    rng = np.random.default_rng(n)
    # every third pixel, the first one with a whole window
    r, c = (1 + 3 * ((h + 1) // 3) for h in hw)
    rows, cols = r + hw[0] + 4, c + hw[1] + 5
    amp = rng.rayleigh(3.0, size=(n, rows, cols)).astype(np.float32)
    got = dp.estimate_neighbors(halfwin_rowcol=hw, strides=dp.Strides(3, 3), amp_stack=amp, alpha=0.05, method="ks")
    x = np.sort(amp, axis=0)
    win = x[:, r - hw[0]:r + hw[0] + 1, c - hw[1]:c + hw[1] + 1]
    want = O.ks_max_cdf_dist(np.broadcast_to(x[:, r, c], (win[0].size, n)), win.reshape(n, -1).T) < \
        O.ks_critical_distance(n, 0.05)
    want = want.reshape(win.shape[1:])
    want[hw] = False
    np.testing.assert_array_equal(got[r // 3, c // 3], want)


def test_ks_critical_distance_without_the_library(monkeypatch, tmp_path):
    from dolphin_gb300 import _lib
    from dolphin_gb300.shp import ks_critical_distance

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "missing.so")
    for n, alpha in [(1, 0.05), (20, 0.001), (64, 0.5)]:
        assert ks_critical_distance(n, alpha) == O.ks_critical_distance(n, alpha)
