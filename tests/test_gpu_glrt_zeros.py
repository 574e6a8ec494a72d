"""GLRT masks of a scene with a zero-filled border (no data: mean and variance 0): the
masks are the oracle's, and the border does not cost more than the scene itself."""

import numpy as np
import pytest

from oracle import phase_link as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402

# dates and alpha of each test form: the interval, the ratio, the logarithms
FORMS = [(30, 0.001), (2, 0.001), (1, 1e-10)]


def _scene(rows, cols, border):
    rng = np.random.default_rng(5)
    mean = rng.gamma(4.0, 1.0, (rows, cols)).astype(np.float32)
    var = (mean * rng.uniform(0.1, 1.0, (rows, cols))).astype(np.float32)
    mean[:, :border] = 0
    var[:, :border] = 0
    return mean, var


@pytest.mark.parametrize("nslc,alpha", FORMS)
def test_masks(nslc, alpha):
    mean, var = _scene(40, 60, 25)
    kw = dict(halfwin_rowcol=(3, 6), alpha=alpha, mean=mean, var=var, nslc=nslc)
    with np.errstate(all="ignore"):
        expect = O.estimate_neighbors_glrt(mean, var, (3, 6), (1, 1), nslc, alpha)
    assert not expect[:, :25].any()
    got = dp.estimate_neighbors(**kw)
    assert not got[:, :25].any()
    # decisions within the oracle's own float32 rounding may differ
    assert (got != expect).mean() < 1e-4


@pytest.mark.parametrize("nslc,alpha", FORMS)
def test_time(nslc, alpha):
    def best(border):
        m, v = (torch.from_numpy(x).cuda() for x in _scene(1024, 1024, border))
        kw = dict(halfwin_rowcol=(5, 11), alpha=alpha, mean=m, var=v, nslc=nslc)
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            dp.estimate_neighbors(**kw)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[1:])

    # a pixel of the border has no neighbour: no test of it needs the double-precision route
    assert best(512) < 1.5 * best(0) + 0.05
