"""Outputs whose tiles do not fit the tensor-core covariance (large strides and windows):
the block covariance and the register solver against the plain form, at the edges of the
covariance's block sizes and over masks, options and ragged sizes."""

import numpy as np
import pytest

from parity import phase_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402


@pytest.mark.parametrize("n,hw,strides,kw", [
    (2, (5, 11), (3, 6), {}),
    (7, (5, 11), (3, 6), {"shp": True}),
    (8, (5, 11), (6, 3), {"nodata": True}),
    (14, (9, 31), (2, 5), {}),
    (21, (5, 11), (3, 6), {"shp": True, "nodata": True}),
    (22, (5, 11), (3, 6), {"use_evd": True}),
    (35, (5, 11), (3, 6), {"baseline_lag": 9, "beta": 0.05}),
    (49, (5, 11), (3, 6), {"shp": True}),
    (50, (5, 11), (3, 6), {}),
    (64, (5, 11), (3, 6), {"shp": True, "zero_correlation_threshold": 0.05}),
])
def test_matches_the_plain_form(n, hw, strides, kw):
    kw = dict(kw)
    z = make_stack(StackConfig(nslc=n, rows=61, cols=100, seed=500 + n, ps_frac=0.02))
    if kw.pop("nodata", False):
        z[:, :9, :20] = np.nan
        z[1, 30, 40:50] = np.nan
    nb = None
    if kw.pop("shp", False):
        mean, disp, _ = dp.calc_ps_block(np.abs(z))
        nb = dp.estimate_neighbors(halfwin_rowcol=hw, alpha=0.001, strides=dp.Strides(*strides), mean=mean,
                                   var=(disp * mean) ** 2, nslc=n)
    a = dp.run_phase_linking(z, hw, strides, neighbor_arrays=nb, **kw)
    b = dp.run_phase_linking(z, hw, strides, neighbor_arrays=nb, covariance_form="simt", **kw)
    np.testing.assert_array_equal(a.estimator, b.estimator)
    np.testing.assert_array_equal(a.shp_counts, b.shp_counts)
    np.testing.assert_array_equal(np.isnan(a.cpx_phase), np.isnan(b.cpx_phase))
    good = b.temp_coh > 0.3
    assert good.any()
    assert phase_err(a.cpx_phase[:, good], b.cpx_phase[:, good]).max() < 1e-3
    assert np.abs(a.temp_coh - b.temp_coh)[good].max() < 1e-4
    np.testing.assert_allclose(a.eigenvalues[good], b.eigenvalues[good], rtol=1e-3)
    np.testing.assert_allclose(a.crlb_std_dev[:, good], b.crlb_std_dev[:, good], rtol=3e-3, atol=1e-5)
    # the closure phases are those of the same sums, rounded alike up to N = 32
    if n > 2:
        assert phase_err(np.exp(1j * a.closure_phases[good]), np.exp(1j * b.closure_phases[good])).max() < 1e-5
