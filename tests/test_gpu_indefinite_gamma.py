"""Flagged pixels that the dense eigensolver cannot take over: |Gamma| + 1e-6 I positive to
float32 elimination but indefinite in double.  They keep the last iterate of the inverse
iteration, as without the fallback."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402


@pytest.mark.parametrize("n,noise", [(6, 4e-4), (8, 5e-4), (10, 5e-4), (10, 6e-4), (20, 1e-3)])
def test_keep_the_last_iterate(n, noise):
    rng = np.random.default_rng(n)
    rows, cols, hw = 400, 410, (2, 3)
    # one phase history for all pixels (coherence near 1), fewer looks than make |Gamma| safe
    hist = np.exp(1j * rng.uniform(-np.pi, np.pi, (n, 1, 1)))
    z = hist * (1 + noise * (rng.normal(size=(n, rows, cols)) + 1j * rng.normal(size=(n, rows, cols))))
    z = (10 * z).astype(np.complex64)
    flags = np.zeros((rows, cols), np.uint8)
    kw = dict(zero_correlation_threshold=1e-3)  # |Gamma| by the correctly rounded root
    out = dp.run_phase_linking(z, hw, nonconverged=flags, **kw)
    last = dp.run_phase_linking(z, hw, eigh_fallback=False, **kw)
    # |Gamma| as the kernels round it; its smallest eigenvalue in double
    C = dp.estimate_stack_covariance(z, hw)
    im2 = (C.imag * C.imag).astype(np.float64)
    gamma = np.sqrt((C.real.astype(np.float64) ** 2 + im2).astype(np.float32)).astype(np.float64)
    indefinite = np.linalg.eigvalsh(gamma + 1e-6 * np.eye(n))[..., 0] < -1e-12
    keep = flags.astype(bool) & indefinite & (out.estimator == 1)
    assert keep.any()
    print(f"n={n} noise={noise}: {int(flags.sum())} flagged, {int(indefinite.sum())} indefinite, {int(keep.sum())} both (EMI)")
    np.testing.assert_array_equal(out.cpx_phase[:, keep], last.cpx_phase[:, keep])
    np.testing.assert_array_equal(out.temp_coh[keep], last.temp_coh[keep])
    np.testing.assert_array_equal(out.eigenvalues[keep], last.eigenvalues[keep])
