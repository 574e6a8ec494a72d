"""Register solver at the edges of its instances: odd depths (a padded row), the smallest
and largest of each group size, and pixels whose coherence has zero entries (their
temporal coherence takes the pairs one by one)."""

import numpy as np
import pytest

from oracle import phase_link as O
from parity import phase_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402


@pytest.mark.parametrize("n", [2, 3, 8, 9, 15, 16, 17, 31, 32, 33, 34, 46, 47, 63, 64])
def test_depths_and_zero_entries(n):
    z = make_stack(StackConfig(nslc=n, rows=14, cols=15, seed=300 + n, ps_frac=0.0))
    C = O.estimate_stack_covariance(z, (6, 6), (1, 1)).reshape(-1, n, n)
    for k, (i, j) in enumerate([(n - 1, 0), (1, 0), (n - 1, n - 2)]):
        C[3 + 7 * k, i, j] = C[3 + 7 * k, j, i] = 0.0
    vec, val, est, crlb, tc, clos = dp.process_coherence_matrices(C, num_looks=5.0, return_metrics=True)
    rv, rl, re_, rc = O.process_coherence_matrices(C, num_looks=5.0)
    rtc = O.estimate_temp_coh(rv, C)
    np.testing.assert_array_equal(est, re_)
    good = rtc > 0.3
    assert phase_err(vec[good], rv[good]).max() < 1e-3
    assert np.abs(tc - rtc)[good].max() < 1e-4
    np.testing.assert_allclose(val, rl, rtol=1e-3)
    np.testing.assert_allclose(crlb, rc, rtol=3e-3, atol=1e-5)
