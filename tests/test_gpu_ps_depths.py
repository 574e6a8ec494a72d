"""PS selection at the edges of the kernel's depths, with and without NaN samples."""

import numpy as np
import pytest

from oracle import phase_link as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402


@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 17, 32, 33, 56, 57, 63, 64, 65])
def test_bit_exact(n):
    rng = np.random.default_rng(n)
    mag = rng.lognormal(0, 0.4, size=(n, 19, 27)).astype(np.float32)
    mag[rng.random(mag.shape) < 0.01] = np.nan
    mag[n // 2, 2, 3] = np.inf
    mag[:, 4, 5] = np.nan
    mag[:, 6, 7] = 0.0
    with np.errstate(all="ignore"):
        want = O.calc_ps_block(mag.copy(), 0.3, n // 2)
    for a, b in zip(dp.calc_ps_block(mag, 0.3, n // 2), want):
        np.testing.assert_array_equal(a, b)
