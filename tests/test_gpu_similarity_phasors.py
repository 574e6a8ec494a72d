"""Phasors of the similarity's preparation at the edges of their direct form: magnitudes
around its bounds, zeros, infinities and NaN, layer counts that are not a multiple of its
load group."""

import numpy as np
import pytest

from oracle import similarity as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402


@pytest.mark.parametrize("m", [1, 3, 4, 5, 30])
def test_magnitudes(m):
    rng = np.random.default_rng(m)
    rows, cols = 24, 40
    z = np.exp(1j * rng.uniform(-np.pi, np.pi, (m, rows, cols)))
    # |z|^2 from far below the direct form's range to far above it
    z *= 10.0 ** rng.choice([-22, -15.1, -14.9, 0, 14.9, 15.1, 19], size=(rows, cols))
    z = z.astype(np.complex64)
    z[:, 3, 4:9] = 0
    z[0, 6, 5] = np.nan
    z[-1, 7, 9] = complex(np.inf, -np.inf)
    z[:, 9, 10] = -1.0
    # phasors are float32: a pair's product is off by 4e-7 at most, and so is their mean
    for name in ("median_similarity", "max_similarity"):
        got = getattr(dp, name)(z, search_radius=3)
        want = getattr(O, name)(z, search_radius=3)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        np.testing.assert_allclose(got, want, atol=5e-6, rtol=0)
