"""Mask bytes of the tensor-core covariance: window widths and image widths at which a tile
row's bytes start at every alignment, ragged last tiles, and bytes other than 0 and 1."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402


@pytest.mark.parametrize("hw,strides,shape", [
    ((0, 0), (1, 1), (17, 33)), ((1, 0), (1, 1), (20, 35)), ((0, 3), (1, 1), (16, 31)), ((2, 2), (1, 1), (33, 16)),
    ((3, 7), (1, 2), (18, 70)), ((5, 11), (1, 1), (21, 47)), ((2, 15), (2, 1), (37, 50)), ((1, 31), (1, 1), (19, 65)),
])
def test_counts_and_coherence(hw, strides, shape):
    rng = np.random.default_rng(hw[0] * 100 + hw[1])
    n, (rows, cols) = 6, shape
    z = (rng.normal(size=(n, rows, cols)) + 1j * rng.normal(size=(n, rows, cols))).astype(np.complex64)
    wy, wx = 2 * hw[0] + 1, 2 * hw[1] + 1
    orow, ocol = rows // strides[0], cols // strides[1]
    m = rng.integers(0, 3, size=(orow, ocol, wy, wx)).astype(np.uint8)
    m[m == 2] = rng.choice([16, 128, 255], size=int((m == 2).sum()))
    zd, md = torch.from_numpy(z).cuda(), torch.from_numpy(m).cuda()
    out = dp.run_phase_linking(zd, hw, strides, neighbor_arrays=md)
    np.testing.assert_array_equal(out.shp_counts.cpu().numpy(), (m != 0).sum((2, 3)))
    a = dp.estimate_stack_covariance(zd, hw, strides, md)
    b = dp.estimate_stack_covariance(zd, hw, strides, md, covariance_form="simt")
    # two bf16 parts per product: 2^-16 of sqrt(amp_i amp_j), and the float32 sums
    assert (a - b).abs().max() < 2.0**-15
