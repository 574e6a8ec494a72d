"""The dense eigensolver for non-converged pixels at the edges of its launch shapes: one
and two warps per pixel (N <= 16, a long and a short list), four above, one row of a
Householder vector per lane and two (N > 32)."""

import numpy as np
import pytest

from oracle import phase_link as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402

HW = (3, 3)


@pytest.mark.parametrize("n,size,listed", [(9, 24, 1), (16, 24, 1), (16, 150, 2500), (17, 24, 1), (32, 24, 1),
                                           (33, 24, 1), (64, 24, 1)])
def test_listed_pixels_against_float64(n, size, listed):
    z = make_stack(StackConfig(nslc=n, rows=size, cols=size + 1, seed=700 + n, gamma_inf=0.02, disk_gamma0=0.95,
                               disk_radius=0.45, ps_frac=0.0))
    flags = np.zeros(z.shape[1:], np.uint8)
    out = dp.run_phase_linking(z, HW, use_evd=True, nonconverged=flags)
    assert flags.sum() >= listed, flags.sum()
    # float64 on the middle 24 x 24 pixels, the windows of the inner 18 x 18 whole
    o = (size - 24) // 2
    crop = z[:, o:o + 24, o:o + 24]
    C = O.estimate_stack_covariance(crop, HW, (1, 1), dtype=np.float64)[3:-3, 3:-3]
    sel = (slice(o + 3, o + 21), slice(o + 3, o + 21))
    f = flags[sel].astype(bool)
    assert f.any()
    A = C * np.abs(C)
    w, v = np.linalg.eigh(A)
    top = np.argmax(np.abs(w), -1)
    x = np.take_along_axis(v, top[..., None, None], -1)[..., 0]
    mag = np.sort(np.abs(w), -1)
    gap = mag[..., -1] - mag[..., -2]
    # |A| to 2^-16 (the tensor-core products of C, twice) and the float32 eigensolver's n eps,
    # over the gap: the error of the vector; at worst all of it on one entry and on the
    # reference's entry
    delta = (2.0**-16 + n * 2.0**-23) * mag[..., -1] / gap
    tol = delta[..., None] * (1 / np.abs(x) + 1 / np.abs(x[..., :1]))
    err = np.abs(np.angle(np.moveaxis(out.cpx_phase[(slice(None), *sel)], 0, -1) * (x * x[..., :1].conj()).conj()))
    print(f"n={n}: {int(flags.sum())} listed, {int(f.sum())} compared, max error {err[f].max():.1e} rad, "
          f"max error / bound {(err / tol)[f].max():.2f}")
    assert (err <= tol)[f].all()
