"""Strided outputs whose tiles do not fit the tensor-core covariance: the errors against the
FP64 form are those of the plain form over every pixel, the coherent and the
ill-conditioned ones among them.

The last iterates are compared (no dense eigensolver), where all three agree about the
estimator.  Both float32 forms stop at a step below 1e-5: a pixel that the register solver
keeps has taken 24 steps at most, a factor of 0.62 each or less, which leaves 2.6e-5; 1e-4
covers a step more or less on either side.  Root mean squares: a float32 phasor's last place
(6e-8) is allowed for."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402


def _coherent(n, rows, cols, noise):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)

    def normal(*shape):
        return torch.randn(shape, dtype=torch.complex64, generator=g, device="cuda")

    ramp = torch.linspace(0.0, 6.0, n, device="cuda")[:, None, None]
    return (normal(rows, cols) + noise * normal(n, rows, cols)) * torch.polar(torch.ones_like(ramp), ramp)


def _rms(x):
    return x[~torch.isnan(x)].double().square().mean().sqrt().item()


@pytest.mark.parametrize("n", [5, 12, 21, 33, 45, 64])
@pytest.mark.parametrize("noise,hw,kw", [
    (None, (5, 11), {}),
    (None, (3, 4), {}),
    (0.1, (5, 11), {}),
    (0.3, (5, 5), {}),
    (0.5, (5, 5), {}),
    (0.1, (5, 11), {"use_evd": True}),
    (None, (3, 4), {"use_evd": True}),
    (None, (5, 11), {"beta": 0.01}),
    (None, (5, 11), {"zero_correlation_threshold": 0.1}),
])
def test_errors_are_the_plain_forms(n, noise, hw, kw):
    if noise is None:
        z = torch.from_numpy(make_stack(StackConfig(nslc=n, rows=150, cols=240, seed=n, ps_frac=0.02))).cuda()
    else:
        z = _coherent(n, 150, 240, noise)
    ref, plain, got = (dp.run_phase_linking(z, dp.HalfWindow(*hw), dp.Strides(3, 6), covariance_form=form,
                                            eigh_fallback=False, **kw) for form in ("fp64", "simt", "tensor"))
    assert torch.equal(plain.estimator, got.estimator)
    same = ref.estimator == plain.estimator
    for field, factor, rms_floor, top_floor in (("cpx_phase", 1.25, 6e-8, 1e-4), ("temp_coh", 1.25, 6e-8, 1e-5),
                                                ("crlb_std_dev", 1.1, 1e-8, 1e-4)):
        r, p, w = (getattr(o, field)[..., same] for o in (ref, plain, got))
        if field == "crlb_std_dev":
            ep, ew = ((x - r).abs()[1:] / r[1:] for x in (p, w))
        else:
            ep, ew = (p - r).abs(), (w - r).abs()
        assert torch.equal(torch.isnan(p), torch.isnan(w)), field
        if bool(torch.isnan(ep).all()):
            continue
        assert _rms(ew) <= factor * _rms(ep) + rms_floor, field
        assert torch.nan_to_num(ew).max() <= 1.5 * torch.nan_to_num(ep).max() + top_floor, field
