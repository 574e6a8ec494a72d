"""Strided outputs (block covariance, register solver) where the register solver lists every
pixel as ill-conditioned: the listed pixels come out as the plain form gives them, bit for
bit, and the call takes no longer than the plain form."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402

ST = dp.Strides(3, 6)


def _coherent(n, rows, cols, noise=0.1):
    """One speckle field seen on every date, with a little noise: |Gamma| is nearly singular."""
    g = torch.Generator(device="cuda")
    g.manual_seed(n)

    def normal(*shape):
        return torch.randn(shape, dtype=torch.complex64, generator=g, device="cuda")

    ramp = torch.linspace(0.0, 6.0, n, device="cuda")[:, None, None]
    return (normal(rows, cols) + noise * normal(n, rows, cols)) * torch.polar(torch.ones_like(ramp), ramp)


def _listed(monkeypatch, z, hw, **kw):
    """(outputs, number of pixels in the ill-conditioned list of the call's workspace)."""
    import dolphin_gb300._device as D

    kept = []
    workspace = D.workspace
    monkeypatch.setattr(D, "workspace", lambda nbytes, device=None: kept.append(workspace(nbytes)) or kept[-1])
    out = dp.run_phase_linking(z, dp.HalfWindow(*hw), ST, **kw)
    monkeypatch.undo()
    n, rows, cols = z.shape
    p = (rows // ST[0]) * (cols // ST[1])
    at = 0
    for nbytes in (64, 64, 4 * p * n * n, 4 * (p + 64)):  # status, valid bits, matrices, the LU pass's list
        at += -(-nbytes // 256) * 256
    return out, int(kept[0][at:at + 4].view(torch.int32)[0])


def _best(f, reps=12):
    times = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return min(times[2:])


@pytest.mark.parametrize("n", [8, 21, 32, 33, 45, 64])
@pytest.mark.parametrize("masked", [False, True])
def test_same_bits(monkeypatch, n, masked):
    z = _coherent(n, 63, 120)
    kw = {}
    if masked:
        g = torch.Generator(device="cuda")
        g.manual_seed(1)
        kw["neighbor_arrays"] = (torch.rand((21, 20, 11, 23), generator=g, device="cuda") < 0.6).to(torch.uint8)
    a, count = _listed(monkeypatch, z, (5, 11), **kw)
    assert count == 21 * 20
    b = dp.run_phase_linking(z, dp.HalfWindow(5, 11), ST, covariance_form="simt", **kw)
    for name, x, y in zip(a._fields, a, b):
        assert torch.equal(torch.nan_to_num(torch.view_as_real(x) if x.is_complex() else x.float()),
                           torch.nan_to_num(torch.view_as_real(y) if y.is_complex() else y.float())), name


@pytest.mark.parametrize("n,hw", [(21, (5, 11)), (45, (5, 11)), (30, (1, 2))])
def test_time(n, hw):
    z = _coherent(n, 600, 900)

    def run(form):
        return _best(lambda: dp.run_phase_linking(z, dp.HalfWindow(*hw), ST, covariance_form=form))

    assert run("tensor") < 1.1 * run("simt")
