"""PS selection where NaN samples are scattered over the scene, so that every warp holds a
pixel with one: slower than without NaNs, but not by several times."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300 as dp  # noqa: E402


def _best(mag):
    times = []
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        dp.calc_ps_block(mag, 0.25, mag.shape[0])
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return min(times[2:])


@pytest.mark.parametrize("n", [30, 60])  # one load after the other, 60 took 3.8 times as long
def test_scattered_nans(n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    mag = torch.rand((n, 2048, 2048), generator=g, device="cuda") + 0.5
    plain = _best(mag)
    mag[torch.rand(mag.shape, generator=g, device="cuda") < 0.01] = float("nan")
    assert _best(mag) < 2.8 * plain + 0.03
