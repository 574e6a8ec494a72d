"""A captured block loop owns every buffer that it writes: memory allocated after the
capture is not written by a replay."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300.workflow as W  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402


def test_replay_leaves_other_tensors_alone():
    W.clear_loop_graphs()
    rows, cols = 52, 60
    z = torch.from_numpy(make_stack(StackConfig(nslc=8, rows=rows, cols=cols, seed=3, ps_frac=0.03))).cuda()
    amp = z.abs()
    mean = amp.mean(0)
    kw = dict(half_window=(2, 3), strides=(1, 2), block_shape=(20, 24), shp_method="glrt", shp_alpha=0.05,
              amp_mean=mean, amp_dispersion=amp.std(0, unbiased=False) / mean, similarity=False, graph=True)
    W.run_wrapped_phase_single(z, **kw)
    # tensors of each raster's size, as many as any of them can have been given back
    others = [torch.full((rows * cols // 2,), 7, dtype=torch.int32, device="cuda") for _ in range(64)]
    others += [torch.full((rows * cols,), 7, dtype=torch.int32, device="cuda") for _ in range(64)]
    W.run_wrapped_phase_single(z, **kw)
    torch.cuda.synchronize()
    assert all(bool((t == 7).all()) for t in others)
    (entry,) = W._LOOP_GRAPHS.values()
    kept = {t.data_ptr() for part in entry for t in (part if isinstance(part, (tuple, list)) else [part])
            if isinstance(t, torch.Tensor)}
    assert len(kept) >= 5 + 9 - 1  # the inputs, the nine rasters
    W.clear_loop_graphs()
