"""The block loop with KS neighbours as one CUDA graph: captured, then replayed on other
data of the same shapes, each time the eager loop's results."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import dolphin_gb300.workflow as W  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402


def test_captured_and_replayed():
    W.clear_loop_graphs()
    kw = dict(half_window=(2, 3), strides=(1, 2), block_shape=(20, 24), shp_method="ks", shp_alpha=0.05)
    for seed in (11, 12):
        z = make_stack(StackConfig(nslc=8, rows=52, cols=60, seed=seed, ps_frac=0.03))
        z[:, :30, :40] = 0  # the first block is skipped
        zd = torch.from_numpy(z).cuda()
        eager = W.run_wrapped_phase_single(zd, **kw)
        graphed = W.run_wrapped_phase_single(zd, graph=True, **kw)
        assert len(W._LOOP_GRAPHS) == 1
        for name, a, b in zip(eager._fields, graphed, eager):
            if b is not None:
                np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy(), err_msg=name)
    W.clear_loop_graphs()
