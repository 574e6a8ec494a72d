"""A batch whose stacks share a covariance kernel's shared memory to the last kilobyte: the
small stack's masks fit with an odd number of words per pixel, the batch's do not."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU container
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from dolphin_gb300.batch import PhaseLinkBatch  # noqa: E402
from dolphin_gb300.simulate import StackConfig, make_stack  # noqa: E402


@pytest.mark.parametrize("depths,hw", [((6, 12), (6, 26)), ((6, 12), (14, 29)), ((6, 12), (20, 9))])
def test_batch_at_the_shared_memory_limit(depths, hw):
    stacks = [torch.from_numpy(make_stack(StackConfig(nslc=n, rows=2 * hw[0] + 20, cols=2 * hw[1] + 21, seed=n,
                                                      ps_frac=0.02))).cuda() for n in depths]
    forms = {n: "tensor" for n in depths}
    per = PhaseLinkBatch(stacks, hw, forms=forms, graph=False, persistent=False).run()
    outs = PhaseLinkBatch(stacks, hw, forms=forms, graph=False, persistent=True).run()
    for a, b in zip(per, outs):
        assert torch.equal(a.shp_counts, b.shp_counts)
        assert torch.equal(torch.view_as_real(a.cpx_phase).nan_to_num(), torch.view_as_real(b.cpx_phase).nan_to_num())
        assert torch.equal(a.temp_coh, b.temp_coh)
