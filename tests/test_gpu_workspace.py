"""Who owns the scratch memory of a call, and that what was reserved is enough."""
import pytest
import torch

from shark_platform_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most,counts", [(32, (20, 24, 30, 31, 1)), (1024, (716, 762, 805, 1000, 3))])
def test_pipeline_takes_every_smaller_batch(most, counts):
    """The k split of the Mixtral layer's down product, and with it the workspace, is larger
    at some smaller counts."""
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("pipe", most, 4096, 14336, kind=syn.Q8_0, seed=13)
    case = syn.make_case_on_device(spec, "cuda")
    blk = syn.case_block(case, "auto", "cuda")
    h = syn.case_input(case, "cuda").reshape(most, -1)
    pipe = moe.HostPipeline(blk.layer, most, h.dtype)
    ins = [h[:n].cpu().pin_memory() for n in counts]
    outs = [torch.empty_like(x).pin_memory() for x in ins]
    for x, y in zip(ins, outs):
        pipe.submit(x, y)
    pipe.drain()
    pipe.close()
    for n, y in zip(counts, outs):
        assert torch.equal(y, blk(h[:n]).cpu())
    assert moe.device_status() == 0
