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


def _graph_of(fn):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = fn()
    return graph, y


def _fill_free_memory():
    """Tensors in whatever the allocator has free, with values to find again."""
    return [torch.full((n,), 7.0, device="cuda") for n in (1 << 8, 1 << 12, 1 << 16, 1 << 18, 1 << 20) for _ in range(12)]


def test_captured_layer_call_keeps_its_scratch_after_a_larger_call():
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("graph_grow", 1100, 512, 512, kind=syn.Q8_0, seed=14)
    case = syn.make_case(spec)
    blk = syn.case_block(case, "auto", "cuda")
    h = syn.case_input(case, "cuda").reshape(1100, -1)
    small = h[:40].contiguous()
    want = blk(small)
    graph, y = _graph_of(lambda: blk(small))
    blk(h)
    others = _fill_free_memory()
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert all(bool((t == 7.0).all()) for t in others), "a replay wrote into other tensors"
    assert moe.device_status() == 0


def test_one_layer_on_two_streams():
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("streams", 300, 1024, 2048, kind=syn.Q8_0, seed=15)
    case = syn.make_case(spec)
    blk = syn.case_block(case, "auto", "cuda")
    h = syn.case_input(case, "cuda").reshape(300, -1)
    parts = [h[:40].contiguous(), h[40:300].contiguous()]
    want = [blk(p) for p in parts]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in parts]
    got = [[], []]
    for _ in range(30):
        for s, p, out in zip(streams, parts, got):
            with torch.cuda.stream(s):
                out.append(blk(p))
    torch.cuda.synchronize()
    for w, out in zip(want, got):
        assert all(torch.equal(w, y) for y in out)
    assert moe.device_status() == 0


def test_captured_decode_attention_keeps_its_scratch_after_a_larger_call():
    from shark_platform_b200 import moe
    from test_gpu_attention import _block

    c = syn.make_attn_case(seed=16, bs=24, sl=1024)
    blk, cache, rope = _block(c, cache_dtype=torch.float16)
    state = cache.allocate(c.pages)
    state[0].normal_()
    ids, lens, h = c.page_ids.cuda(), c.seq_lens.cuda(), c.h_decode.cuda()
    call = lambda n: blk(h[:n], embedding=rope, start_positions=lens[:n], cache_state=state, seq_block_ids=ids[:n])
    want = call(2)
    graph, y = _graph_of(lambda: call(2))
    call(24)
    others = _fill_free_memory()
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert all(bool((t == 7.0).all()) for t in others), "a replay wrote into other tensors"
    assert moe.device_status() == 0
