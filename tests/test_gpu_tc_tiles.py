"""Tiles of the tensor kernel that only some sizes reach: row tiles shorter than 128
(narrow token tiles, where they fill the SMs better), two-stage hand-overs and k
splits, on ragged segments, against the streaming kernel and the oracle."""
import pytest
import torch

from oracle import moe_oracle as orc
from shark_platform_b200 import synthetic as syn
from helpers import b200_block, device_input, oracle_params

pytestmark = pytest.mark.gpu


# ffn 1792 = 16 x 112 = 14 x 128, 768 = 8 x 96 = 6 x 128, 1280 = 10 x 128
@pytest.mark.parametrize("kind", [syn.Q8_0, syn.Q4_K])
@pytest.mark.parametrize("ffn,activation", [(1792, "silu"), (768, "gelu"), (1280, "silu")])
@pytest.mark.parametrize("tokens", [1, 17, 129, 400])
def test_short_row_tiles_match_the_oracle(kind, ffn, activation, tokens):
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("tiles", tokens, 512, ffn, kind=kind, activation=activation, router_bias="zipf",
                        norm_weight="perturbed", seed=71)
    case = syn.make_case(spec)
    h = device_input(case)
    got = b200_block(case, regime="tensor")(h)
    again = b200_block(case, regime="tensor")(h)
    assert torch.equal(got, again), "two runs differ: a race"
    stream = b200_block(case, regime="stream")(h)
    assert moe.device_status() == 0
    assert orc.rel_l2(got.float().cpu(), stream.float().cpu()) < 5e-3  # both rounded to bf16
    want, _ = orc.moe_block(case.h, oracle_params(case), form="per_expert")
    assert orc.rel_l2(got.float().cpu(), want) < 2e-2


def test_fewer_tokens_after_more_still_fit_the_workspace():
    """The k split, and with it the bytes per row, is larger at some smaller token counts."""
    spec = syn.CaseSpec("shrink", 1100, 512, 512, kind=syn.Q8_0, seed=72)
    case = syn.make_case(spec)
    h = device_input(case)
    blk = b200_block(case)
    for n in (1100, 512, 100, 3, 1):
        want = b200_block(case)(h[:n] if h.dim() == 2 else h.reshape(-1, 512)[:n])
        assert torch.equal(blk(h.reshape(-1, 512)[:n]), want)


@pytest.mark.parametrize("tokens", [1, 40, 300])
def test_captured_layer_call_equals_the_eager_one(tokens):
    """The layer's kernels are launched as programmatic dependents: the same under capture."""
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("graph", tokens, 512, 768, kind=syn.Q8_0, seed=73)
    case = syn.make_case(spec)
    blk = b200_block(case)
    h = device_input(case).reshape(tokens, -1).contiguous()
    want = blk(h)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        blk(h)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = blk(h)
    for _ in range(3):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    assert moe.device_status() == 0


# 6 experts: the count rows are added up entry by entry; 129: one CTA past the decode
# front; 515: a last router CTA of three tokens and a last permutation CTA of three
@pytest.mark.parametrize("experts,top_k", [(4, 1), (6, 2), (16, 4), (64, 8)])
@pytest.mark.parametrize("tokens", [129, 515])
@pytest.mark.parametrize("act_dtype", ["bf16", "f32"])
def test_prefill_front_routes_as_the_oracle(experts, top_k, tokens, act_dtype):
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("front", tokens, 512, 256, experts, top_k, kind=syn.Q4_K if experts < 64 else syn.Q8_0,
                        act_dtype=act_dtype, norm_weight="perturbed", router_bias="zipf", seed=74)
    case = syn.make_case(spec)
    y, ex, gates = b200_block(case).layer.forward(device_input(case), want_routing=True)
    assert moe.device_status() == 0
    want, mid = orc.moe_block(case.h, oracle_params(case), form="per_expert")
    # a logit is an fp32 sum of 512 products of order one: off by about sqrt(512) * 2^-24
    # = 1.3e-6, and so is a probability at most; tokens closer to a tie than 1e-5 are left out
    p = torch.sort(mid["prob"], dim=-1, descending=True).values[:, : top_k + 1]
    clear = (p[:, :-1] - p[:, 1:]).min(dim=1).values > 1e-5
    assert clear.float().mean() > 0.9
    assert torch.equal(ex.cpu().to(torch.int64)[clear], mid["experts"][clear])
    assert orc.rel_l2(y.float().cpu().reshape(tokens, -1)[clear], want.reshape(tokens, -1)[clear]) < 2e-2


# one token to each side of where the tensor kernel takes over: 32, and 24 for 4-bit stacks
# of four or more experts
@pytest.mark.parametrize("kind,experts,ffn,first", [(syn.Q8_0, 8, 2048, 32), (syn.Q4_K, 8, 2048, 24),
                                                    (syn.Q4_K, 2, 5120, 32)])
@pytest.mark.parametrize("tokens", [23, 24, 31, 32])
def test_change_over_between_the_kernels(kind, experts, ffn, first, tokens):
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("change", tokens, 512, ffn, experts, 2, kind=kind, norm_weight="perturbed", seed=75)
    case = syn.make_case(spec)
    h = device_input(case)
    got = b200_block(case)(h)
    assert torch.equal(got, b200_block(case, regime="tensor" if tokens >= first else "stream")(h))
    assert moe.device_status() == 0
    want, _ = orc.moe_block(case.h, oracle_params(case), form="per_expert")
    assert orc.rel_l2(got.float().cpu(), want) < 2e-2


# gate/up rows for half of the SMs or fewer: the streaming kernel up to 55 tokens, beside a
# down product on the tensor kernel from 32 (24) on
@pytest.mark.parametrize("kind", [syn.Q8_0, syn.Q4_K])
@pytest.mark.parametrize("tokens", [23, 32, 48, 55, 56])
def test_change_over_of_few_row_tiles(kind, tokens):
    from shark_platform_b200 import moe

    spec = syn.CaseSpec("few_tiles", tokens, 512, 1024, 8, 2, kind=kind, norm_weight="perturbed", router_bias="zipf",
                        seed=76)
    case = syn.make_case(spec)
    h = device_input(case)
    got = b200_block(case)(h)
    if tokens in (23, 56):
        assert torch.equal(got, b200_block(case, regime="tensor" if tokens == 56 else "stream")(h))
    assert moe.device_status() == 0
    want, _ = orc.moe_block(case.h, oracle_params(case), form="per_expert")
    assert orc.rel_l2(got.float().cpu(), want) < 2e-2
