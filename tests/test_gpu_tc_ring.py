"""The 128-token variant of the tensor kernel (41 to 96 expected rows per matrix) with
weights that do not fit L2, so that loads land late and out of step with the groups that
wait for them: many passes, bit-equal, against the streaming kernel and the oracle."""
import dataclasses

import pytest
import torch

from oracle import moe_oracle as orc
from shark_platform_b200 import synthetic as syn
from helpers import ExpertWeightStream, sampled_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [syn.Q8_0, syn.Q4_K])
def test_layer_of_the_128_token_variant(kind):
    from shark_platform_b200 import moe

    # 8 experts, top 2: 164 tokens are 41 rows per expert, 387 are 96
    spec = syn.CaseSpec("ring", 387, 4096, 14336, kind=kind, seed=11)
    case = syn.make_case_on_device(spec, "cuda")
    auto, stream = syn.case_block(case, "auto", "cuda"), syn.case_block(case, "stream", "cuda")
    weights = ExpertWeightStream(case, keep=True)
    for tokens in (164, 200, 380, 387):
        h = syn.case_input(dataclasses.replace(case, h=case.h[:, :tokens].contiguous()), "cuda")
        y = auto(h)
        for _ in range(40):
            assert torch.equal(auto(h), y), "two passes differ: a race"
        want = stream(h)
        assert moe.device_status() == 0
        assert orc.rel_l2(y.float().cpu(), want.float().cpu()) < 5e-3  # both rounded to bf16
        if tokens in (200, 380):
            sel = torch.arange(0, tokens, 8)
            ref, mid = sampled_oracle(case, tokens, sel, weights)
            p = torch.sort(mid["prob"], dim=-1, descending=True).values[sel, : spec.top_k + 1]
            clear = (p[:, :-1] - p[:, 1:]).min(dim=1).values > 1e-5
            got = y.reshape(tokens, -1)[sel.cuda()].float().cpu()
            assert orc.rel_l2(got[clear], ref.reshape(len(sel), -1)[clear]) < 2e-2


@pytest.mark.parametrize("kind", [syn.Q8_0, syn.Q4_K])
@pytest.mark.parametrize("rows", [41, 64, 96])
def test_linears_of_the_128_token_variant(kind, rows):
    from shark_platform_b200 import moe, types as T

    n = k = 4096
    count = 9 if kind == syn.Q8_0 else 18  # 160 MB of weights
    spec = syn.CaseSpec("ring_linear", 1, k, n, count, 1, kind=kind, seed=12)
    planes = syn.make_case_on_device(spec, "cuda").gate
    ws, dense = [], []
    for e in range(count):
        p = {name: v[e] for name, v in planes.items()}
        lay = (T.BlockScaledLayout([n, k], p["d"], p["qs"]) if kind == syn.Q8_0
               else T.SuperBlockOffsetScaled_4_6_Layout([n, k], **p))
        ws.append(moe.prepare_linear(T.PlanarQuantizedTensor(shape=[n, k], layout=lay)))
        dense.append(orc.dequant_torch(kind, {name: v.cpu() for name, v in p.items()}) if e < 3 else None)
    gen = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, k, generator=gen).to(torch.bfloat16).cuda()
    groups = [ws[i:i + 3] for i in range(0, count, 3)] + [[w] for w in ws]  # q, k and v together, and one by one
    first = [moe.linear_rows(x, g, out_dtype=torch.float32) for g in groups]
    for _ in range(25):
        for g, ys in zip(groups, first):
            for a, b in zip(moe.linear_rows(x, g, out_dtype=torch.float32), ys):
                assert torch.equal(a, b), "two passes differ: a race"
    assert moe.device_status() == 0
    flat = [y for ys in first[:count // 3] for y in ys]
    for e, w in enumerate(dense):
        if w is not None:
            # fp16 operands: 2^-11 relative, four times that
            assert orc.rel_l2(flat[e].cpu().double(), x.cpu().double() @ w.double().mT) < 2e-3
