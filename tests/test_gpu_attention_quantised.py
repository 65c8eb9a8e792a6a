"""The attention block with quantised projections (norm, q, k and v in one call, K rotated
in place, fp16 decode rows into a Q8_0 output projection, the residual in the projection)
against the attention oracle on the dequantised weights."""
import dataclasses

import pytest
import torch

from oracle import attention_oracle as ao
from oracle import moe_oracle as orc
from shark_platform_b200 import synthetic as syn
from helpers import np_planes
from test_attention_oracle import attn_params, masks

pytestmark = pytest.mark.gpu

# about four times what fp16 operands and the rounding of the results to the type give
TOL = {torch.float32: 1.6e-3, torch.float16: 1.6e-3, torch.bfloat16: 1e-2}


def _quantise(kind, like, gen):
    """A planar weight of the shape of `like` with about its standard deviation, and its
    dense values."""
    from shark_platform_b200 import types as T

    n, k = like.shape
    mk = syn.q8_0_planes if kind == syn.Q8_0 else syn.q4_k_planes
    planes = {name: v[0] for name, v in mk(gen, 1, n, k).items()}
    scale = float(like.std() / torch.from_numpy(orc.dequant(kind, np_planes(planes))).float().std())
    for name in ("d", "dmin"):
        if name in planes:
            planes[name] = (planes[name].float() * scale).to(torch.float16)
    dense = torch.from_numpy(orc.dequant(kind, np_planes(planes))).float()
    cuda = {name: v.cuda() for name, v in planes.items()}
    lay = (T.BlockScaledLayout([n, k], cuda["d"], cuda["qs"]) if kind == syn.Q8_0
           else T.SuperBlockOffsetScaled_4_6_Layout([n, k], **cuda))
    return T.PlanarQuantizedTensor(shape=[n, k], layout=lay), dense


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("softcap", [None, 30.0])
@pytest.mark.parametrize("kinds,biases", [
    ((syn.Q8_0,) * 4, ""), ((syn.Q4_K,) * 4, ""), ((syn.Q8_0, syn.Q4_K, syn.Q8_0, syn.Q4_K), ""),
    ((syn.Q8_0,) * 4, "qkv"), ((syn.Q4_K,) * 4, "qkvo")])
@pytest.mark.parametrize("bs,sl", [(2, 48), (40, 32)])  # 96 rows / 2 decode rows; 1280 rows / 40 decode rows
def test_quantised_attention_block_matches_the_oracle(dtype, softcap, kinds, biases, bs, sl):
    from shark_platform_b200 import attention as A, moe, types as T

    c = syn.make_attn_case(seed=81, bs=bs, sl=sl, hidden=512, head_count=8, head_count_kv=4, head_dim=64,
                           softcap=softcap)
    gen = torch.Generator().manual_seed(82)
    c = dataclasses.replace(c, h=c.h.to(dtype).float(), h_decode=c.h_decode.to(dtype).float())
    P = lambda t: T.DefaultPrimitiveTensor(data=t.cuda())
    tree, dense, bias = {"attn_norm": {"weight": P(c.norm_w)}}, {}, {}
    for short, kind, name in zip("qkvo", kinds, ("attn_q", "attn_k", "attn_v", "attn_output")):
        w, dense["w" + short] = _quantise(kind, getattr(c, "w" + short), gen)
        tree[name] = {"weight": w}
        if short in biases:
            bias[short] = torch.randn(w.shape[0], generator=gen) * 0.3
            tree[name]["bias"] = P(bias[short])
    c = dataclasses.replace(c, **dense)
    cache = A.PagedKVCache(transformer_block_count=c.blocks, attn_head_count=c.head_count_kv, attn_head_dim=c.head_dim,
                           block_seq_stride=c.stride, dtype=dtype, device="cuda")
    blk = A.B200PagedAttentionBlock(T.Theta(tree), block_index=c.block_index, cache=cache, head_count=c.head_count,
                                    head_dim=c.head_dim, head_count_kv=c.head_count_kv, rms_epsilon=c.eps,
                                    softcap=c.softcap)
    rope = A.RotaryEmbeddingLayer(rope_dimension_count=c.head_dim, max_seqlen=4096, rope_freq_base=c.rope_base)
    params = dataclasses.replace(attn_params(c), bias=bias)
    geo = ao.CacheGeometry(c.blocks, c.stride, c.head_count_kv, c.head_dim)
    state, slab = cache.allocate(c.pages), geo.allocate(c.pages)
    mask, dmask = masks(c)
    valid = torch.arange(sl)[None, :] < c.seq_lens[:, None]
    clip = lambda m: m.clamp_min(torch.finfo(dtype).min).to(dtype).cuda()
    y = blk(c.h.to(dtype).cuda(), embedding=rope, start_index=0, attention_mask=clip(mask), cache_state=state,
            seq_block_ids=c.page_ids[:, :sl // c.stride].cuda())
    want = ao.attention_block(c.h, params, slab, geo, c.page_ids[:, :sl // c.stride], mask)
    assert moe.device_status() == 0
    assert y.dtype == dtype
    # the rows of real tokens, and the pages that were written
    assert orc.rel_l2(y.float().cpu()[valid], want[valid]) < TOL[dtype]
    assert orc.rel_l2(state[0].float().cpu(), slab) < TOL[dtype]
    yd = blk(c.h_decode.to(dtype).cuda(), embedding=rope, start_positions=c.seq_lens.cuda(), cache_state=state,
             seq_block_ids=c.page_ids.cuda())
    want_d = ao.attention_block(c.h_decode, params, slab, geo, c.page_ids, dmask, start_positions=c.seq_lens)
    assert moe.device_status() == 0
    assert orc.rel_l2(yd.float().cpu(), want_d) < TOL[dtype]
    assert orc.rel_l2(state[0].float().cpu(), slab) < TOL[dtype]
