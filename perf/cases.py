"""The work this package is used for, as cases that can be timed and compared.

Every case is one call of a public block on one GPU: `B200MoeBlock` (the MoE FFN
layer of a transformer block, over Q8_0, Q4_K, Q4_1 or dense expert weights) or
`B200PagedAttentionBlock` (the attention half of the same transformer block,
decode and prefill).  Inputs are drawn on the device from a seed with the
distributions of `shark_platform_b200.synthetic`.

  listed()    the cases that stand for the range
  draw(rng)   one more case of the same range
  prepare     the block and the activations a serving loop holds before the call
  run         one forward call
  work        bytes and flops one call cannot do without
  tolerance   what two correct implementations at the same precision may differ by
"""
from __future__ import annotations

import math

import torch

from shark_platform_b200 import attention as A
from shark_platform_b200 import synthetic as syn
from shark_platform_b200 import types as T


def _moe(name, tokens, kind=syn.Q8_0, hidden=4096, ffn=14336, experts=8, top_k=2, activation="silu",
         act_dtype="bf16", out_norm=False, router_bias="", decode=False):
    return {"name": name, "block": "moe", "tokens": tokens, "kind": kind, "hidden": hidden, "ffn": ffn,
            "experts": experts, "top_k": top_k, "activation": activation, "act_dtype": act_dtype,
            "out_norm": out_norm, "router_bias": router_bias, "decode": decode}


def _attn(name, mode, bs, positions, proj=syn.Q8_0, dtype="bf16", hidden=4096, heads=32, kv_heads=8, head_dim=128):
    return {"name": name, "block": "attn", "mode": mode, "bs": bs, "positions": positions, "proj": proj,
            "dtype": dtype, "hidden": hidden, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim}


def listed():
    return [
        # a single stream of tokens: one decode step reads the two experts of one token
        _moe("moe_q8_decode_1", 1, decode=True),
        # the ordinary decode batch
        _moe("moe_q8_decode_32", 32, decode=True),
        # a layer of a deep stack at batch 64 whose router prefers some experts (load imbalance)
        _moe("moe_q8_decode_64_zipf", 64, router_bias="zipf", decode=True),
        # a large decode batch
        _moe("moe_q8_decode_128", 128, decode=True),
        # one short prompt of an odd length
        _moe("moe_q8_prefill_777", 777),
        # the ordinary prefill batch
        _moe("moe_q8_prefill_4096", 4096),
        # the same layer with 4-bit super-block experts
        _moe("moe_q4k_decode_32", 32, kind=syn.Q4_K, decode=True),
        _moe("moe_q4k_prefill_2048", 2048, kind=syn.Q4_K),
        # the widest configuration: GELU experts, output norm, long prompts
        _moe("moe_grok_prefill_8192", 8192, hidden=6144, ffn=32768, activation="gelu", out_norm=True),
        # the smallest layer, dense experts and fp32 activations: launches and host work
        _moe("moe_dense_small_64", 64, kind=syn.DENSE, hidden=512, ffn=1024, act_dtype="f32"),
        # attention of a decode batch of ragged sequences over the page cache, quantised projections
        _attn("attn_decode_32x4096", "decode", 32, 4096),
        # attention of a prompt batch with the model's causal and padding mask
        _attn("attn_prefill_4x1024", "prefill", 4, 1024),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    if rng.random() < 0.25:
        mode = rng.choice(["decode", "decode", "prefill"])
        hidden, heads, kv_heads, head_dim = rng.choice(
            [(4096, 32, 8, 128), (4096, 32, 8, 128), (6144, 48, 8, 128), (2048, 32, 8, 64)])
        proj = rng.choice([syn.Q8_0, syn.Q8_0, syn.Q4_K, syn.DENSE])
        dtype = rng.choice(["bf16", "bf16", "f16"])
        if mode == "decode":
            bs, positions = _log_int(rng, 1, 64), _log_int(rng, 64, 8192)
        else:
            bs, positions = _log_int(rng, 1, 8), 32 * _log_int(rng, 1, 64)
        c = _attn("", mode, bs, positions, proj, dtype, hidden, heads, kv_heads, head_dim)
    else:
        kind = rng.choice([syn.Q8_0] * 5 + [syn.Q4_K] * 3 + [syn.Q4_1, syn.DENSE])
        if kind in (syn.DENSE, syn.Q4_1):
            # drawn on the host: kept small
            hidden, ffn = 256 * rng.randint(1, 4), 256 * rng.randint(2, 8)
            tokens = _log_int(rng, 1, 512)
        else:
            hidden, ffn = rng.choice([(4096, 14336), (4096, 14336), (6144, 16384), (2048, 256 * rng.randint(4, 32)),
                                      (4096, 256 * rng.randint(8, 48))])
            tokens = _log_int(rng, 1, 6144)
        experts, top_k = rng.choice([(8, 2), (8, 2), (8, 2), (16, 2), (8, 4)])
        if experts * ffn * hidden > 8 * 16384 * 6144:
            experts = 8
        while syn.layer_flops(tokens, top_k, hidden, ffn) > syn.layer_flops(8192, 2, 6144, 32768):
            tokens //= 2
        act_dtype = "f32" if kind == syn.DENSE else rng.choice(["bf16", "bf16", "bf16", "f32"])
        c = _moe("", tokens, kind, hidden, ffn, experts, top_k, rng.choice(["silu", "silu", "gelu"]), act_dtype,
                 rng.random() < 0.25, rng.choice(["", "", "zipf"]), tokens <= 128)
    del c["name"]
    return c


# ------------------------------------------------------------------------ MoE layer
def _prepare_moe(case, seed):
    spec = syn.CaseSpec("perf", case["tokens"], case["hidden"], case["ffn"], case["experts"], case["top_k"],
                        kind=case["kind"], activation=case["activation"], act_dtype=case["act_dtype"],
                        out_norm=case["out_norm"], router_bias=case["router_bias"] or None, seed=seed)
    make = syn.make_case if case["kind"] in (syn.DENSE, syn.Q4_1) else syn.make_case_on_device
    layer = make(spec)
    h = syn.case_input(layer)
    # a decode step brings one token per sequence, a prefill one batch of prompt tokens
    h = h.reshape(case["tokens"], 1, -1) if case["decode"] else h
    return {"block": syn.case_block(layer), "h": h.contiguous()}


def _active_experts(case):
    """Expected number of experts that at least one token is routed to."""
    e, k = case["experts"], case["top_k"]
    return e * (1.0 - (1.0 - k / e) ** case["tokens"])


def _work_moe(case):
    d, f, t = case["hidden"], case["ffn"], case["tokens"]
    io = 2 if case["act_dtype"] == "bf16" else 4
    weights = 2 * syn.weight_bytes(case["kind"], f, d) + syn.weight_bytes(case["kind"], d, f)
    return {"bytes": _active_experts(case) * weights + 2 * t * d * io + case["experts"] * d * 4,
            "flops": syn.layer_flops(t, case["top_k"], d, f) + 2 * t * case["experts"] * d}


# ------------------------------------------------------------------------ attention
_STRIDE, _BLOCKS, _BLOCK_INDEX = 32, 2, 1  # positions per page, transformer blocks in the slab, the block called


def _lengths(case):
    """Cached positions before the step (decode) or prompt lengths (prefill):
    ragged, between half of `positions` and all of it."""
    bs, n = case["bs"], case["positions"]
    return [n - (i * (n // 2)) // bs - (1 if case["mode"] == "decode" else 0) for i in range(bs)]


def _projection(kind, n, k, gen):
    """A weight of standard deviation about 0.02 in the given format."""
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    if kind == syn.DENSE:
        return T.DefaultPrimitiveTensor(data=(rn(n, k) * 0.02).to(torch.bfloat16))
    ri = lambda lo, hi, *s: torch.randint(lo, hi, s, generator=gen, device="cuda", dtype=torch.int16)
    if kind == syn.Q8_0:
        lay = T.BlockScaledLayout([n, k], (rn(n, k // 32, 1).abs() * 2.7e-4).to(torch.float16),
                                  ri(-127, 128, n, k // 32, 32).to(torch.int8))
    else:
        # sub-scales and sub-mins in 0..63: w = d*sc*q - dmin*m, about zero-mean
        sup = k // 256
        u8 = lambda *s: ri(0, 256, *s).to(torch.uint8)
        lay = T.SuperBlockOffsetScaled_4_6_Layout(
            [n, k], d=(rn(n, sup, 1).abs() * 6e-5).to(torch.float16),
            dmin=(rn(n, sup, 1).abs() * 4.5e-4).to(torch.float16),
            sb_scales_high=u8(n, sup, 2), sb_scales_low=u8(n, sup, 4),
            sb_mins_high=u8(n, sup, 2), sb_mins_low=u8(n, sup, 4), qs=u8(n, sup, 8, 16))
    return T.PlanarQuantizedTensor(shape=[n, k], layout=lay)


def _prepare_attn(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float16
    d, heads, kvh, hd, bs = case["hidden"], case["heads"], case["kv_heads"], case["head_dim"], case["bs"]
    decode = case["mode"] == "decode"
    weight = lambda n, k: {"weight": _projection(case["proj"], n, k, gen)}
    theta = T.Theta({"attn_norm": {"weight": T.DefaultPrimitiveTensor(data=torch.ones(d, device="cuda"))},
                     "attn_q": weight(heads * hd, d), "attn_k": weight(kvh * hd, d), "attn_v": weight(kvh * hd, d),
                     "attn_output": weight(d, heads * hd)})
    cache = A.PagedKVCache(transformer_block_count=_BLOCKS, attn_head_count=kvh, attn_head_dim=hd,
                           block_seq_stride=_STRIDE, dtype=dtype, device="cuda")
    block = A.B200PagedAttentionBlock(theta, block_index=_BLOCK_INDEX, cache=cache, head_count=heads, head_dim=hd,
                                      head_count_kv=kvh, rms_epsilon=1e-5)
    rope = A.RotaryEmbeddingLayer(rope_dimension_count=hd, max_seqlen=8192)
    per_seq = -(-case["positions"] // _STRIDE)
    pages = bs * per_seq + 1
    state = cache.allocate(pages)
    if decode:
        # scores of standard deviation about 2: a few dozen positions carry the softmax
        state[0].normal_(std=1.5, generator=gen)
    ids = (1 + torch.randperm(pages - 1, generator=gen, device="cuda")).view(bs, per_seq)
    lens = torch.tensor(_lengths(case), device="cuda")
    kw = {"embedding": rope, "cache_state": state, "seq_block_ids": ids}
    if decode:
        h = torch.randn(bs, 1, d, generator=gen, device="cuda").to(dtype)
        kw["start_positions"] = lens
    else:
        sl = per_seq * _STRIDE
        h = torch.randn(bs, sl, d, generator=gen, device="cuda").to(dtype)
        pos = torch.arange(sl, device="cuda")
        blocked = (pos[None, :] > pos[:, None])[None] | (pos[None, None, :] >= lens[:, None, None])
        kw["start_index"] = 0
        kw["attention_mask"] = torch.zeros(bs, 1, sl, sl, dtype=dtype, device="cuda").masked_fill_(
            blocked[:, None], torch.finfo(dtype).min)
    return {"block": block, "h": h, "kw": kw}


def _work_attn(case):
    d, heads, kvh, hd, bs = case["hidden"], case["heads"], case["kv_heads"], case["head_dim"], case["bs"]
    decode = case["mode"] == "decode"
    lens = _lengths(case)
    rows = bs if decode else bs * (-(-case["positions"] // _STRIDE) * _STRIDE)
    qkv_rows = (heads + 2 * kvh) * hd
    weights = syn.weight_bytes(case["proj"], qkv_rows, d) + syn.weight_bytes(case["proj"], d, heads * hd)
    # every cached row is read (decode) or written (prefill) once; the step's own rows are written
    kv_rows = sum(lens) + bs if decode else rows
    attended = sum(n + 1 for n in lens) if decode else sum(n * (n + 1) / 2 for n in lens)
    return {"bytes": weights + 2 * rows * d * 2 + kv_rows * 2 * kvh * hd * 2,
            "flops": 2 * rows * d * (qkv_rows + heads * hd) + 4 * attended * heads * hd}


# ------------------------------------------------------------------------ the interface
def prepare(case, seed):
    return _prepare_moe(case, seed) if case["block"] == "moe" else _prepare_attn(case, seed)


def run(state):
    if "kw" in state:
        y = state["block"](state["h"], **state["kw"])
        return {"y": y, "cache": state["kw"]["cache_state"][0]}
    return state["block"](state["h"])


def work(case):
    return _work_moe(case) if case["block"] == "moe" else _work_attn(case)


def tolerance(case):
    """About four times the distance from the same call evaluated in 64 bits (on the
    same dequantised weights): fp32 activations 2.6e-5 over dense experts and 2.2e-4 ..
    3.9e-4 over quantised ones (fp16 operands), bf16 activations 1.7e-3 (the rounding of
    the result), attention 2.2e-4 .. 3.9e-4 in fp16 and 1.7e-3 .. 3.4e-3 in bf16."""
    if case["block"] == "attn":
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 1.6e-3}
    if case["act_dtype"] == "bf16":
        return {"rel": 7e-3}
    return {"rel": 1e-4 if case["kind"] == syn.DENSE else 1.6e-3}
