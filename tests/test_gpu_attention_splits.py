"""Decode attention where the number of position splits is at its largest: one kv head and
a long context, against softmax(q K^T / sqrt(hd)) V in 64 bits over the same cache."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# 16385 and 20000 positions: 32 and 39 splits of a 16-bit cache; 40000: 64
@pytest.mark.parametrize("cache_dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 1e-2), (torch.float16, 1.6e-3)])
@pytest.mark.parametrize("kv_heads,seq", [(1, 16385), (1, 20000), (2, 40000)])
def test_long_context_of_few_kv_heads(kv_heads, seq, cache_dtype, tol):
    from shark_platform_b200 import _cabi as C, moe

    stride, hd, heads, bs = 32, 128, kv_heads * 8, 1
    per = -(-seq // stride)
    gen = torch.Generator(device="cuda").manual_seed(seq)
    slab = (torch.randn(per + 3, 2, stride, kv_heads, hd, generator=gen, device="cuda") * 0.7).to(cache_dtype)
    ids = torch.randperm(per + 3, generator=gen, device="cuda")[:per].to(torch.int32).view(1, per)
    q = torch.randn(bs, heads, hd, generator=gen, device="cuda").to(cache_dtype)
    lens = torch.tensor([seq - 5], dtype=torch.int32, device="cuda")
    out = torch.empty_like(q)
    dt = {torch.float32: C.DT_F32, torch.float16: C.DT_F16, torch.bfloat16: C.DT_BF16}[cache_dtype]
    desc = C.KvCacheDesc(1, stride, kv_heads, hd, per + 3)
    nbytes = C.lib.b200moe_attn_decode_scratch_bytes(ctypes.byref(desc), bs, heads, per * stride)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    C.check(C.lib.b200moe_attn_decode(p(q), dt, p(slab), dt, ctypes.byref(desc), 0, p(ids), p(lens), bs, per, heads,
                                      per * stride, hd ** -0.5, 0.0, p(out), dt, p(scratch), nbytes,
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "attn_decode")
    assert moe.device_status() == 0
    kv = slab[ids[0].long()].transpose(0, 1).reshape(2, per * stride, kv_heads, hd)[:, :seq - 5].double()
    k, v = (t.repeat_interleave(8, dim=1) for t in kv)
    w = torch.softmax(torch.einsum("hd,nhd->hn", q[0].double(), k) * hd ** -0.5, dim=-1)
    want = torch.einsum("hn,nhd->hd", w, v)
    # fp32: sums of 128 and of up to 40000 products; 16 bits: probabilities and result rounded to the type
    assert (out[0].double() - want).norm() / want.norm() < tol
