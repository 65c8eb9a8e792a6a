"""Quantised linears as one library call (`b200moe_linear`) and the vector path of
the rotary kernel, against plain fp32 torch on the same dequantised weights."""
import ctypes

import pytest
import torch

from oracle import moe_oracle as orc
from shark_platform_b200 import synthetic as syn
from helpers import np_planes

pytestmark = pytest.mark.gpu

# fp16 operands: both the row and the weight carry a relative rounding of 2^-11, so a
# product of them is off by about 2^-11 in the 2-norm; four times that, plus the
# rounding of the output type
TOL = {torch.float32: 2e-3, torch.float16: 2e-3, torch.bfloat16: 6e-3}


def _weight(kind, n, k, seed):
    from shark_platform_b200 import types as T

    gen = torch.Generator().manual_seed(seed)
    mk = syn.q8_0_planes if kind == syn.Q8_0 else syn.q4_k_planes
    planes = {name: v[0] for name, v in mk(gen, 1, n, k).items()}
    dense = torch.from_numpy(orc.dequant(kind, np_planes(planes))).double()
    cuda = {name: v.cuda() for name, v in planes.items()}
    lay = (T.BlockScaledLayout([n, k], cuda["d"], cuda["qs"]) if kind == syn.Q8_0
           else T.SuperBlockOffsetScaled_4_6_Layout([n, k], **cuda))
    return T.PlanarQuantizedTensor(shape=[n, k], layout=lay), dense


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kinds", [(syn.Q8_0,), (syn.Q4_K,), (syn.Q8_0, syn.Q4_K, syn.Q8_0)])
@pytest.mark.parametrize("rows", [1, 7, 96, 97, 385])
def test_linear_rows_with_norm_and_residual(dtype, kinds, rows):
    from shark_platform_b200 import moe

    k, sizes = 512, (512, 256, 256)
    pairs = [_weight(kind, n, k, 50 + i) for i, (kind, n) in enumerate(zip(kinds, sizes))]
    gen = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, k, generator=gen).to(dtype)
    res = torch.randn(rows, sizes[0], generator=gen).to(dtype)
    norm = 1 + 0.1 * torch.randn(k, generator=gen)
    prep = [moe.prepare_linear(w) for w, _ in pairs]
    xd = x.double()
    nd = norm.double() * (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5))
    for args, xr in ((dict(), xd), (dict(norm_weight=norm.cuda(), eps=1e-5), nd)):
        outs = moe.linear_rows(x.cuda(), prep, **args)
        for out, (_, dense) in zip(outs, pairs):
            assert out.dtype == dtype
            assert orc.rel_l2(out.cpu().double(), xr @ dense.mT) < TOL[dtype]
        plus = moe.linear_rows(x.cuda(), prep, residual=res.cuda(), **args)
        assert torch.equal(plus[0], outs[0] + res.cuda())
        for a, b in zip(plus[1:], outs[1:]):
            assert torch.equal(a, b)
    assert moe.device_status() == 0


def test_linear_takes_empty_misaligned_and_strided_inputs():
    from shark_platform_b200 import moe

    w, dense = _weight(syn.Q8_0, 256, 256, 3)
    assert moe.matmul_quantized(torch.empty(0, 256, device="cuda"), w, transpose_rhs=True).shape == (0, 256)
    base = torch.randn(5 * 256 + 3, device="cuda")
    x = base[3:].view(5, 256)  # contiguous, four-byte aligned
    wide = torch.randn(5, 2, 256, device="cuda")[:, 1]
    for v in (x, wide, x.double()):
        y = moe.matmul_quantized(v, w, transpose_rhs=True)
        assert y.dtype == v.dtype
        assert orc.rel_l2(y.cpu().double(), v.cpu().double() @ dense.mT) < TOL[torch.float32]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hd,heads,kv_heads", [(128, 8, 2), (64, 6, 3), (8, 4, 1)])
@pytest.mark.parametrize("tokens_per_seq", [1, 37])
def test_rope_vector_path_equals_the_scalar_path(dtype, hd, heads, kv_heads, tokens_per_seq):
    """The scalar path runs on the same values when the cache type differs from the
    activations'; q, k_out and v_out do not depend on the cache type."""
    from shark_platform_b200 import _cabi as C, moe

    bs, stride, blocks = 3, 16, 2
    per = (tokens_per_seq + 900) // stride + 1
    gen = torch.Generator().manual_seed(hd)
    n = bs * tokens_per_seq
    q = torch.randn(n, heads, hd, generator=gen).to(dtype).cuda()
    k = torch.randn(n, kv_heads, hd, generator=gen).to(dtype).cuda()
    v = torch.randn(n, kv_heads, hd, generator=gen).to(dtype).cuda()
    pos = (torch.arange(tokens_per_seq).repeat(bs) + 900 - 900 * (tokens_per_seq > 1)).to(torch.int32).cuda()
    ids = torch.randperm(bs * per, generator=gen).view(bs, per).to(torch.int32).cuda()
    freqs = (1.0 / 10000.0 ** (torch.arange(hd // 2).float() / (hd // 2))).cuda()
    dt = {torch.float32: C.DT_F32, torch.float16: C.DT_F16, torch.bfloat16: C.DT_BF16}
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    desc = C.KvCacheDesc(blocks, stride, kv_heads, hd, bs * per)
    got = {}
    for cache_dtype in (dtype, torch.float32):
        slab = torch.zeros(bs * per, blocks * 2 * stride * kv_heads * hd, dtype=cache_dtype, device="cuda")
        qq, kk = q.clone(), k.clone()
        # in place for K, V untouched: what the attention block asks for
        C.check(C.lib.b200moe_attn_rope_kv_write(p(qq), p(kk), p(v), p(kk), p(v), dt[dtype], p(slab), dt[cache_dtype],
                                                 ctypes.byref(desc), 1, p(pos), p(ids), p(freqs), n, tokens_per_seq,
                                                 per, heads, st), "rope")
        assert moe.device_status() == 0
        got[cache_dtype] = (qq, kk, slab.float())
    # one rounding of the rotated pair apart at most: the compiler contracts the two paths alike or not
    for a, b in zip(got[dtype], got[torch.float32]):
        d = (a.float() - b.float()).abs().max()
        assert d <= 4 * torch.finfo(dtype).eps, d
    ang = pos.double().cpu()[:, None] * freqs.double().cpu()
    x = q.double().cpu()
    want = torch.stack([x[..., 0::2] * ang.cos()[:, None] - x[..., 1::2] * ang.sin()[:, None],
                        x[..., 1::2] * ang.cos()[:, None] + x[..., 0::2] * ang.sin()[:, None]], -1).flatten(-2)
    # fp32 angles of up to 937 rad carry an absolute error of 937 * 2^-24
    assert orc.rel_l2(got[dtype][0].cpu().double(), want) < torch.finfo(dtype).eps


# K of 256 and 768 leaves k unsplit: from 32 rows on the tensor kernel's drain rounds, adds
# the residual and stores by itself (31 rows: the streaming kernel and the finish kernel)
@pytest.mark.parametrize("k", [256, 768])
@pytest.mark.parametrize("rows", [31, 32, 97, 385])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("kinds", [(syn.Q8_0,), (syn.Q4_K,) * 3, (syn.Q8_0,) * 3])
def test_unsplit_linears_write_finished_outputs(k, rows, dtype, kinds):
    from shark_platform_b200 import moe

    sizes = (512, 256, 256)
    pairs = [_weight(kind, n, k, 90 + i) for i, (kind, n) in enumerate(zip(kinds, sizes))]
    gen = torch.Generator().manual_seed(rows + k)
    x = torch.randn(rows, k, generator=gen)
    prep = [moe.prepare_linear(w) for w, _ in pairs]
    for x_dtype in (torch.float32, torch.float16):
        xs = x.to(x_dtype)
        outs = moe.linear_rows(xs.cuda(), prep, out_dtype=dtype)
        for out, (_, dense) in zip(outs, pairs):
            assert out.dtype == dtype
            assert orc.rel_l2(out.cpu().double(), xs.double() @ dense.mT) < TOL[dtype]
        res = torch.randn(rows, sizes[0], generator=gen).to(dtype).cuda()
        plus = moe.linear_rows(xs.cuda(), prep, residual=res, out_dtype=dtype)
        assert torch.equal(plus[0], outs[0] + res)
        for a, b in zip(plus[1:], outs[1:]):
            assert torch.equal(a, b)
    assert moe.device_status() == 0
