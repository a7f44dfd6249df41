"""Operands of the FP8 attention in one launch (b200q_fp8_attention_quantize), strided inputs and results, and the
abs-max of three column ranges: bit for bit what the separate calls on contiguous copies give."""
import ctypes

import pytest
import torch

import oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk,D,stride", [
    (1, 1, 1, 1, 1, 16, 16), (2, 4, 2, 127, 129, 48, 144), (1, 2, 1, 128, 128, 128, 128), (1, 3, 3, 300, 77, 80, 512), (2, 2, 1, 5, 0, 64, 16)])
def test_codes_and_scales(b200, B, Hq, Hkv, Sq, Sk, D, stride, dtype):
    from tensorrt_b200 import _lib

    g = torch.Generator().manual_seed(Sq + Sk)
    q, k, v = ((torch.randn(B, h, s, D, generator=g) * 3).to(dtype) for h, s in ((Hq, Sq), (Hkv, Sk), (Hkv, Sk)))
    am = [(t.float().abs().max() if t.numel() else torch.tensor(2.0)) for t in (q, k, v)]
    am[1] = am[1] * 0.5                                        # some keys saturate
    dev = [t.cuda() for t in (q, k, v)]
    amd = [a.reshape(1).cuda() for a in am]
    qc, kc = torch.full((B, Hq, Sq, D), 0xAA, dtype=torch.uint8, device="cuda"), torch.full((B, Hkv, Sk, D), 0xAA, dtype=torch.uint8, device="cuda")
    vt, sc = torch.full((B, Hkv, D, stride), 0xAA, dtype=torch.uint8, device="cuda"), torch.zeros(3, device="cuda")
    st = (ctypes.c_int64 * 9)(Hq * Sq * D, Sq * D, D, Hkv * Sk * D, Sk * D, D, Hkv * Sk * D, Sk * D, D)
    args = lambda ts: [t.data_ptr() if t.numel() else None for t in ts]  # noqa: E731
    assert _lib.load().b200q_fp8_attention_quantize(*args(dev), {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype], st, *args(amd),
                                                    *args([qc, kc, vt]), sc.data_ptr(), B, Hq, Hkv, Sq, Sk, stride, D,
                                                    torch.cuda.current_stream().cuda_stream) == 0
    for t, a, codes, i in ((q, am[0], qc, 0), (k, am[1], kc, 1)):
        ref, rs = o.fp8_quantize(t, a)
        assert torch.equal(codes.cpu(), ref) and sc[i].item() == rs.item()
    if Sk:
        ref, rs = o.fp8_quantize(v, am[2])
        assert sc[2].item() == rs.item()
        assert torch.equal(vt[..., :Sk].cpu(), ref.transpose(2, 3)) and int(vt[..., Sk:].max() if stride > Sk else 0) == 0


@pytest.mark.parametrize("batch,s,n_q,n_kv,d", [(1, 1, 1, 1, 16), (2, 130, 4, 2, 64), (3, 64, 8, 1, 48), (1, 300, 2, 2, 128)])
def test_packed_projection_equals_head_major_copies(b200, batch, s, n_q, n_kv, d):
    capi = b200.capi
    g = torch.Generator().manual_seed(s)
    qkv = torch.randn(batch * s, (n_q + 2 * n_kv) * d, generator=g).bfloat16().cuda()
    heads = lambda t, n: t.reshape(batch, s, n, d).permute(0, 2, 1, 3).contiguous()  # noqa: E731
    q, k, v = (heads(t, n) for t, n in zip(qkv.split([n_q * d, n_kv * d, n_kv * d], 1), (n_q, n_kv, n_kv)))
    ref = capi.fp8_sdpa(q, k, v, capi.amax(q), capi.amax(k), capi.amax(v), True).permute(0, 2, 1, 3).reshape(batch * s, n_q * d)
    assert torch.equal(capi.fp8_sdpa_packed(qkv, batch, n_q, n_kv, d, True), ref)
    # views of every kind give what their contiguous copies give
    views = [q.transpose(1, 2).contiguous().transpose(1, 2), torch.empty(batch, n_q, s, d + 8, dtype=q.dtype, device="cuda")[..., :d].copy_(q),
             torch.empty(batch, n_q, s, d + 1, dtype=q.dtype, device="cuda")[..., 1:].copy_(q), q.transpose(2, 3).contiguous().transpose(2, 3)]
    plain = capi.fp8_sdpa(q, k, v, capi.amax(q), capi.amax(k), capi.amax(v))
    for t in views:
        if t.is_contiguous() and t.data_ptr() % 16:            # one row, misaligned: refused, as every other kernel does
            continue
        out = capi.fp8_sdpa(t, k, v, capi.amax(q), capi.amax(k), capi.amax(v))
        assert out.is_contiguous() and torch.equal(out, plain)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,c", [(1, (16, 0, 0)), (7, (64, 16, 16)), (333, (512, 128, 128)), (5000, (256, 0, 48))])
def test_amax_columns(b200, rows, c, dtype):
    from tensorrt_b200 import _lib

    x = torch.randn(rows, sum(c), generator=torch.Generator().manual_seed(rows)).to(dtype).cuda()
    out = torch.full((3,), 7.0, device="cuda")
    assert _lib.load().b200q_amax_columns(x.data_ptr(), {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype], rows, *c, out.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream) == 0
    for i, part in enumerate(x.split(list(c), 1)):
        assert out[i].item() == (part.float().abs().max().item() if part.numel() else 0.0)
