"""FP8 attention that quantizes its own queries (b200q_fp8_attention): bit for bit the operand launch for Q, K and V followed by
b200q_fp8_sdpa_strided, for every input type, at the edges of a tile of queries, for rows off a 32-byte boundary, values beyond the
given range, NaN and infinities."""
import ctypes

import pytest
import torch

DT = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}


def _both(q, k, v, am, causal):
    from tensorrt_b200 import _lib

    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    B, Hq, Sq, D = q.shape
    Hkv, Sk = k.shape[1:3]
    strides = (ctypes.c_int64 * 9)(*q.stride()[:3], *k.stride()[:3], *v.stride()[:3])
    out_strides = (ctypes.c_int64 * 3)(Hq * Sq * D, Sq * D, D)
    p = lambda t: t.data_ptr() if t.numel() else None  # noqa: E731
    ref, out = (torch.full((B, Hq, Sq, D), 3.0, dtype=q.dtype, device="cuda") for _ in range(2))
    stride = max((Sk + 15) // 16 * 16, 16)
    qc, kc = torch.empty(B, Hq, Sq, D, dtype=torch.uint8, device="cuda"), torch.empty(B, Hkv, Sk, D, dtype=torch.uint8, device="cuda")
    vt, sc = torch.empty(B, Hkv, D, stride, dtype=torch.uint8, device="cuda"), torch.empty(3, device="cuda")
    a = [t.data_ptr() for t in am]
    assert lib.b200q_fp8_attention_quantize(p(q), p(k), p(v), DT[q.dtype], strides, *a, p(qc), p(kc), p(vt), p(sc), B, Hq, Hkv, Sq, Sk, stride, D, st) == 0
    s = sc.data_ptr()
    assert lib.b200q_fp8_sdpa_strided(p(qc), p(kc), p(vt), s, s + 4, s + 8, p(ref), out_strides, DT[q.dtype], B, Hq, Hkv, Sq, Sk, stride, D, D ** -0.5,
                                      causal, st) == 0
    n = lib.b200q_fp8_attention_workspace_bytes(B, Hkv, Sk, D)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    call = lambda size: lib.b200q_fp8_attention(p(q), p(k), p(v), DT[q.dtype], strides, *a, p(out), out_strides, ws.data_ptr(), size, B, Hq, Hkv, Sq, Sk, D,  # noqa: E731
                                                D ** -0.5, causal, st)
    assert call(n - 1) != 0                          # refused before anything is launched
    assert call(n) == 0
    return ref, out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk,D,causal", [
    (1, 1, 1, 1, 1, 16, 0), (2, 4, 2, 127, 129, 48, 1), (1, 2, 1, 128, 128, 128, 1), (1, 3, 3, 300, 77, 80, 0), (2, 2, 1, 129, 300, 112, 1), (1, 2, 1, 40, 0, 64, 0)])
def test_equals_the_separate_calls(b200, B, Hq, Hkv, Sq, Sk, D, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(Sq + Sk)
    q, k, v = ((torch.randn(B, h, s, D, device="cuda", generator=g) * 3).to(dtype) for h, s in ((Hq, Sq), (Hkv, Sk), (Hkv, Sk)))
    am = [(t.float().abs().max().reshape(1) if t.numel() else torch.full((1,), 2.0, device="cuda")) for t in (q, k, v)]
    am[0] = am[0] * 0.5                              # some queries saturate, a piece beyond 512 / 448 of the range among them
    views = [q, torch.empty(B, Hq, Sq, D + 32 // q.element_size() // 2, dtype=dtype, device="cuda")[..., :D].copy_(q),
             q.transpose(1, 2).contiguous().transpose(1, 2)]
    for t in views:
        ref, out = _both(t, k, v, am, causal)
        assert torch.equal(ref, out)
    assert b200.capi.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 0.0])   # the shared-divisor range, beyond it (true division), an all-zero range
def test_values_that_are_not_finite(b200, scale, dtype):
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(1, 1, 130, 64, device="cuda", generator=g).to(dtype) for _ in range(3))
    q[0, 0, 3, 5], q[0, 0, 4, 17], q[0, 0, 129, 63], q[0, 0, 7, 0] = float("nan"), float("inf"), float("-inf"), -0.0
    am = [torch.full((1,), a, device="cuda") for a in (2.0 * scale, 2.0, 2.0)]
    ref, out = _both(q, k, v, am, 0)
    assert torch.equal(ref.view(torch.int32 if dtype == torch.float32 else torch.int16), out.view(torch.int32 if dtype == torch.float32 else torch.int16))


@pytest.mark.gpu
@pytest.mark.parametrize("keys", [640, 700])              # five key tiles, and more
@pytest.mark.parametrize("ctas", ["sms - 1", "sms", "sms + 1", "2 * sms", "2 * sms + 1"])
def test_ways_of_launching(b200, ctas, keys):
    """One CTA per SM, a plain and a programmatic launch, by the number of CTAs and the length of the key axis: the same bits."""
    heads = eval(ctas, {"sms": torch.cuda.get_device_properties(0).multi_processor_count})
    g = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randn(1, heads, s, 64, device="cuda", generator=g).bfloat16() for s in (100, keys, keys))
    am = [t.float().abs().max().reshape(1) for t in (q, k, v)]
    for causal in (0, 1):
        ref, out = _both(q, k, v, am, causal)
        assert torch.equal(ref, out)
    assert b200.capi.device_status() == 0
