"""Exponentials and probabilities of the FP8 attention.  bf16 results take an eighth of the exponentials from the FMA pipe and keep
those of the last key tile; fp16 and fp32 results take all of them, twice, from the special-function unit.  Both forms: the range of
scores where the result underflows, NaN at every column of a key tile (which unit computes a score depends on its column), every
probability code against 64 bits; and the stored bits of the second."""
import hashlib

import pytest
import torch

import oracle as o

DT = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}


def _sdpa(lib, qc, kc, vt, scales, B, H, Sq, Sk, D, causal, dtype):
    out = torch.full((B, H, Sq, D), 7.0, device="cuda", dtype=dtype)
    s = scales.data_ptr()
    assert lib.b200q_fp8_sdpa(qc.data_ptr(), kc.data_ptr(), vt.data_ptr(), s, s + 4, s + 8, out.data_ptr(), DT[dtype], B, H, H, Sq, Sk, vt.shape[-1], D,
                              D ** -0.5, causal, torch.cuda.current_stream().cuda_stream) == 0
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("spread", [0.0, 1.0, 8.0, 60.0])
def test_range_of_scores(b200, spread, causal):
    """Scores within one value, and down to 2^-127 and 2^-8000 of the largest: zero codes there, no wrapped exponents.  Tolerance of
    test_gpu_attention (rel-L2 <= 1e-2: a probability beside a rounding boundary may take the next code)."""
    g = torch.Generator().manual_seed(int(spread) + 1)
    q = (torch.randn(1, 2, 256, 64, generator=g) * spread).bfloat16()
    k = (torch.randn(1, 2, 256, 64, generator=g) * spread).bfloat16()
    v = torch.randn(1, 2, 256, 64, generator=g).bfloat16()
    am = [t.float().abs().max() for t in (q, k, v)]
    ref = o.fp8_sdpa_ref(q, k, v, *am, is_causal=causal)
    out = b200.capi.fp8_sdpa(q.cuda(), k.cuda(), v.cuda(), *(a.cuda() for a in am), is_causal=causal)
    assert o.rel_l2(out.float().cpu(), ref.float()) <= 1e-2


# one key tile, several, and a ragged last one
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("sk,causal", [(128, 0), (256, 0), (256, 1), (200, 1), (300, 0), (300, 1)])
def test_nan_key_reaches_every_row_that_sees_it(b200, sk, causal, dtype):
    """And nothing else.  (As codes: a quantizer with a given range clamps NaN to it.)"""
    from tensorrt_b200 import _lib

    lib, D, H = _lib.load(), 32, sk                      # head h: key h is NaN
    g = torch.Generator(device="cuda").manual_seed(sk)
    codes = lambda *shape: (torch.randn(*shape, device="cuda", generator=g)).to(torch.float8_e4m3fn).view(torch.uint8)  # noqa: E731
    stride = (sk + 15) // 16 * 16
    qc, kc, vt = codes(1, H, sk, D), codes(1, H, sk, D), codes(1, H, D, stride)
    vt[..., sk:] = 0
    for h in range(H):
        kc[0, h, h, 5] = 0x7F
    out = _sdpa(lib, qc, kc, vt, torch.ones(3, device="cuda"), 1, H, sk, sk, D, causal, dtype)
    seen = torch.ones(sk, sk, dtype=torch.bool, device="cuda").tril() if causal else torch.ones(sk, sk, dtype=torch.bool, device="cuda")
    nan = out[0].isnan()                                  # [head = NaN key, query, D]
    assert torch.equal(nan.all(dim=2), seen.t()) and torch.equal(nan.any(dim=2), seen.t())


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("scale", [0.002, 0.02, 0.125, 0.5])
def test_every_probability_code(b200, scale, dtype):
    """Causal rows of 1 to 200 keys whose scores and quantized operands are small integers, so that both contractions are exact:
    a value may differ from 64 bits by the rounding to its type and by those probabilities alone that lie so near a boundary of E4M3
    that fp32 may take either code.  How near: the exponent's argument carries the roundings of its factor (4), of the offset (2) and
    of the FMA (1), each 2^-24 of the largest score in bits, and those of log2(448 / row sum) (16 in units of 2^-24); ex2, the sum of
    200 terms and the quotient add 2^-21."""
    S, D = 200, 64
    g = torch.Generator().manual_seed(int(scale * 1000))
    q, k, v = (torch.randint(-n, n + 1, (1, h, S, D), generator=g) for n, h in ((4, 4), (4, 2), (8, 2)))
    am = torch.tensor(448.0, device="cuda")               # scale 1: the codes are the integers
    out = b200.capi.fp8_sdpa(*(t.to(dtype).cuda() for t in (q, k, v)), am, am, am, is_causal=True, scale=scale)[0].double().cpu()
    s = (q[0].double() @ k[0].repeat_interleave(2, 0).double().transpose(1, 2)) * float(torch.tensor(scale, dtype=torch.float32))
    p = 448.0 * torch.softmax(s.masked_fill(~torch.ones(S, S, dtype=torch.bool).tril(), float("-inf")), -1)
    bits = s.abs().amax(-1, keepdim=True) * 1.4427
    near = 0.6931 * (8 * bits + 16) * 2.0 ** -24 + 2.0 ** -21
    code = lambda t: o.e4m3_decode(o.e4m3_encode(t.float())).double()  # noqa: E731
    vv = v[0].repeat_interleave(2, 0).double()
    ref = code(p) @ vv / 448.0
    either = (code(p * (1 + near)) - code(p * (1 - near))) @ vv.abs() / 448.0
    half_step = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -22}[dtype]   # fp32: the kernel's own two roundings
    assert ((either > 0).sum() < 0.01 * either.numel()) and bool(((out - ref).abs() <= either + half_step * ref.abs() + 2.0 ** -25).all())


# Written by the kernel with every exponential on the special-function unit and two exponentials per score.
STORED = {("fp16", 0): "24ac576e8932384a", ("fp16", 1): "a6672c6ae7a6e4c9", ("fp16", 2): "d87886f81c1219a9",
          ("fp32", 0): "7901623bf340a69a", ("fp32", 1): "451f732068b8aeaa", ("fp32", 2): "39519c128d196f6c"}
SHAPES = [(1, 2, 2, 130, 130, 64, True), (2, 4, 2, 200, 333, 80, False), (1, 2, 1, 300, 300, 128, True)]


@pytest.mark.gpu
@pytest.mark.parametrize("name,case", STORED)
def test_bits_of_fp16_and_fp32_results(b200, name, case):
    B, Hq, Hkv, Sq, Sk, D, causal = SHAPES[case]
    g = torch.Generator().manual_seed(Sq + Sk)
    dtype = {"fp16": torch.float16, "fp32": torch.float32}[name]
    q, k, v = ((torch.randint(-96, 97, (B, h, s, D), generator=g).float() / 32).to(dtype).cuda() for h, s in ((Hq, Sq), (Hkv, Sk), (Hkv, Sk)))
    am = torch.tensor(3.0, device="cuda")
    out = b200.capi.fp8_sdpa(q, k, v, am, am, am, is_causal=causal)
    assert hashlib.sha256(out.cpu().contiguous().view(torch.uint8).numpy().tobytes()).hexdigest()[:16] == STORED[name, case]
