"""Exponentials of the FP8 attention on the special-function unit and on the FMA pipe: the range of scores where the result
underflows, and NaN at every column of a key tile (which of the two computes a score depends on its column)."""
import pytest
import torch

import oracle as o


def _sdpa(lib, qc, kc, vt, scales, B, H, Sq, Sk, D, causal):
    out = torch.full((B, H, Sq, D), 7.0, device="cuda")
    s = scales.data_ptr()
    assert lib.b200q_fp8_sdpa(qc.data_ptr(), kc.data_ptr(), vt.data_ptr(), s, s + 4, s + 8, out.data_ptr(), 0, B, H, H, Sq, Sk, vt.shape[-1], D,
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


@pytest.mark.gpu
@pytest.mark.parametrize("sk,causal", [(128, 0), (256, 0), (200, 1)])
def test_nan_key_reaches_every_row_that_sees_it(b200, sk, causal):
    from tensorrt_b200 import _lib

    lib, D, H = _lib.load(), 32, sk                      # head h: key h is NaN
    g = torch.Generator(device="cuda").manual_seed(sk)
    codes = lambda *shape: (torch.randn(*shape, device="cuda", generator=g)).to(torch.float8_e4m3fn).view(torch.uint8)  # noqa: E731
    stride = (sk + 15) // 16 * 16
    qc, kc, vt = codes(1, H, sk, D), codes(1, H, sk, D), codes(1, H, D, stride)
    vt[..., sk:] = 0
    for h in range(H):
        kc[0, h, h, 5] = 0x7F
    out = _sdpa(lib, qc, kc, vt, torch.ones(3, device="cuda"), 1, H, sk, sk, D, causal)
    seen = torch.ones(sk, sk, dtype=torch.bool, device="cuda").tril() if causal else torch.ones(sk, sk, dtype=torch.bool, device="cuda")
    nan = out[0].isnan()                                  # [head = NaN key, query, D]
    assert torch.equal(nan.all(dim=2), seen.t()) and torch.equal(nan.any(dim=2), seen.t())
