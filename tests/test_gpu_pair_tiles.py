"""FP8 GEMM on CTA pairs with 256 x 192 tiles: the same bits as with 256 x 256 (the same products in the same order of K), forced and
where the library chooses it, at ragged rows, columns and K."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 8, 16), (129, 192, 128), (256, 193, 400), (257, 1001, 256), (300, 384, 1040), (200, 10240, 256), (512, 10240, 384),
                                   (600, 8192, 128), (5000, 200, 256)])
def test_same_bits_as_wide_tiles(b200, m, n, k):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, w = torch.randn(m, k, device="cuda", generator=g).bfloat16(), torch.randn(n, k, device="cuda", generator=g).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g).bfloat16()
    ops = (*capi.fp8_quantize(x), *capi.fp8_quantize(w), bias)
    wide = capi.fp8_gemm(*ops, tile_n=512)
    assert torch.equal(capi.fp8_gemm(*ops, tile_n=448), wide)
    if m >= 200 and n >= 8192:
        assert torch.equal(capi.fp8_gemm(*ops), wide)
    assert capi.device_status() == 0
