"""The kernel the library chooses for a problem with more than 128 rows, on both sides of the points where the choice
changes (rounds of tiles over the SMs), against the smallest tile forced: the same products, summed in fp32 in the same
order of K, so results differ by a bf16 rounding at most (rel-L2 <= 2^-9)."""
import pytest
import torch

import oracle as o

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(129, 4096, 512), (256, 10240, 256), (257, 10240, 256), (384, 10240, 256), (385, 10240, 256), (513, 4096, 512),
                                   (600, 28672, 256), (768, 28672, 256), (1100, 6144, 512), (2100, 1536, 512), (300, 1001, 544)])
def test_choice(b200, m, n, k):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, w = torch.randn(m, k, device="cuda", generator=g).bfloat16(), torch.randn(n, k, device="cuda", generator=g).bfloat16()
    bias = torch.randn(n, device="cuda", generator=g).bfloat16()
    fp8 = (*capi.fp8_quantize(x), *capi.fp8_quantize(w))
    nv = (*capi.nvfp4_quantize(x, capi.amax(x)), *capi.nvfp4_quantize(w, capi.amax(w)))
    for gemm, ops in ((capi.fp8_gemm, fp8), (capi.nvfp4_gemm, nv)):
        assert o.rel_l2(gemm(*ops, bias).float(), gemm(*ops, bias, tile_n=128).float()) <= 2.0 ** -9
    assert capi.device_status() == 0


@pytest.mark.parametrize("m,n", [(300, 4096), (600, 4104), (129, 1001)])
def test_output_on_a_16_byte_boundary(b200, m, n):
    """`out` may start on any 16-byte boundary, whichever kernel is chosen."""
    capi, k = b200.capi, 256
    x, w = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    fp8 = (*capi.fp8_quantize(x), *capi.fp8_quantize(w))
    nv = (*capi.nvfp4_quantize(x, capi.amax(x)), *capi.nvfp4_quantize(w, capi.amax(w)))
    for gemm, ops in ((capi.fp8_gemm, fp8), (capi.nvfp4_gemm, nv)):
        out = torch.empty(m * n + 8, device="cuda", dtype=torch.bfloat16)[8:].view(m, n)
        assert out.data_ptr() % 32 == 16
        gemm(*ops, out=out)
        assert torch.equal(out, gemm(*ops))
