"""NVFP4 gate/up GEMM with silu(gate) * up and its quantizer in the epilogue: codes, swizzled scales (padding rows of the last
128-row tile included) and global scale equal GEMM on the same tiles, silu_mul and nvfp4_quantize bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 127, 129, 256, 300, 385, 513])
@pytest.mark.parametrize("F,K", [(128, 32), (384, 1056), (2048, 512)])
def test_matches_separate_kernels(b200, M, F, K):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(M + F + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(2 * F, K, device="cuda", generator=g).bfloat16()
    xq, wq = capi.nvfp4_quantize(x, capi.amax(x)), capi.nvfp4_quantize(w, capi.amax(w))
    act = capi.silu_mul(capi.nvfp4_gemm(*xq, *wq, tile_n=512))
    top = capi.amax(act)
    for amax in (top, top * 0.25, torch.zeros((), device="cuda")):
        got, ref = capi.nvfp4_gemm_silu_mul_quantize(*xq, *wq, amax), capi.nvfp4_quantize(act, amax)
        assert all(a.shape == b.shape and torch.equal(a, b) for a, b in zip(got, ref))
    assert capi.device_status() == 0


def test_argument_errors(b200):
    capi = b200.capi
    xq, wq = capi.nvfp4_quantize_dynamic(torch.randn(4, 64, device="cuda")), capi.nvfp4_quantize_dynamic(torch.randn(384, 64, device="cuda"))
    with pytest.raises(ValueError):
        capi.nvfp4_gemm_silu_mul_quantize(*xq, *wq, torch.ones((), device="cuda"))          # F not a multiple of 128
