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


def test_nan_beside_values_above_the_range(b200):
    """A weight block of NaN makes one gate column and one up column NaN; under a range below the data the blocks around them
    saturate, and the NaN's codes are decided there."""
    capi = b200.capi
    M, F, K = 300, 256, 512
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(2 * F, K, device="cuda", generator=g).bfloat16()
    top = capi.amax(w)
    w[21, 16:32] = float("nan")
    w[F + 133, :16] = float("nan")
    xq, wq = capi.nvfp4_quantize(x, capi.amax(x)), capi.nvfp4_quantize(w, top)
    act = capi.silu_mul(capi.nvfp4_gemm(*xq, *wq, tile_n=512))
    assert int(act.isnan().sum()) == 2 * M
    for amax in (capi.amax(act), capi.amax(act) * 0.01):
        got, ref = capi.nvfp4_gemm_silu_mul_quantize(*xq, *wq, amax), capi.nvfp4_quantize(act, amax)
        assert all(torch.equal(a, b) for a, b in zip(got, ref))


@pytest.mark.parametrize("M,F", [(129, 128), (300, 384)])
def test_code_buffer_off_a_32_byte_boundary(b200, M, F):
    """Codes that start 16 bytes behind a 32-byte boundary leave in 16-byte stores: the same bytes, and none beside them."""
    from tensorrt_b200 import _lib

    capi = b200.capi
    K = 512
    g = torch.Generator(device="cuda").manual_seed(M + F)
    xq = capi.nvfp4_quantize_dynamic(torch.randn(M, K, device="cuda", generator=g).bfloat16())
    wq = capi.nvfp4_quantize_dynamic(torch.randn(2 * F, K, device="cuda", generator=g).bfloat16())
    amax = torch.tensor([50.0], device="cuda")
    ref = capi.nvfp4_gemm_silu_mul_quantize(*xq, *wq, amax)
    store = torch.full((M * F // 2 + 64,), 0xA5, dtype=torch.uint8, device="cuda")
    codes = store[16:16 + M * F // 2]
    assert codes.data_ptr() % 32 == 16
    sf, out_g = torch.empty_like(ref[1]), torch.empty_like(ref[2])
    assert _lib.load().b200q_nvfp4_gemm_silu_mul_quantize(*(t.data_ptr() for t in (*xq, *wq, amax, codes, sf, out_g)), M, 2 * F, K,
                                                          torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(codes.view(M, -1), ref[0].view(M, -1)) and torch.equal(sf, ref[1]) and torch.equal(out_g, ref[2])
    assert bool((store[:16] == 0xA5).all()) and bool((store[16 + M * F // 2:] == 0xA5).all())


def test_argument_errors(b200):
    capi = b200.capi
    xq, wq = capi.nvfp4_quantize_dynamic(torch.randn(4, 64, device="cuda")), capi.nvfp4_quantize_dynamic(torch.randn(384, 64, device="cuda"))
    with pytest.raises(ValueError):
        capi.nvfp4_gemm_silu_mul_quantize(*xq, *wq, torch.ones((), device="cuda"))          # F not a multiple of 128
