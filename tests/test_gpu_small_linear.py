"""FP8 linear of a few tokens in one launch (the GEMM quantizes its activation): the same bits as the quantize kernel
followed by the GEMM, for every way of scaling, at the edges of its range (activation bytes, tokens, K tiles per CTA,
weight tiles, ragged N and K) and outside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("m,n,k", [(1, 4096, 4096), (1, 128, 16), (1, 130, 144), (2, 1000, 2064), (7, 257, 1040), (16, 4096, 4096), (16, 8192, 4112),
                                   (15, 384, 4368), (9, 512, 7280), (1, 1024, 28672), (2, 28672, 32768), (1, 136, 65536), (17, 256, 1024),
                                   (1, 1921, 16), (1, 1920, 16), (8, 4096, 1024), (8, 2049, 512), (9, 4096, 512), (2, 4100, 4096), (2, 4096, 2048),
                                   (3, 2001, 1360), (5, 2100, 1024), (5, 2100, 1040), (7, 6144, 144), (1, 28672, 512), (1, 28672, 528),
                                   (1, 10240, 1008), (2, 14336, 1024), (4, 28672, 256), (1, 4096, 4112), (6, 4097, 640)])
def test_same_bits_as_two_launches(b200, m, n, k, dtype):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n + k)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    w, ws = capi.fp8_quantize((torch.randn(n, k, device="cuda", generator=g) * 0.02).bfloat16(), None)
    bias = torch.randn(n, device="cuda", generator=g).bfloat16()
    per_token = x.abs().amax(dim=1).float() * 0.5                          # some elements saturate
    for amax, b in ((None, None), (x.abs().max().float(), bias), (per_token, bias), (torch.zeros((), device="cuda"), None)):
        xq, xs = capi.fp8_quantize(x, amax)
        ref = capi.fp8_gemm(xq, xs, w, ws, b)
        assert torch.equal(b200.fp8_linear(x, w, ws, b, amax), ref)
    assert torch.equal(b200.fp8_linear(torch.zeros_like(x), w, ws), torch.zeros(m, n, device="cuda", dtype=torch.bfloat16))
    assert capi.device_status() == 0


@pytest.mark.parametrize("m,n,k", [(1, 4224, 1024), (1, 4352, 1024), (8, 4352, 512), (2, 4736, 1536), (4, 9088, 512), (1, 9216, 512), (3, 9472, 512)])
def test_cluster_counts_around_what_is_resident(b200, m, n, k):
    """33, 34, 37, 71, 72 and 74 weight tiles: at most as many clusters as are resident at once, else smaller ones (or, where
    the K slices are then too long, two launches).  The same bits as two launches at any cluster size."""
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(n + k)
    x = torch.randint(-2, 3, (m, k), device="cuda", generator=g).bfloat16()       # sums that are the same in any order
    w = torch.randint(-2, 3, (n, k), device="cuda", generator=g).float().to(torch.float8_e4m3fn).view(torch.uint8)
    one = torch.ones((), device="cuda")
    y = b200.fp8_linear(x, w, one.reshape(1), None, one * 448)
    assert torch.equal(y, (x.double() @ w.view(torch.float8_e4m3fn).double().t()).bfloat16())
    assert capi.device_status() == 0
