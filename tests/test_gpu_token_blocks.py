"""The GEMM above 128 rows as blocks of tokens with K split over clusters: sizes around the block limits (256 tokens FP8, 128 NVFP4),
ragged weight rows and K, a bias, and every cluster size that the library chooses.  Operands are small integers, so that every
order of summation gives the same fp32 value and the result is compared bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# on 148 SMs: tiles, then clusters of 1, 2, 4 and 8
FP8_SIZES = [(129, 1024, 1024), (144, 1001, 528), (255, 256, 4096), (256, 4096, 2048), (257, 2048, 1040), (512, 1024, 2048), (513, 264, 1024),
             (257, 8190, 528), (144, 520, 2064), (700, 128, 4096),
             (647, 6266, 3088),
             (129, 6150, 4096), (513, 1530, 14336),
             (144, 520, 4112), (257, 1001, 8192),
             (129, 130, 8192), (333, 136, 8192), (255, 512, 14336), (1200, 264, 28672)]
# tiles, then clusters of 2, 4 and 8
NVFP4_SIZES = [(129, 1024, 1024), (144, 4090, 2080), (384, 2048, 2048), (257, 256, 2080),
               (144, 4090, 4128), (384, 2048, 8192),
               (256, 1001, 4096),
               (129, 520, 14336), (500, 136, 8192), (257, 256, 6176)]


@pytest.mark.parametrize("M,N,K", FP8_SIZES)
def test_fp8(b200, M, N, K):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    ints = lambda *shape: torch.randint(-2, 3, shape, device="cuda", generator=g).float()  # noqa: E731
    x, w, bias = ints(M, K), ints(N, K), ints(N).bfloat16()
    xs = 2.0 ** torch.randint(-2, 3, (M,), device="cuda", generator=g).float()             # a scale per token tells the rows apart
    to_codes = lambda t: t.to(torch.float8_e4m3fn).view(torch.uint8)  # noqa: E731
    y = capi.fp8_gemm(to_codes(x), xs, to_codes(w), torch.ones(N, device="cuda"), bias)
    ref = ((x.double() @ w.double().t()) * xs.double()[:, None] + bias.double()).float().bfloat16()
    assert torch.equal(y, ref) and capi.device_status() == 0


@pytest.mark.parametrize("M,N,K", NVFP4_SIZES)
def test_nvfp4(b200, M, N, K):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    values = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device="cuda")

    def operand(rows):
        codes = torch.randint(0, 5, (rows, K), device="cuda", generator=g) + 8 * torch.randint(0, 2, (rows, K), device="cuda", generator=g)
        block = 2.0 ** torch.randint(0, 2, (rows, 1), device="cuda", generator=g).float()   # one block scale per row, 1 or 2
        from oracle import swizzle_scales
        sf = (block * torch.ones(rows, K // 16, device="cuda")).to(torch.float8_e4m3fn).view(torch.uint8).cpu()
        ref = values[codes & 7] * torch.where(codes >= 8, -1.0, 1.0) * block
        return ((codes[:, 0::2] | (codes[:, 1::2] << 4)).to(torch.uint8), swizzle_scales(sf).cuda(), torch.ones(1, device="cuda")), ref

    (xq, x), (wq, w) = operand(M), operand(N)
    y = capi.nvfp4_gemm(*xq, *wq)
    assert torch.equal(y, (x.double() @ w.double().t()).float().bfloat16()) and capi.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(512, 2048, 8192), (1500, 1024, 8192), (129, 6150, 4096)])
@pytest.mark.parametrize("force", [1001, 1002, 1004, 1008])
def test_forced_cluster_size_is_for_128_rows(b200, M, N, K, force):
    """Above 128 rows it is ignored: the bits of the library's own choice (other kernels sum K in another order)."""
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    ops = (*capi.fp8_quantize(x), *capi.fp8_quantize(w))
    assert torch.equal(capi.fp8_gemm(*ops, tile_n=force), capi.fp8_gemm(*ops)) and capi.device_status() == 0
