"""The GEMM above 128 rows as blocks of tokens with K split over clusters: sizes around the block limits (256 tokens FP8, 128 NVFP4),
ragged weight rows and K, a bias, every cluster size forced and the library's choice.  Operands are small integers, so that every
order of summation gives the same fp32 value and the result is compared bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(129, 1024, 1024), (144, 1001, 528), (255, 256, 4096), (256, 4096, 2048), (257, 2048, 1040), (333, 136, 8192), (512, 1024, 2048), (513, 264, 1024),
         (700, 128, 4096)]


@pytest.mark.parametrize("force", [0, 1001, 1002, 1004, 1008])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_fp8(b200, M, N, K, force):
    capi = b200.capi
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    ints = lambda *shape: torch.randint(-2, 3, shape, device="cuda", generator=g).float()  # noqa: E731
    x, w, bias = ints(M, K), ints(N, K), ints(N).bfloat16()
    xs = 2.0 ** torch.randint(-2, 3, (M,), device="cuda", generator=g).float()             # a scale per token tells the rows apart
    to_codes = lambda t: t.to(torch.float8_e4m3fn).view(torch.uint8)  # noqa: E731
    if force > 1000 and (K + 127) // 128 < force - 1000:
        force = 0
    y = capi.fp8_gemm(to_codes(x), xs, to_codes(w), torch.ones(N, device="cuda"), bias, tile_n=force)
    ref = ((x.double() @ w.double().t()) * xs.double()[:, None] + bias.double()).float().bfloat16()
    assert torch.equal(y, ref) and capi.device_status() == 0


@pytest.mark.parametrize("force", [0, 1001, 1002, 1004, 1008])
@pytest.mark.parametrize("M,N,K", [(129, 1024, 1024), (256, 1001, 4096), (257, 256, 2080), (384, 2048, 2048), (500, 136, 8192)])
def test_nvfp4(b200, M, N, K, force):
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

    if force > 1000 and (K // 2 + 127) // 128 < force - 1000:
        force = 0
    (xq, x), (wq, w) = operand(M), operand(N)
    y = capi.nvfp4_gemm(*xq, *wq, tile_n=force)
    assert torch.equal(y, (x.double() @ w.double().t()).float().bfloat16()) and capi.device_status() == 0
